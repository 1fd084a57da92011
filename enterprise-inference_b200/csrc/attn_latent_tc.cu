// Paged causal attention over latent cache rows on tcgen05 (bf16 serving mode of B200_MIXER_LATENT).
//
// One kv head serves every query head and a key row's leading `rank` entries are its value.  A work item is 128 (row, head)
// pairs of one run of consecutive rows of a sequence (128 / heads rows) on the MMA's M dimension times one half of the value
// columns; per tile of 64 keys
//   S[128][64] = Q[128][krow] . K_tile^T            O[128][<= 256] += P[128][64] . V_tile   (V_tile: columns of K_tile, MN-major)
// The two halves of the value columns are items of their own because O takes all 512 TMEM columns otherwise: the scores are
// computed twice (1.5 x the operations), and nothing is exchanged between CTAs.
//
// What bounds it: the issue and execution of 36 score MMAs of 64 columns a tile (about 1.6 us per tile, krow 576), then the query
// staging and the output at an item's ends.  Q is the large operand (krow 576: 147 KB of bf16), so the part that matches the value
// columns lives in TMEM (columns 384..511, A operand read from there) and only the rest in shared memory, which leaves room for
// two tiles of keys.  TMEM: O 0..255, two score buffers of 64 columns, the Q part.
// The weights overwrite the scores in place (A operand of the second product, per 32 scores 16 columns of bf16 pairs and 16 of what
// rounding took from them) and never touch shared memory.
// Against the mma.sync kernel of attn_latent.cu with 16 pairs a CTA, which reads every key tile once per row: 2 048 rows of 16
// heads over 512 + 64 at contexts 1..2048 907 -> 170 us among other calls; error against 64 bits 2.57e-3 -> 2.30e-3 (decode rows: attn_latent_rows.cu).  (With weights of one bf16 term, as there, about a tenth faster, but 2.61e-3 and 2.72e-3: the
// lazily followed maximum costs the exactness of the largest weight.)
// Warps: TMA producer, MMA issuer, four softmax warps (a thread owns a pair), eight that stage the next item's queries.
// The running maximum is only followed when it rises by more than 2^8 (the scaling of all terms is the same, so the
// quotient is exact); a warp then rescales its own 32 rows of O in TMEM.
// Every wait is bounded and reported (tc.cuh).
#include <algorithm>
#include <type_traits>

#include "runs.cuh"
#include "tc.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int kLtKeys = 64, kLtPairs = 128, kLtThreads = 448;
constexpr int kLtChunk = kLtKeys * 128;        // [64 keys][64 columns] bf16: 8 KiB
constexpr int kLtQChunk = kLtPairs * 128;      // [128 pairs][64 columns] bf16: 16 KiB
constexpr int kLtMaxStages = 4, kLtMaxRest = 5, kLtMaxRestStages = 4;
constexpr int kLtSmem = 232448, kLtTail = 2048;
constexpr int kLtTable = 32;                   // items of a CTA whose description is worked out ahead
constexpr uint32_t kTmS = 256, kTmQ = 384;     // TMEM columns: O at 0, scores (then weights) of even / odd tiles, Q part

// 64-wide chunks of the values, and those that are a half's own: of more than 256 columns half of the chunks, the last ones in the second half.  Of an odd count
// the middle chunk is in both, and the second half writes it: either half then runs the same code (halves of 4 and 3 chunks, each with straight code of its own: 448 + 64
// 241 us for 2 048 rows of 16 heads behind 300 tokens, though either half by itself took 166 and 181; 172 so)
__host__ __device__ __forceinline__ int lt_value_chunks(int rank) { return (rank + 63) >> 6; }
__host__ __device__ __forceinline__ int lt_own(int rank) { return rank > 256 ? (lt_value_chunks(rank) + 1) >> 1 : lt_value_chunks(rank); }

struct LtParams {
  const float* q;
  const int32_t* block_table;
  const int32_t* row_to_seq;
  const int32_t* ctx_lens;
  const int32_t* runs;      // (first row, rows) pairs: at most 16 rows of one sequence, contexts rising by one
  const int32_t* n_runs;
  const float* sink;
  __nv_bfloat16* out;
  float* part;
  uint32_t* status;
  int n_rows, bt_stride, heads, krow, rank, block_size, n_splits, window, own_stages, rest_stages, halves, rows_per_item, items_per_run;
  float scale;
  LatentShare share;
};

struct LtItem {
  int t0, nr, half, split, seq, ctx0, ctx_max, tile_lo, tile_hi;   // ctx0: context of the item's first row
};

// item `it` of the list (run, part of the run, split, half); false: nothing there
__device__ __forceinline__ bool lt_item(const LtParams& p, int n_runs, int it, LtItem& w) {
  w.half = it % p.halves;
  it /= p.halves;
  w.split = it % p.n_splits;
  it /= p.n_splits;
  // mostly whole runs (prefill): a run's parts follow each other, all by falling context.  Mostly short runs (decode rows): the first
  // parts of all runs lead, so that the parts that do not exist fall to the end of the list and every CTA gets its share of work
  const bool whole = p.n_rows >= n_runs * p.rows_per_item;
  const int part = whole ? p.items_per_run - 1 - it % p.items_per_run : it / n_runs;
  const int run = n_runs - 1 - (whole ? it / p.items_per_run : it % n_runs);
  const int2 r = __ldg(reinterpret_cast<const int2*>(p.runs) + run);
  w.t0 = r.x + part * p.rows_per_item;
  w.nr = min((r.y & kRunLength) - part * p.rows_per_item, p.rows_per_item);
  if (w.nr <= 0) return false;
  w.seq = p.row_to_seq ? __ldg(p.row_to_seq + w.t0) : w.t0;
  w.ctx0 = __ldg(p.ctx_lens + w.t0);
  w.ctx_max = __ldg(p.ctx_lens + w.t0 + w.nr - 1);
  const int tile0 = p.window > 0 ? max(w.ctx0 - p.window, 0) / kLtKeys : 0;
  const int tiles = max((w.ctx_max + kLtKeys - 1) / kLtKeys - tile0, 0), per = (tiles + p.n_splits - 1) / p.n_splits;
  w.tile_lo = tile0 + min(tiles, w.split * per);
  w.tile_hi = tile0 + min(tiles, (w.split + 1) * per);
  return true;
}

__global__ void __launch_bounds__(kLtThreads, 1) latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map, const LtParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (p.krow + 63) >> 6, ksteps = p.krow >> 4;
  const int own = lt_own(p.rank), rest = chunks - own, second = lt_value_chunks(p.rank) - own;   // second: the second half's first chunk
  unsigned char* qs = smem;                                  // [rest][128][64] queries of the columns outside the half
  unsigned char* own_ring = qs + rest * kLtQChunk;       // [own_stages][own][64][64] value columns of a tile
  unsigned char* rest_ring = own_ring + p.own_stages * own * kLtChunk;   // [rest_stages][rest][64][64] a tile's other chunks
  uint64_t* own_full = reinterpret_cast<uint64_t*>(rest_ring + p.rest_stages * rest * kLtChunk);
  uint64_t* own_free = own_full + kLtMaxStages;
  uint64_t* rest_full = own_free + kLtMaxStages;
  uint64_t* rest_free = rest_full + kLtMaxRestStages;
  uint64_t* s_full = rest_free + kLtMaxRestStages;    // [2]
  uint64_t* p_ready = s_full + 2;                // [2]
  uint64_t* o_full = p_ready + 2;                // [2]
  uint64_t* q_ready = o_full + 2;
  uint64_t* q_free = q_ready + 1;
  uint64_t* last = q_free + 1;                   // the MMAs in flight when a wait ran out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(last + 1);   // and, behind it, the mark of a wait that ran out
  const Waits mbar_wait(tmem_slot + 1, p.status);
  if (p.share.plan) {
    pdl_wait();
    if (latent_by_rows(p.share)) return;
  }
  LtItem* table = reinterpret_cast<LtItem*>(tmem_slot + 2);   // nr 0: nothing there
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.own_stages; ++s) {
      mbar_init(own_full + s, 1);
      mbar_init(own_free + s, 1);
    }
    for (int s = 0; s < p.rest_stages; ++s) {
      mbar_init(rest_full + s, 1);
      mbar_init(rest_free + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + s, 1);
      mbar_init(p_ready + s, 4);
      mbar_init(o_full + s, 1);
    }
    mbar_init(q_ready, 8);
    mbar_init(q_free, 1);
    mbar_init(last, 1);
    tmem_slot[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  pdl_wait();
  pdl_launch_dependents();
  const int n_runs = *p.n_runs, n_items = n_runs * p.items_per_run * p.n_splits * p.halves;
  // the descriptions hang on a chain of loads (run, contexts, sequence): all of the CTA's first ones at once, for every role
  if (warp == 6 && (int)(blockIdx.x + lane * gridDim.x) < n_items) {
    LtItem w;
    if (!lt_item(p, n_runs, blockIdx.x + lane * gridDim.x, w)) w.nr = 0;
    table[lane] = w;
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  int turn = 0;   // of the role's walk over the CTA's items
  auto next_item = [&](int it, LtItem& w) {
    const int k = turn++;
    if (k >= kLtTable) return lt_item(p, n_runs, it, w);
    w = table[k];
    return w.nr > 0;
  };

  if (warp == 0) {
    // ===== TMA: per tile the chunks outside the half first (the scores take them first), then the half's own =====
    const bool issuer = elect_one();
    if (issuer) asm volatile("prefetch.tensormap [%0];" ::"l"(&map) : "memory");
    int st = 0, sl = 0;
    uint32_t st_ph = 1, sl_ph = 1;   // parity of the release that a slot's next load waits for (the first round finds it free)
    bool stop = false;
    for (int it = blockIdx.x; it < n_items && !stop; it += gridDim.x) {
      LtItem w;
      if (!next_item(it, w)) continue;
      const int first = w.half * second;
      const int32_t* bt = p.block_table + (int64_t)w.seq * p.bt_stride;
      for (int i = w.tile_lo; i < w.tile_hi && !(stop = mbar_wait.stop()); ++i) {
        const int tok = i * kLtKeys;
        const int blk = __shfl_sync(0xffffffffu, __ldg(bt + tok / p.block_size), 0);
        const int row = blk * p.block_size + tok % p.block_size;
        if (rest > 0) {
          mbar_wait(rest_free + sl, sl_ph);
          if (issuer) {
            mbar_expect_tx(rest_full + sl, rest * kLtChunk);
            for (int c = 0; c < rest; ++c) tma_load_2d(rest_ring + (sl * rest + c) * kLtChunk, &map, (c < first ? c : c + own) * 64, row, rest_full + sl);
          }
          if (++sl == p.rest_stages) sl = 0, sl_ph ^= 1;
        }
        mbar_wait(own_free + st, st_ph);
        if (issuer) {
          mbar_expect_tx(own_full + st, own * kLtChunk);
          for (int c = 0; c < own; ++c) tma_load_2d(own_ring + (st * own + c) * kLtChunk, &map, (first + c) * 64, row, own_full + st);
        }
        __syncwarp();
        if (++st == p.own_stages) st = 0, st_ph ^= 1;
      }
    }
    if (mbar_wait.stop()) {   // the loads in flight: a slot's last one filled it in this round of the ring or in the one before
      for (int s = 0; s < p.own_stages; ++s) mbar_wait.drain(own_full + s, s < st ? st_ph ^ 1 : st_ph);
      for (int s = 0; s < p.rest_stages; ++s) mbar_wait.drain(rest_full + s, s < sl ? sl_ph ^ 1 : sl_ph);
    }
  } else if (warp == 1) {
    // ===== MMA: the scores of tile n + 1 are issued before the weights of tile n are waited for.  The whole warp walks the loop; bounds
    // and addresses that come from memory are broadcast, so that they are uniform to the compiler =====
    const uint32_t one = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t desc_q = make_desc(smem_u32(qs), 16, 1024), desc_own = make_desc(smem_u32(own_ring), 16, 1024),
                   desc_rest = make_desc(smem_u32(rest_ring), 16, 1024), desc_v = make_desc(smem_u32(own_ring), kLtChunk, 1024);
    const int items = __shfl_sync(0xffffffffu, n_items, 0);
    int st = 0, sl = 0, pv_st = 0;   // own stage and rest slot of the next scores, own stage of the next second product
    uint32_t st_ph = 0, sl_ph = 0;
    int n = 0, active = 0;   // n: tiles walked by the items before
    // An item of nt key tiles whose half has O chunks of its own and R others.  Issuing is what bounds the walk (with MMAs a quarter as wide it took as long) and
    // branches between the MMAs cost it: straight code for every pair of counts, but for the row's last chunk where it is not whole (`own_tail`, `rest_tail`: its
    // 16-wide steps, 4 otherwise).  2 048 rows of 16 heads behind 300 tokens, us, with a loop over chunks and a wait for each / so: 512 + 64 219 / 189, 256 + 32
    // 91 / 83, 448 + 64 201 / 172, 320 + 32 168 / 134, 192 + 64 83 / 74, 64 + 64 67 / 65.
    auto walk = [&](auto own_c, auto rest_c, int nt, uint32_t id_o, int own_tail, int rest_tail) {
      constexpr int O = decltype(own_c)::value, R = decltype(rest_c)::value;
      const uint32_t id_s = idesc_bf16(kLtKeys, 0);
      auto last_chunk = [&](int tail, auto&& step, auto base_c) {
        constexpr int base = decltype(base_c)::value;
        if (tail == 4) {
#pragma unroll
          for (int j = 0; j < 4; ++j) step(base + j);
        } else {
          step(base);
          if (tail > 1) step(base + 1);
          if (tail > 2) step(base + 2);
        }
      };
      auto scores = [&](int m) {
        const uint32_t d = tm + kTmS + (m & 1) * kLtKeys;
        if constexpr (R > 0) {
          mbar_wait(rest_full + sl, sl_ph);
          fence_after();
          const uint64_t dr = desc_rest + (uint64_t)((sl * rest * kLtChunk) >> 4);
          auto step = [&](int j) {
            mma_ss(one, d, desc_q + (uint64_t)(((j >> 2) * kLtQChunk >> 4) + (j & 3) * 2), dr + (uint64_t)(((j >> 2) * kLtChunk >> 4) + (j & 3) * 2), id_s, j ? 1u : 0u);
          };
#pragma unroll
          for (int j = 0; j < 4 * (R - 1); ++j) step(j);
          last_chunk(rest_tail, step, std::integral_constant<int, 4 * (R - 1)>());
          commit(one, rest_free + sl);
          if (++sl == p.rest_stages) sl = 0, sl_ph ^= 1;
        }
        mbar_wait(own_full + st, st_ph);
        fence_after();
        const uint64_t dk = desc_own + (uint64_t)((st * own * kLtChunk) >> 4);
        auto step = [&](int j) { mma_ts(one, d, tm + kTmQ + j * 8, dk + (uint64_t)(((j >> 2) * kLtChunk >> 4) + (j & 3) * 2), id_s, R > 0 || j ? 1u : 0u); };
#pragma unroll
        for (int j = 0; j < 4 * (O - 1); ++j) step(j);
        last_chunk(own_tail, step, std::integral_constant<int, 4 * (O - 1)>());
        commit(one, s_full + (m & 1));
        if (++st == p.own_stages) st = 0, st_ph ^= 1;
      };
      scores(n);
      if (nt == 1) commit(one, q_free);
      for (int i = 0; i < nt; ++i) {
        const int m = n + i;
        if (i + 1 < nt) {
          scores(m + 1);
          if (i + 2 == nt) commit(one, q_free);   // the item's last scores are on their way
        }
        mbar_wait(p_ready + (m & 1), (m >> 1) & 1);
        fence_after();
        const uint64_t dv = desc_v + (uint64_t)((pv_st * own * kLtChunk) >> 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // 16 keys per step: 8 columns of weights, 16 further those of the second term
          const uint32_t pa = tm + kTmS + (m & 1) * kLtKeys + (j >> 1) * 32 + (j & 1) * 8;
          mma_ts(one, tm, pa, dv + (uint64_t)((j * 2048) >> 4), id_o, (i | j) ? 1u : 0u);
          mma_ts(one, tm, pa + 16, dv + (uint64_t)((j * 2048) >> 4), id_o, 1u);
        }
        commit(one, own_free + pv_st);
        commit(one, o_full + (m & 1));
        if (++pv_st == p.own_stages) pv_st = 0;
      }
    };
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
      LtItem w;
      const bool have = next_item(it, w);
      const int nt = __shfl_sync(0xffffffffu, have ? w.tile_hi - w.tile_lo : 0, 0);
      if (nt <= 0) continue;
      const int half = __shfl_sync(0xffffffffu, w.half, 0);
      const uint32_t id_o = idesc_bf16(min(own * 64, p.rank - half * second * 64), 1);
      const int tail = ksteps & 3 ? ksteps & 3 : 4;
      const bool own_last = half * second + own == chunks;   // the row's last chunk is one of the half's own
      mbar_wait(q_ready, active & 1);
      fence_after();
      using std::integral_constant;
#define LT_WALK(O, R) \
  case O * 8 + R: walk(integral_constant<int, O>(), integral_constant<int, R>(), nt, id_o, own_last ? tail : 4, own_last ? 4 : tail); break;
#define LT_WALKS(O) LT_WALK(O, 0) LT_WALK(O, 1) LT_WALK(O, 2) LT_WALK(O, 3) LT_WALK(O, 4) LT_WALK(O, 5)
      static_assert(kLtMaxRest == 5, "counts of the other chunks");
      switch (own * 8 + rest) { LT_WALKS(1) LT_WALKS(2) LT_WALKS(3) LT_WALKS(4) }
#undef LT_WALKS
#undef LT_WALK
      n += nt;
      ++active;
    }
    if (mbar_wait.stop()) {
      commit(one, last);
      mbar_wait.drain(last, 0);
    }
  } else if (warp >= 6) {
    // ===== queries of the next item: fp32 rows -> bf16, the half's own columns to TMEM, the others to shared memory.  Two warps
    // per quarter of the pairs, the chunks dealt alternately.  The own part travels into registers while the item before is still
    // computed; the shared-memory part follows once its last scores have been taken. =====
    const int quad = warp & 3, sub = (warp - 6) >> 2;
    int active = 0;
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
      LtItem w;
      if (!next_item(it, w) || w.tile_hi <= w.tile_lo) continue;
      const int first = w.half * second;
      const int live = w.nr * p.heads;
      const float* qbase = p.q + (int64_t)w.t0 * p.heads * p.krow;   // pair m = (row m / heads, head m % heads): row m of this
      // four lanes take 64 neighbouring bytes of a row, eight rows per load: the fragment layout of the 16-lane store
      uint32_t r[2][2][16];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int c = sub + 2 * k;
#pragma unroll
        for (int hl = 0; hl < 2; ++hl) {
          float4 v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {   // piece j / 2 of 16 columns, rows x / 4 (j even) and x / 4 + 8
            const int col = (first + c) * 64 + (j >> 1) * 16 + (lane & 3) * 4, mm = quad * 32 + hl * 16 + (j & 1) * 8 + (lane >> 2);
            v[j] = c < own && mm < live && col < p.krow ? __ldg(reinterpret_cast<const float4*>(qbase + (int64_t)mm * p.krow + col))
                                                        : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            r[k][hl][2 * j] = pack_bf16(v[j].x, v[j].y);
            r[k][hl][2 * j + 1] = pack_bf16(v[j].z, v[j].w);
          }
        }
      }
      if (active > 0) mbar_wait(q_free, (active - 1) & 1);
      fence_after();
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (sub + 2 * k < own) {
          const uint32_t a = tmem + kTmQ + (sub + 2 * k) * 32 + ((uint32_t)(quad * 32) << 16);
          st_16x256b_x4(a, r[k][0]);
          st_16x256b_x4(a + (16u << 16), r[k][1]);
        }
      // eight lanes per row of a chunk (16-byte pieces), four rows per step
      for (int c = sub; c < rest; c += 2) {
        const int col = (c < first ? c : c + own) * 64 + (lane & 7) * 8;
        float4 v[16];
#pragma unroll
        for (int r4 = 0; r4 < 8; ++r4) {
          const int mm = quad * 32 + r4 * 4 + (lane >> 3);
          const bool ok = mm < live && col < p.krow;
          const float4* src = reinterpret_cast<const float4*>(qbase + (int64_t)mm * p.krow + col);
          v[2 * r4] = ok ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[2 * r4 + 1] = ok ? __ldg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r4 = 0; r4 < 8; ++r4) {
          const int mm = quad * 32 + r4 * 4 + (lane >> 3);
          const float4 a = v[2 * r4], b = v[2 * r4 + 1];
          *reinterpret_cast<uint4*>(qs + c * kLtQChunk + (mm >> 3) * 1024 + (mm & 7) * 128 + (((lane & 7) ^ (mm & 7)) << 4)) =
              make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
        }
      }
      st_wait();
      fence_async_smem();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_ready);
      ++active;
    }
  } else {
    // ===== softmax and output: a thread owns a pair =====
    const int quad = warp & 3, m = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const int r = m / p.heads, h = m % p.heads;
    const float sc2 = p.scale * 1.4426950408889634f;   // scores in the log2 domain
    int n = 0;
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
      LtItem w;
      if (!next_item(it, w)) continue;
      const bool alive = r < w.nr;
      const int ctx = alive ? w.ctx0 + r : 0, lo = p.window > 0 ? max(ctx - p.window, 0) : 0;
      const int col0 = w.half * second * 64, width = min(own * 64, p.rank - col0), written = p.halves > 1 && w.half == 0 ? second * 64 : width;   // the middle chunk: by the second half
      float mu = -INFINITY, l = 0.f;
      for (int i = w.tile_lo; i < w.tile_hi; ++i, ++n) {
        const int base = i * kLtKeys;
        mbar_wait(s_full + (n & 1), (n >> 1) & 1);
        fence_after();
        const uint32_t s_addr = tmem + lane_off + kTmS + (n & 1) * kLtKeys;
        uint32_t s[64];
        ld32(s_addr, s);
        ld32(s_addr + 32, s + 32);
        ld_wait<64>(s);
        const int j_lo = lo - base, j_hi = ctx - base;   // live columns [j_lo, j_hi)
        if (__any_sync(0xffffffffu, j_lo > 0 || j_hi < kLtKeys)) {
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (j < j_lo || j >= j_hi) s[j] = 0xff800000u;   // -inf
        }
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 64; ++j) mx = fmaxf(mx, __uint_as_float(s[j]));
        mx *= sc2;
        const bool jump = mx > mu + 8.f;   // also the first live key (mu = -inf)
        if (__any_sync(0xffffffffu, jump)) {
          const float mn = jump ? mx : mu, f = jump && mu != -INFINITY ? exp2_fast(mu - mn) : 1.f;
          if (i > w.tile_lo) {
            mbar_wait(o_full + ((n - 1) & 1), ((n - 1) >> 1) & 1);
            fence_after();
            if (__any_sync(0xffffffffu, f != 1.f))
              for (int c = 0; c < width; c += 16) {
                uint32_t o[16];
                ld16(tmem + lane_off + c, o);
                ld_wait<16>(o);
#pragma unroll
                for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                st16(tmem + lane_off + c, o);
              }
          }
          l *= f;
          mu = mn;
        }
        const float mref = mu > -INFINITY ? mu : 0.f;
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 2; ++c) {   // per 32 keys 16 columns of bf16 pairs, 16 of what that rounding took
          uint32_t pk[32];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float p0 = exp2_fast(fmaf(__uint_as_float(s[c * 32 + 2 * j]), sc2, -mref)), p1 = exp2_fast(fmaf(__uint_as_float(s[c * 32 + 2 * j + 1]), sc2, -mref));
            sum[j & 1] += p0 + p1;
            const uint32_t h0 = __float_as_uint(p0) & 0xffff0000u, h1 = __float_as_uint(p1) & 0xffff0000u;
            pk[j] = __byte_perm(h0, h1, 0x7632);
            pk[16 + j] = pack_bf16(p0 - __uint_as_float(h0), p1 - __uint_as_float(h1));
          }
          st32(s_addr + c * 32, pk);
        }
        l += sum[0] + sum[1];
        const int n_valid = w.ctx_max - base;
        if (n_valid < kLtKeys) {
          // value rows past the context may hold anything, and 0 * NaN = NaN: zero them under their zero weights
          const int st = n % p.own_stages;
          mbar_wait(own_full + st, (n / p.own_stages) & 1);
          unsigned char* vb = own_ring + st * own * kLtChunk;
          for (int c = 0; c < own; ++c)
            for (int e = n_valid * 8 + m; e < kLtKeys * 8; e += 128) *reinterpret_cast<uint4*>(vb + c * kLtChunk + e * 16) = make_uint4(0u, 0u, 0u, 0u);
          fence_async_smem();
        }
        st_wait();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready + (n & 1));
      }
      const bool any = w.tile_hi > w.tile_lo;
      if (any) {
        mbar_wait(o_full + ((n - 1) & 1), ((n - 1) >> 1) & 1);
        fence_after();
      }
      const int64_t pair = (int64_t)(w.t0 + r) * p.heads + h;
      if (p.n_splits > 1) {
        // sums [pair][split][rank | maximum | denominator], the maximum in natural units.  Two halves add a score's terms in different orders and may follow
        // the maximum at different tiles: theirs are normalised, with the logarithm of the denominator in the maximum
        float* dst = p.part + (pair * p.n_splits + w.split) * (p.rank + 2);
        const bool whole = p.halves == 1;
        const float norm = whole || l <= 0.f ? 1.f : 1.f / l;
        if (alive && w.half == 0) {
          dst[p.rank] = (whole || l <= 0.f ? mu : mu + log2f(l)) * 0.6931471805599453f;
          dst[p.rank + 1] = whole || l <= 0.f ? l : 1.f;
        }
        for (int c = 0; c < written; c += 16) {
          uint32_t o[16];
          if (any) {
            ld16(tmem + lane_off + c, o);
            ld_wait<16>(o);
          }
          if (alive) {
            float2* d2 = reinterpret_cast<float2*>(dst + col0 + c);   // rank + 2 is even: 8-byte aligned rows
#pragma unroll
            for (int j = 0; j < 8; ++j) d2[j] = any ? make_float2(__uint_as_float(o[2 * j]) * norm, __uint_as_float(o[2 * j + 1]) * norm) : make_float2(0.f, 0.f);
          }
        }
      } else {
        float f = 1.f;
        if (p.sink != nullptr && alive) {   // one more term of the denominator
          const float sk = __ldg(p.sink + h) * 1.4426950408889634f, mn = fmaxf(mu, sk);
          f = exp2_fast(mu - mn);
          l = l * f + exp2_fast(sk - mn);
        }
        const float inv = l > 0.f ? f / l : 0.f;
        __nv_bfloat16* dst = p.out + pair * p.rank + col0;
        for (int c = 0; c < written; c += 16) {
          uint32_t o[16], v[8];
          if (any) {
            ld16(tmem + lane_off + c, o);
            ld_wait<16>(o);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = any ? pack_bf16(__uint_as_float(o[2 * j]) * inv, __uint_as_float(o[2 * j + 1]) * inv) : 0u;
          if (alive) store_sector(dst + c, v);   // rank % 16 == 0: whole sectors
        }
      }
      fence_before();
      // all four warps have read O before any of them hands over the next item's first weights (whose product restarts O):
      // the hand-over needs an arrival of every warp
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

struct LtShape {
  int halves, own_stages, rest_stages;
};
// false: a shape whose queries or key tiles do not fit beside each other.  The other chunks of a tile share a
// stage: one wait and one commit a tile, so that a tile's MMAs stand in straight code.
bool lt_shape(int heads, int krow, int rank, LtShape& s) {
  if (heads < 1 || heads > kLtPairs || krow % 16 || rank % 16 || rank < 16 || rank > 512 || rank > krow) return false;
  s.halves = latent_attn_tc_halves(rank);
  const int chunks = (krow + 63) / 64, own = lt_own(rank), rest = chunks - own;
  if (rest > kLtMaxRest) return false;
  const int slots = (kLtSmem - 1024 - kLtTail - rest * kLtQChunk) / kLtChunk;
  for (s.own_stages = kLtMaxStages; s.own_stages >= 2; --s.own_stages)
    if (s.own_stages * own + 2 * rest <= slots) {   // (two of either always fit)
      s.rest_stages = rest ? std::min((slots - s.own_stages * own) / rest, kLtMaxRestStages) : 1;
      return true;
    }
  return false;
}

}  // namespace

bool latent_attn_tc_supported(int heads, int krow, int rank, int block_size) {
  LtShape s;
  return block_size > 0 && block_size % kLtKeys == 0 && lt_shape(heads, krow, rank, s);
}

int latent_attn_tc_rows(int heads) { return std::min(kLtPairs / heads, kRunRows); }   // of an item
int latent_attn_tc_halves(int rank) { return rank > 256 ? 2 : 1; }

// one launch over the step's run list; part given: n_splits CTAs per item leave unnormalised sums (the caller merges)
int latent_attn_tc(const float* q, const __nv_bfloat16* kc, const int32_t* block_table, int bt_stride, const int32_t* row_to_seq,
                   const int32_t* ctx_lens, __nv_bfloat16* out, const int32_t* runs, const int32_t* n_runs, int T, int heads, int krow,
                   int rank, int block_size, float scale, const float* sink, cudaStream_t s, int n_splits, float* part, int window,
                   const LatentShare& share) {
  LtShape sh;
  B200_REQUIRE(latent_attn_tc_supported(heads, krow, rank, block_size) && lt_shape(heads, krow, rank, sh), B200_ERR_UNSUPPORTED,
               "latent_attn_tc: shape %d / %d / %d", heads, krow, rank);
  if (const int e = wait_status()) return e;
  CUtensorMap map;
  const int rc = get_tensor_map_2d(kc, 1ull << 31, krow, krow, kLtKeys, &map);   // rows touched come from the block table
  if (rc) return rc;
  LtParams p = {};
  p.q = q;
  p.block_table = block_table;
  p.row_to_seq = row_to_seq;
  p.ctx_lens = ctx_lens;
  p.runs = runs;
  p.n_runs = n_runs;
  p.sink = sink;
  p.out = out;
  p.part = part;
  p.status = wait_status_word();
  p.n_rows = T;
  p.bt_stride = bt_stride;
  p.heads = heads;
  p.krow = krow;
  p.rank = rank;
  p.block_size = block_size;
  p.n_splits = n_splits;
  p.window = window;
  p.own_stages = sh.own_stages;
  p.rest_stages = sh.rest_stages;
  p.halves = sh.halves;
  p.rows_per_item = latent_attn_tc_rows(heads);
  p.items_per_run = (16 + p.rows_per_item - 1) / p.rows_per_item;
  p.scale = scale;
  p.share = share;
  static bool done[64] = {};
  B200_CUDA(ensure_dynamic_smem(latent_attn_tc_kernel, kLtSmem, done));
  const int64_t most = (int64_t)T * p.items_per_run * n_splits * sh.halves;   // upper bound; the kernel reads the real count
  B200_CUDA(launch(latent_attn_tc_kernel, dim3((unsigned)std::min<int64_t>(most, kNumSMs)), dim3(kLtThreads), (size_t)kLtSmem, s, map, p));
  return B200_OK;
}

}  // namespace b200
