// Paged causal grouped-query attention on tcgen05 for steps with runs of rows, key and value heads of 64 or 128 entries.
//
// The (row, head) pairs of one kv head fill the MMA's M dimension.  A work item is up to two tiles of 128 pairs (consecutive rows of one
// sequence times the G heads of a kv head) that share every key and value tile of 64 keys:
//   S_x[128][64] = Q_x . K_tile^T        O_x[128][vdim] += P_x . V_tile           x = the item's first, second tile of pairs
// The scores of key tile n + 1 are issued before the weights of tile n are waited for (two score buffers per tile of pairs), so the
// softmax of either tile never waits for the tensor core once the walk is under way: with one tile of pairs and 128 keys (the kernel
// this one replaces) S -> softmax -> P V was one dependent chain of 1.85 us (2 048 rows 212 us), and with two tiles of pairs but single score
// buffers of 128 keys a tile's softmax and its own products still came one after the other (177 us; two buffers of 64 keys 118).
// The weights overwrite the scores in TMEM (A operand of the second product): per 32 scores 16 columns of bf16 pairs and 16 more with what
// rounding took from them (P has 16 bits, as attn_tc.cu has it).  TMEM per tile of pairs: two score buffers of 64
// columns, O 128.
// Scores may be capped, biased by distance (each score takes its own distance's bias and no other: tables may end in -inf or any sentinel),
// windowed with kept first keys (EX); outputs may have a sink in the denominator and a gate per head.  The running maximum is only followed when it rises by more than 2^8 (exact: all terms are scaled alike); a warp then
// rescales its 32 rows of O in TMEM.
// Bound by the tensor core or the softmax's issue slots: 2 048 rows at contexts 1001..3048, 32 heads over 8: 117 us among other calls (119 with branches between
// the issuing warp's MMAs and the maximum of a key tile in one chain, 211 on the kernel before); 1 900
// rows of three sequences, 16 heads over 4, capped, biased, window 1024: 74 us (278 us on the mma.sync kernel of attn_latent.cu).
// Warps: four softmax warps per tile (a thread owns a pair), TMA, MMA, two that stage queries.  Every wait is bounded and
// reported (tc.cuh).
#include <algorithm>
#include <type_traits>

#include "runs.cuh"
#include "tc.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int kArKeys = 64, kArThreads = 384;
constexpr int kArQChunk = 128 * 128;           // [128 pairs][64 columns] bf16: 16 KiB
constexpr int kArChunk = kArKeys * 128;        // [64 keys][64 columns] bf16: 8 KiB
constexpr int kArTile = 2 * kArChunk;
// key and value tiles in turn; EX gives one of them to the table of score biases of an item's heads
__host__ __device__ constexpr int ar_slots(bool ex) { return ex ? 8 : 9; }
constexpr int kArBiasFloats = kArTile / 4, kArBiasPad = 96;   // entries in front (masked keys) and behind (far keys) of a head's, see fill_bias
constexpr int kArStage = 8 * 2048;             // output staging: 2 KiB per softmax warp
constexpr int kArTable = 32;                   // items of a CTA whose description is worked out ahead
constexpr int kArSmem = 232448;
static_assert(1024 + 4 * kArQChunk + 9 * kArTile + kArStage + (2 * 9 + 16) * 8 + 16 + kArTable * 40 <= kArSmem, "shared memory");

struct RowsItem {
  int row0, nrows, seq, ctx_max;   // attn_prefill.cu's plan
};

struct RowsParams {
  const void* q;
  int64_t ldq;                 // elements between rows of q
  const int32_t* block_table;
  const int32_t* row_to_seq;
  const int32_t* ctx_lens;
  const int32_t* runs;         // (first row, rows) pairs whose contexts rise by one, or
  const int32_t* n_runs;
  const RowsItem* plan;          // runs of one sequence with their longest context; plan[0].row0 of them from plan[1]
  const float* sink;
  __nv_bfloat16* out;
  int64_t ldo;
  float* part;
  uint32_t* status;
  int n_rows, bt_stride, heads, kv_heads, dim, vdim, block_size, n_splits, window, tile_rows, parts;   // parts: items that a run is cut into
  float scale;
  RunShare share;
  AttnExtra ex;
};

struct RowsWork {
  int row0, nrows, seq, kvh, split, lead, tile0, lo, hi, ctx_max;   // walk [lo, hi): key tile w < lead ? w : w - lead + tile0
};

__device__ __forceinline__ int ar_tile(const RowsWork& w, int i) { return i < w.lead ? i : i - w.lead + w.tile0; }

// item `it`: (run, part, kv head, split), the longest contexts (the last runs) first; false: nothing there, or not this kernel's (short_pairs)
__device__ __forceinline__ bool ar_work(const RowsParams& p, int n_runs, int short_pairs, int it, RowsWork& w) {
  w.split = it % p.n_splits;
  it /= p.n_splits;
  w.kvh = it % p.kv_heads;
  it /= p.kv_heads;
  const int run = n_runs - 1 - it / p.parts, row = (p.parts - 1 - it % p.parts) * p.tile_rows;
  w.tile0 = w.lead = 0;
  if (p.plan) {
    const RowsItem* r = p.plan + 1 + run;
    w.row0 = __ldg(&r->row0);
    w.nrows = __ldg(&r->nrows);
    w.seq = __ldg(&r->seq);
    w.ctx_max = __ldg(&r->ctx_max);
  } else {
    w.row0 = __ldg(p.runs + 2 * run);
    const int length = __ldg(p.runs + 2 * run + 1);
    if (short_pairs && run_is_short(short_pairs, length, p.heads / p.kv_heads)) return false;
    w.row0 += row;
    w.nrows = (length & kRunLength) - row;
    if (w.nrows <= 0) return false;
    if (p.parts > 1) w.nrows = min(w.nrows, p.tile_rows);
    w.seq = p.row_to_seq ? __ldg(p.row_to_seq + w.row0) : w.row0;
    w.ctx_max = __ldg(p.ctx_lens + w.row0 + w.nrows - 1);
    if (p.window > 0) {
      w.tile0 = max(__ldg(p.ctx_lens + w.row0) - p.window, 0) / kArKeys;
      w.lead = min((p.ex.keep_first + kArKeys - 1) / kArKeys, w.tile0);
    }
  }
  const int tiles = max((w.ctx_max + kArKeys - 1) / kArKeys - w.tile0, 0) + w.lead, per = (tiles + p.n_splits - 1) / p.n_splits;
  w.lo = min(tiles, w.split * per);
  w.hi = min(tiles, (w.split + 1) * per);
  return true;
}

template <typename QT> __device__ __forceinline__ uint4 ar_q8(const QT* p);   // eight query entries as bf16
template <> __device__ __forceinline__ uint4 ar_q8<__nv_bfloat16>(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
template <> __device__ __forceinline__ uint4 ar_q8<float>(const float* p) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}

template <typename QT, bool EX>
__global__ void __launch_bounds__(kArThreads, 1)
attn_rows_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const RowsParams p) {
  constexpr int kArSlots = ar_slots(EX);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* qs = smem;                        // two tiles of [2][128 pairs][64]
  unsigned char* ring = qs + 4 * kArQChunk;        // [kArSlots][2][64 keys][64]
  float* bias_tab = reinterpret_cast<float*>(ring + kArSlots * kArTile);   // EX only
  unsigned char* ostage = ring + 9 * kArTile;
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(ostage + kArStage);
  uint64_t* kv_free = kv_full + kArSlots;
  uint64_t* s_full = kv_free + kArSlots;           // [tile of pairs][2] scores of an even / odd key tile are there
  uint64_t* p_ready = s_full + 4;                  // [tile of pairs][2] its weights are
  uint64_t* o_full = p_ready + 4;                  // [tile of pairs][2] its second product has finished
  uint64_t* q_ready = o_full + 4;
  uint64_t* q_first = q_ready + 1;                 // the CTA's first queries, staged by the softmax warps as well
  uint64_t* q_free = q_first + 1;
  uint64_t* last = q_free + 1;                     // the MMAs in flight when a wait ran out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(last + 1);   // and, behind it, the mark of a wait that ran out
  const Waits mbar_wait(tmem_slot + 1, p.status);
  int* n_table = reinterpret_cast<int*>(tmem_slot + 2);   // entries of the table; the first round of items behind it
  RowsWork* table = reinterpret_cast<RowsWork*>(n_table + 2);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kArSlots; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_free + s, 1);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(s_full + s, 1);
      mbar_init(p_ready + s, 4);
      mbar_init(o_full + s, 1);
    }
    mbar_init(q_ready, 2);
    mbar_init(q_first, 10);
    mbar_init(q_free, 1);
    mbar_init(last, 1);
    tmem_slot[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();
  pdl_launch_dependents();
  if (p.share.ticket && blockIdx.x == 0 && threadIdx.x == 0) *p.share.ticket = 0;
  const int n_runs = p.plan ? p.plan[0].row0 : *p.n_runs, short_pairs = p.share.n_runs ? run_share(p.share, p.heads / p.kv_heads) : 0;
  const int n_items = short_pairs == kRunsAll || (short_pairs && n_runs == p.n_rows) ? 0 : n_runs * p.parts * p.kv_heads * p.n_splits;
  if (n_items == 0) return;   // a step of runs that are all the other kernel's
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  const int G = p.heads / p.kv_heads, R = p.tile_rows;
  // every other round backwards: the CTA that had the longest item of one gets the shortest of the next
  const int grid = gridDim.x, cta = blockIdx.x;
  auto item_of = [&](int round) { return round * grid + ((round & 1) ? grid - 1 - cta : cta); };
  // the descriptions hang on a chain of loads (run, sequence, contexts): a round to a lane, until the table is full, for every role
  if (warp == 10) {
    int filled = 0, round = 0;
    while (filled < kArTable && round * grid < n_items) {
      RowsWork w;
      const int it = item_of(round + lane);
      const bool have = it < n_items && ar_work(p, n_runs, short_pairs, it, w);
      const unsigned all = __ballot_sync(0xffffffffu, have);
      const int at = filled + __popc(all & ((1u << lane) - 1u));
      if (have && at < kArTable) table[at] = w;
      const unsigned late = __ballot_sync(0xffffffffu, have && at >= kArTable);   // beyond the table: their rounds come again
      filled = min(filled + __popc(all), kArTable);
      round += late ? __ffs(late) - 1 : 32;
    }
    if (lane == 0) n_table[0] = filled, n_table[1] = round;
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;   // per tile of pairs 256 columns: scores of even, odd key tiles, O
  const int n_tab = n_table[0], tab_round = n_table[1];
  // a role's next item (k: its count of calls so far); false: there is none
  auto next_work = [&](int& k, RowsWork& w) {
    if (k < n_tab) {
      w = table[k++];
      return true;
    }
    for (;;) {
      const int round = tab_round + k - n_tab;
      if (round * grid >= n_items) return false;
      ++k;
      if (item_of(round) < n_items && ar_work(p, n_runs, short_pairs, item_of(round), w)) return true;
    }
  };
  // the two A operands of an item, thread i of `threads`: 16-byte pieces of rows
  auto stage_q = [&](const RowsWork& w, int i, int threads) {
    const QT* q0 = static_cast<const QT*>(p.q) + (int64_t)w.row0 * p.ldq + (int64_t)w.kvh * G * p.dim;
    const int pieces = (w.nrows > R ? 2 : 1) * 128 * 16;
    constexpr int U = 8;
#pragma unroll 1
    for (int e0 = i; e0 < pieces; e0 += U * threads) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * threads, m = e >> 4, chunk = e & 15, r = (m & 127) / G, g = (m & 127) % G, row = (m >> 7) * R + r;
        v[u] = make_uint4(0u, 0u, 0u, 0u);
        if (e < pieces && r < R && row < w.nrows && chunk * 8 < p.dim) v[u] = ar_q8<QT>(q0 + (int64_t)row * p.ldq + g * p.dim + chunk * 8);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * threads, m = e >> 4, chunk = e & 15, mm = m & 127;
        if (e < pieces)
          *reinterpret_cast<uint4*>(qs + (2 * (m >> 7) + (chunk >> 3)) * kArQChunk + (mm >> 3) * 1024 + (mm & 7) * 128 + (((chunk & 7) ^ (mm & 7)) << 4)) = v[u];
      }
    }
    fence_async_smem();
    __syncwarp();
  };

  if (warp == 8) {
    // ===== TMA: key tile, value tile, key tile, ... =====
    const bool issuer = elect_one();
    if (issuer) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    }
    const int kc = (p.dim + 63) >> 6, vc = (p.vdim + 63) >> 6;
    int slot = 0;
    uint32_t ph = 1;
    bool stop = false;
    RowsWork w;
    for (int k = 0; !stop && next_work(k, w);) {
      const int32_t* bt = p.block_table + (int64_t)w.seq * p.bt_stride;
      for (int i = w.lo; i < w.hi && !(stop = mbar_wait.stop()); ++i) {
        const int tok = ar_tile(w, i) * kArKeys;
        const int blk = __shfl_sync(0xffffffffu, __ldg(bt + tok / p.block_size), 0);
        const int row = (blk * p.kv_heads + w.kvh) * p.block_size + tok % p.block_size;
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          mbar_wait(kv_free + slot, ph);
          if (issuer) {
            unsigned char* dst = ring + slot * kArTile;
            const int nc = kv ? vc : kc;
            mbar_expect_tx(kv_full + slot, nc * kArChunk);
            for (int c = 0; c < nc; ++c) tma_load_2d(dst + c * kArChunk, kv ? &map_v : &map_k, c * 64, row, kv_full + slot);
          }
          __syncwarp();
          if (++slot == kArSlots) slot = 0, ph ^= 1;
        }
      }
    }
    if (mbar_wait.stop())   // the loads in flight: a slot's last one filled it in this round of the ring or in the one before
      for (int s = 0; s < kArSlots; ++s) mbar_wait.drain(kv_full + s, s < slot ? ph ^ 1 : ph);
  } else if (warp == 9) {
    // ===== MMA: per key tile, for either tile of pairs: the next key tile's scores, then this one's second product.  The whole warp
    // walks the loop; bounds and addresses that come from memory are broadcast, so that they are uniform to the compiler =====
    const uint32_t one = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t desc_q = make_desc(smem_u32(qs), 16, 1024), desc_k = make_desc(smem_u32(ring), 16, 1024),
                   desc_v = make_desc(smem_u32(ring), kArChunk, 1024);
    const uint32_t id_s = idesc_bf16(kArKeys, 0), id_o = idesc_bf16(p.vdim, 1);
    const int ksteps = p.dim >> 4;
    int slot = 0, active = 0, n[2] = {0, 0};   // n: key tiles walked by either tile of pairs so far
    uint32_t ph = 0;
    auto next_slot = [&]() {
      if (++slot == kArSlots) slot = 0, ph ^= 1;
    };
    // an item of nt key tiles: straight code for either count of pair tiles and for the widest heads (branches between the MMAs cost the issuing warp)
    auto walk = [&](auto tiles_c, auto steps_c, int nt) {
      constexpr int TILES = decltype(tiles_c)::value, STEPS = decltype(steps_c)::value;
      auto scores = [&](int x, int nx, int k_slot) {
        const uint64_t da = desc_q + (uint64_t)((x * 2 * kArQChunk) >> 4), db = desc_k + (uint64_t)((k_slot * kArTile) >> 4);
        const uint32_t d = tm + x * 256 + (nx & 1) * kArKeys;
        if constexpr (STEPS > 0) {
#pragma unroll
          for (int j = 0; j < STEPS; ++j)
            mma_ss(one, d, da + ((j >> 2) * kArQChunk + (j & 3) * 32) / 16, db + ((j >> 2) * kArChunk + (j & 3) * 32) / 16, id_s, j ? 1u : 0u);
        } else {
          for (int j = 0; j < ksteps; ++j)
            mma_ss(one, d, da + ((j >> 2) * kArQChunk + (j & 3) * 32) / 16, db + ((j >> 2) * kArChunk + (j & 3) * 32) / 16, id_s, j ? 1u : 0u);
        }
        commit(one, s_full + 2 * x + (nx & 1));
      };
      mbar_wait(kv_full + slot, ph);
      fence_after();
      int k_slot = slot;
      next_slot();
#pragma unroll
      for (int x = 0; x < TILES; ++x) scores(x, n[x], k_slot);
      commit(one, kv_free + k_slot);
      commit(nt == 1 ? one : 0u, q_free);
      auto step = [&](auto more_c, int i) {
        constexpr bool MORE = decltype(more_c)::value;
        const int v_slot = slot;
        const uint32_t v_ph = ph;
        next_slot();
        if constexpr (MORE) {
          mbar_wait(kv_full + slot, ph);
          fence_after();
          k_slot = slot;
          next_slot();
        }
        const uint64_t dv = desc_v + (uint64_t)((v_slot * kArTile) >> 4);
#pragma unroll
        for (int x = 0; x < TILES; ++x) {
          if constexpr (MORE) scores(x, n[x] + 1, k_slot);
          if (MORE && x == TILES - 1) {
            commit(one, kv_free + k_slot);
            commit(i + 2 == nt ? one : 0u, q_free);   // the item's last scores are on their way
          }
          if (x == 0) mbar_wait(kv_full + v_slot, v_ph);
          mbar_wait(p_ready + 2 * x + (n[x] & 1), (n[x] >> 1) & 1);
          fence_after();
          const uint32_t pa = tm + x * 256 + (n[x] & 1) * kArKeys, d = tm + x * 256 + 128;
#pragma unroll
          for (int j = 0; j < 4; ++j) {   // 16 keys per step: 8 columns of weights, 16 further those of the second term
            mma_ts(one, d, pa + (j >> 1) * 32 + (j & 1) * 8, dv + (uint64_t)((j * 2048) >> 4), id_o, (i | j) ? 1u : 0u);
            mma_ts(one, d, pa + (j >> 1) * 32 + (j & 1) * 8 + 16, dv + (uint64_t)((j * 2048) >> 4), id_o, 1u);
          }
          if (x == TILES - 1) commit(one, kv_free + v_slot);
          commit(one, o_full + 2 * x + (n[x] & 1));
          ++n[x];
        }
      };
      for (int i = 0; i + 1 < nt; ++i) step(std::true_type(), i);
      step(std::false_type(), nt - 1);
    };
    RowsWork w;
    for (int k = 0; __shfl_sync(0xffffffffu, next_work(k, w), 0);) {
      const int nt = __shfl_sync(0xffffffffu, w.hi - w.lo, 0), tiles = __shfl_sync(0xffffffffu, w.nrows > R ? 2 : 1, 0);
      if (nt <= 0) continue;
      if (active == 0) mbar_wait(q_first, 0);
      else mbar_wait(q_ready, (active - 1) & 1);
      if (tiles == 2) {
        if (ksteps == 8) walk(std::integral_constant<int, 2>(), std::integral_constant<int, 8>(), nt);
        else walk(std::integral_constant<int, 2>(), std::integral_constant<int, 0>(), nt);
      } else {
        if (ksteps == 8) walk(std::integral_constant<int, 1>(), std::integral_constant<int, 8>(), nt);
        else walk(std::integral_constant<int, 1>(), std::integral_constant<int, 0>(), nt);
      }
      ++active;
    }
    if (mbar_wait.stop()) {
      commit(one, last);
      mbar_wait.drain(last, 0);
    }
  } else if (warp >= 10) {
    // ===== queries of the next item -> the two A operands =====
    int active = 0;
    RowsWork w;
    for (int k = 0; next_work(k, w);) {
      if (w.hi <= w.lo) continue;
      if (active == 0) {
        stage_q(w, threadIdx.x - 64, 320);   // (beside the softmax warps' threads 0..255)
        if (lane == 0) mbar_arrive(q_first);
      } else {
        mbar_wait(q_free, (active - 1) & 1);
        stage_q(w, threadIdx.x - 320, 64);
        if (lane == 0) mbar_arrive(q_ready);
      }
      ++active;
    }
  } else {
    // ===== softmax and output: a thread owns a pair of tile x =====
    const int x = warp >> 2, quad = warp & 3, m = quad * 32 + lane;
    const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + x * 256;
    const int r = m / G, g = m % G, row = x * R + r;
    constexpr float kLog2e = 1.4426950408889634f;
    const float sc2 = p.scale * kLog2e;   // scores in the log2 domain
    const float cap2 = EX ? p.ex.softcap * kLog2e : 0.f, cap_in = EX && p.ex.softcap > 0.f ? 2.0f * sc2 / p.ex.softcap : 0.f;
    // bias in the log2 domain; a finite sentinel stays finite (a row that sees nothing but sentinels averages, as exp would have it)
    auto bias2 = [&](float b) {
      const float v = b * kLog2e;
      return isinf(v) ? b : v;
    };
    // the item's heads' biases by distance; in front zeros (masked keys), behind the farthest distance's, so that a tile that holds some
    // near key indexes it without clamping each distance
    const int bias_row = p.ex.bias_dist + 2 * kArBiasPad + 8;
    const bool tab = EX && p.ex.dist_bias != nullptr && G * bias_row <= kArBiasFloats;
    auto fill_bias = [&](int kvh) {
      asm volatile("bar.sync 2, 256;" ::: "memory");
      for (int e = threadIdx.x; e < G * bias_row; e += 256) {
        const int gg = e / bias_row, d = e % bias_row - kArBiasPad;
        bias_tab[e] = d >= 0 ? bias2(__ldg(p.ex.dist_bias + (int64_t)(kvh * G + gg) * p.ex.bias_dist + min(d, p.ex.bias_dist - 1))) : 0.f;
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
    };
    bool first = true;
    int n = 0, slot = 0;
    uint32_t ph = 0;   // slot, ph: the ring's position (the key tile of the walk), for the value tile that is cleaned
    RowsWork w;
    for (int k = 0; next_work(k, w);) {
      if (first && w.hi > w.lo) {
        stage_q(w, threadIdx.x, 320);   // (the stagers are threads 256..319 of this)
        if (lane == 0) mbar_arrive(q_first);
        first = false;
      }
      if (tab) fill_bias(w.kvh);
      if (x == 1 && w.nrows <= R) continue;   // the item has one tile of pairs (only tile 0 cleans value tiles)
      const bool alive = r < R && row < w.nrows;
      const int t = w.row0 + row, ctx = alive ? __ldg(p.ctx_lens + t) : 0, lo = p.window > 0 ? max(ctx - p.window, 0) : 0;
      const int h = w.kvh * G + g, keep = EX ? p.ex.keep_first : 0;
      const float* brow = EX && p.ex.dist_bias && alive ? p.ex.dist_bias + (int64_t)h * p.ex.bias_dist : nullptr;
      const float far_bias = EX && brow ? bias2(__ldg(brow + p.ex.bias_dist - 1)) : 0.f;
      float mu = -INFINITY, l = 0.f;
      for (int i = w.lo; i < w.hi; ++i, ++n) {
        const int k0 = ar_tile(w, i) * kArKeys, j_lo = lo - k0, j_hi = ctx - k0;   // live columns [j_lo, j_hi), and those below keep
        mbar_wait(s_full + 2 * x + (n & 1), (n >> 1) & 1);
        fence_after();
        const uint32_t s_addr = base + (n & 1) * kArKeys;
        uint32_t s[64];
        ld32(s_addr, s);
        ld32(s_addr + 32, s + 32);
        ld_wait<64>(s);
        if constexpr (EX) {   // scaled, capped, biased, in the log2 domain
          // a tile of far keys alone takes the last distance's bias with the scaling, one that holds nearer keys each key's own after it
          const bool near = __any_sync(0xffffffffu, brow != nullptr && ctx - 1 - (k0 + kArKeys - 1) < p.ex.bias_dist - 1);
          const float add = near ? 0.f : far_bias;
          if (p.ex.softcap > 0.f) {
            // cap tanh(v / cap) = cap - 2 cap / (1 + e^(2 v / cap)) on the hardware's exponential and reciprocal
            const float top = cap2 + add;
#pragma unroll
            for (int j = 0; j < 64; ++j) {
              float rc;
              asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(1.0f + exp2_fast(__uint_as_float(s[j]) * cap_in)));
              s[j] = __float_as_uint(fmaf(-2.0f * cap2, rc, top));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 64; ++j) s[j] = __float_as_uint(fmaf(__uint_as_float(s[j]), sc2, add));
          }
          if (near && brow) {
            const int d0 = ctx - 1 - k0;
            if (tab) {
              // below -1 every key is masked, from the last distance + 64 on every key is far: the padding covers what lies between
              const float* b = bias_tab + g * bias_row + kArBiasPad + min(max(d0, -1), p.ex.bias_dist + 95);
#pragma unroll
              for (int j = 0; j < 64; ++j) s[j] = __float_as_uint(__uint_as_float(s[j]) + b[-j]);
            } else {
#pragma unroll
              for (int j = 0; j < 64; ++j)
                s[j] = __float_as_uint(__uint_as_float(s[j]) + bias2(__ldg(brow + min(max(d0 - j, 0), p.ex.bias_dist - 1))));
            }
          }
        }
        if (__any_sync(0xffffffffu, (j_lo > 0 && !(EX && k0 + kArKeys <= keep)) || j_hi < kArKeys)) {
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (j >= j_hi || (j < j_lo && !(EX && k0 + j < keep))) s[j] = 0xff800000u;   // -inf
        }
        float mx = max64(s);
        if (!EX) mx *= sc2;
        const bool jump = mx > mu + 8.f;   // also the first live key (mu = -inf)
        if (__any_sync(0xffffffffu, jump)) {
          const float mn = jump ? mx : mu, f = jump && mu != -INFINITY ? exp2_fast(mu - mn) : 1.f;
          if (i > w.lo && __any_sync(0xffffffffu, f != 1.f)) {
            mbar_wait(o_full + 2 * x + ((n - 1) & 1), ((n - 1) >> 1) & 1);
            fence_after();
            for (int c = 0; c < p.vdim; c += 16) {
              uint32_t o[16];
              ld16(base + 128 + c, o);
              ld_wait<16>(o);
#pragma unroll
              for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
              st16(base + 128 + c, o);
            }
          }
          l *= f;
          mu = mn;
        }
        const float mref = mu > -INFINITY ? mu : 0.f;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[32];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float s0 = __uint_as_float(s[c * 32 + 2 * j]), s1 = __uint_as_float(s[c * 32 + 2 * j + 1]);
            const float p0 = exp2_fast(EX ? s0 - mref : fmaf(s0, sc2, -mref)), p1 = exp2_fast(EX ? s1 - mref : fmaf(s1, sc2, -mref));
            // the high term truncated, the rest rounded
            sum[j & 3] += p0 + p1;
            const uint32_t h0 = __float_as_uint(p0) & 0xffff0000u, h1 = __float_as_uint(p1) & 0xffff0000u;
            pk[j] = __byte_perm(h0, h1, 0x7632);
            pk[16 + j] = pack_bf16(p0 - __uint_as_float(h0), p1 - __uint_as_float(h1));
          }
          st32(s_addr + c * 32, pk);
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        if (x == 0) {
          const int n_valid = w.ctx_max - k0;
          if (n_valid < kArKeys) {
            // value rows past the context may hold anything, and 0 * NaN = NaN: zero them under their zero weights
            const int vs = slot + 1 == kArSlots ? 0 : slot + 1;
            mbar_wait(kv_full + vs, ph ^ (vs == 0 ? 1 : 0));
            unsigned char* vb = ring + vs * kArTile;
            for (int c = 0; c < (p.vdim + 63) >> 6; ++c)
              for (int e = n_valid * 8 + m; e < kArKeys * 8; e += 128) *reinterpret_cast<uint4*>(vb + c * kArChunk + e * 16) = make_uint4(0u, 0u, 0u, 0u);
            fence_async_smem();
          }
          slot += 2;
          if (slot >= kArSlots) slot -= kArSlots, ph ^= 1;
        }
        st_wait();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready + 2 * x + (n & 1));
      }
      const bool any = w.hi > w.lo;
      if (any) {
        mbar_wait(o_full + 2 * x + ((n - 1) & 1), ((n - 1) >> 1) & 1);
        fence_after();
      }
      if (p.n_splits > 1) {
        // unnormalised sums [pair][split][vdim | maximum | denominator], the maximum in natural units
        float* dst = p.part + (((int64_t)t * p.heads + h) * p.n_splits + w.split) * (p.vdim + 2);
        if (alive) {
          dst[p.vdim] = mu * 0.6931471805599453f;
          dst[p.vdim + 1] = l;
        }
        for (int c = 0; c < p.vdim; c += 16) {
          uint32_t o[16];
          if (any) {
            ld16(base + 128 + c, o);
            ld_wait<16>(o);
          }
          if (alive) {
            float2* d2 = reinterpret_cast<float2*>(dst + c);
#pragma unroll
            for (int j = 0; j < 8; ++j) d2[j] = any ? make_float2(__uint_as_float(o[2 * j]), __uint_as_float(o[2 * j + 1])) : make_float2(0.f, 0.f);
          }
        }
      } else {
        float f = 1.f;
        if (p.sink != nullptr && alive) {   // one more term of the denominator
          const float sk = __ldg(p.sink + h) * kLog2e, mn = fmaxf(mu, sk);
          f = exp2_fast(mu - mn);
          l = l * f + exp2_fast(sk - mn);
        }
        float inv = l > 0.f ? f / l : 0.f;
        if (EX && p.ex.gate && alive) inv /= 1.0f + expf(-__bfloat162float(static_cast<const __nv_bfloat16*>(p.ex.gate)[(int64_t)t * p.ex.ldg + h]));
        // 32 columns at a time through shared memory: a row's 64 bytes leave from four neighbouring lanes (a lane per row touches 32 lines
        // with every store: 4.6 us an item)
        unsigned char* st = ostage + warp * 2048;
        for (int c = 0; c < p.vdim; c += 32) {
          uint32_t o[32];
          if (any) {
            ld32(base + 128 + c, o);
            ld_wait<32>(o);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint32_t v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = any ? pack_bf16(__uint_as_float(o[8 * k + 2 * j]) * inv, __uint_as_float(o[8 * k + 2 * j + 1]) * inv) : 0u;
            *reinterpret_cast<uint4*>(st + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int rr = k * 8 + (lane >> 2), mm = quad * 32 + rr, row2 = x * R + mm / G, col = c + (lane & 3) * 8;
            const uint4 v = *reinterpret_cast<const uint4*>(st + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
            if (mm / G < R && row2 < w.nrows && col < p.vdim)
              *reinterpret_cast<uint4*>(p.out + (int64_t)(w.row0 + row2) * p.ldo + (int64_t)(w.kvh * G + mm % G) * p.vdim + col) = v;
          }
          __syncwarp();
        }
      }
      fence_before();
      // all four warps of a tile have read its O before any of them hands over the next item's first weights (whose product restarts O)
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 9) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

template <typename QT, bool EX>
int ar_launch(const CUtensorMap& mk, const CUtensorMap& mv, const RowsParams& p, int T, cudaStream_t s) {
  if (const int e = wait_status()) return e;
  static bool done[64] = {};
  B200_CUDA(ensure_dynamic_smem(attn_rows_tc_kernel<QT, EX>, kArSmem, done));
  const int64_t most = (int64_t)T * p.kv_heads * p.n_splits;   // upper bound; the kernel reads the real count
  B200_CUDA(launch(attn_rows_tc_kernel<QT, EX>, dim3((unsigned)std::min<int64_t>(most, kNumSMs)), dim3(kArThreads), (size_t)kArSmem, s, mk, mv, p));
  return B200_OK;
}

}  // namespace

// rows of an item: twice what 128 pairs hold; once, where a step of two-tile items would leave half of the SMs without one (64 rows at
// contexts 1001..1064, 32 heads over 8: 31 us with one tile an item, 38 with two)
int attn_rows_tc_rows(int T, int heads, int kv_heads) {
  const int tile = 128 / (heads / kv_heads);
  return (int64_t)T * kv_heads < (int64_t)tile * kNumSMs ? tile : 2 * tile;
}

static bool ar_form(int heads, int kv_heads, int dim, int vdim, int block_size) {
  return heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && heads / kv_heads <= 16 && dim % 16 == 0 && dim >= 16 && dim <= 128 && vdim % 16 == 0 &&
         vdim >= 16 && vdim <= 128 && block_size > 0 && block_size % 64 == 0;
}
// Rows of keys and values are whole boxes of 64 columns.  Two runs over narrower value rows (400 and 420 rows of one sequence, 6 heads over 2, keys of 64, values
// of 32, of which a box takes 64) ended in an illegal address, each behind some hundred other tests; alone the same call passes, and reading has not shown which access
// it was.  Such heads take the mma.sync kernel of attn_latent.cu, which reads their rows through pointers, with weights of 16 bits as here (1 900 rows of three
// sequences, 16 heads of 96 over 4, window 1024: 272 us; heads of 128 here 74).
bool attn_rows_tc_supported(int heads, int kv_heads, int dim, int vdim, int block_size) {
  return ar_form(heads, kv_heads, dim, vdim, block_size) && dim % 64 == 0 && vdim % 64 == 0;
}
bool attn_rows_tc_declined(int heads, int kv_heads, int dim, int vdim, int block_size) {
  return ar_form(heads, kv_heads, dim, vdim, block_size) && !(dim % 64 == 0 && vdim % 64 == 0);
}

// bf16 queries in rows of ldq, weights of 16 bits; plan: attn_prefill.cu's items of at most attn_rows_tc_rows rows
int attn_rows_tc_plan(const __nv_bfloat16* q, int64_t ldq, const __nv_bfloat16* kc, const __nv_bfloat16* vc, const int32_t* block_table, int bt_stride,
                      const int32_t* ctx_lens, __nv_bfloat16* out, int64_t ldo, int T, int heads, int kv_heads, int dim, int block_size, float scale,
                      const void* plan, cudaStream_t s) {
  CUtensorMap mk, mv;
  int rc = get_tensor_map_2d(kc, 1ull << 31, dim, dim, 64, &mk);   // rows touched come from the block table
  if (rc) return rc;
  rc = get_tensor_map_2d(vc, 1ull << 31, dim, dim, 64, &mv);
  if (rc) return rc;
  RowsParams p = {};
  p.q = q;
  p.ldq = ldq;
  p.block_table = block_table;
  p.ctx_lens = ctx_lens;
  p.plan = static_cast<const RowsItem*>(plan);
  p.out = out;
  p.ldo = ldo;
  p.bt_stride = bt_stride;
  p.heads = heads;
  p.kv_heads = kv_heads;
  p.dim = p.vdim = dim;
  p.block_size = block_size;
  p.n_splits = p.parts = 1;
  p.status = wait_status_word();
  p.tile_rows = 128 / (heads / kv_heads);
  p.scale = scale;
  return ar_launch<__nv_bfloat16, false>(mk, mv, p, T, s);
}

// fp32 queries [T][heads][dim], weights of 16 bits; runs, n_runs: the first of the lists that paged_attn_runs_plan leaves for T rows.  Launched
// beside the mma.sync kernel, which takes share's runs.
int attn_rows_tc_runs(const float* q, const __nv_bfloat16* kc, const __nv_bfloat16* vc, const int32_t* block_table, int bt_stride,
                      const int32_t* row_to_seq, const int32_t* ctx_lens, __nv_bfloat16* out, const int32_t* runs, const int32_t* n_runs, int T,
                      int heads, int kv_heads, int dim, int vdim, int block_size, float scale, const float* sink, cudaStream_t s, int n_splits,
                      float* part, int window, const AttnExtra& ex, RunShare* share) {
  CUtensorMap mk, mv;
  int rc = get_tensor_map_2d(kc, 1ull << 31, dim, dim, 64, &mk);
  if (rc) return rc;
  rc = get_tensor_map_2d(vc, 1ull << 31, vdim, vdim, 64, &mv);
  if (rc) return rc;
  // the longest runs whose pairs fit an item: two tiles of 8 << list rows, or one, as attn_rows_tc_rows has it (200 rows in runs of 12, 16 heads
  // over one, contexts 300 to 600: 49.5 us, with two 58; 300 rows of one sequence, 16 over 4: 49 and 60)
  int list = 0;
  while (list + 1 < kRunLists && (16 << (list + 1)) <= 2 * (128 / (heads / kv_heads))) ++list;
  const int tile_rows = 8 << list;
  const bool one = (int64_t)T * kv_heads < (int64_t)tile_rows * kNumSMs;
  if (one && list > 0) --list;
  RowsParams p = {};
  p.q = q;
  p.ldq = (int64_t)heads * dim;
  p.block_table = block_table;
  p.row_to_seq = row_to_seq;
  p.ctx_lens = ctx_lens;
  p.runs = runs + (int64_t)2 * T * list;
  p.n_runs = n_runs + list;
  p.n_rows = T;
  p.sink = sink;
  p.out = out;
  p.ldo = (int64_t)heads * vdim;
  p.part = part;
  p.status = wait_status_word();
  p.bt_stride = bt_stride;
  p.heads = heads;
  p.kv_heads = kv_heads;
  p.dim = dim;
  p.vdim = vdim;
  p.block_size = block_size;
  p.n_splits = n_splits;
  p.window = window;
  p.tile_rows = tile_rows;
  p.parts = one && (kRunRows << list) > tile_rows ? 2 : 1;   // (no list of runs of 8 rows)
  *share = p.share = {p.n_runs, const_cast<int32_t*>(n_runs) + kRunTicket, T, kv_heads * n_splits, p.parts};
  p.scale = scale;
  p.ex = ex;
  return ex.any() ? ar_launch<float, true>(mk, mv, p, T, s) : ar_launch<float, false>(mk, mv, p, T, s);
}

}  // namespace b200

// debug helper (not in the public header): heads of this form in long steps: 1 on this kernel, 2 on the mma.sync one with weights of 16 bits
extern "C" __attribute__((visibility("default"))) int b200_debug_attn_rows_tc(int32_t heads, int32_t kv_heads, int32_t dim, int32_t vdim, int32_t block_size) {
  return b200::attn_rows_tc_supported(heads, kv_heads, dim, vdim, block_size) ? 1 : b200::attn_rows_tc_declined(heads, kv_heads, dim, vdim, block_size) ? 2 : 0;
}
