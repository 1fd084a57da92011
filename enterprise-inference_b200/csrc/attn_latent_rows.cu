// Latent attention (attn_latent.cu) of decode rows on tcgen05: one row's heads, up to 16 of them, are the MMA's N, the keys of a tile its M.
//
// The other tcgen05 kernel (attn_latent_tc.cu) puts 128 (row, head) pairs on M; a row of 16 heads fills an eighth of it and the scores are
// computed twice.  Here the key tile is the large operand, so nothing is computed for pairs that do not exist: per 128 keys
//   S^T[128 keys][16] = K_tile[128][krow] . Q^T            O^T[128 value columns][16 + 16] += V_tile^T . [P_hi | P_lo]   (per 128 value columns)
// where V_tile^T is the key tile itself read MN-major, and the weights' bf16 term and what rounding took from it are the two halves of N, so that
// both cost one pass over the values.
//
// A cluster of C CTAs shares a row's context (C while the device has places for them: eight for up to 15 rows, four for 33, two for 74); their sums
// meet through distributed shared memory, each CTA finishing its share of the columns.  No run list, no second launch.
// Bound by the trip of a tile: 147 KB of keys (krow 576) fill most of shared memory, so the loads of a tile start as the second product of the one
// before gives its columns back, and 68 MMAs of 40 to 50 cycles; 3.5 us per 128 keys.  (Tiles of 64 keys, whose next one would fit: the scores' MMAs cost
// as much, 119 us for 100 rows at contexts 1500..3000 against 86.  Rows asked into L2 ahead, 104 against 101: memory is not it.)
// MMAs of a whole chunk are straight code: in a loop of as many as the chunk has 16-wide steps each took 110 cycles (101 us against 86).
// 16 heads over 512 + 64, us, on attn_latent_tc.cu (with the splits that the caller asks for) and here: 64 rows at contexts 500..1000 49, 27 (among other calls), 100 of
// 3000 208, 96, one of 3000 54, 25, 33 of 3000 122, 43; of one sequence 33 behind 3000 73, 33, 100 behind 3000 87, 86 and behind 16 000 183, 385: what is whose is
// latent_attn_route's and runs.cuh's.  Error against 64 bits as there.
// Warps: TMA producer, MMA issuer, four softmax warps (a thread owns a key, then a value column).  The running maximum is only followed when it
// rises by more than 2^8, as in attn_latent_tc.cu.  Every wait is bounded and reported (tc.cuh).
#include <algorithm>

#include "runs.cuh"
#include "tc.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int kLrKeys = 128, kLrPairs = 16, kLrThreads = 192;
constexpr int kLrChunk = kLrKeys * 128;        // [128 keys][64 columns] bf16: 16 KiB, two of them a slot of the value ring
constexpr int kLrQChunk = kLrPairs * 128;      // [16 heads][64 columns]
constexpr int kLrP = 2 * 2 * kLrPairs * 128;   // [2 x 64 keys][hi 16 | lo 16][64 keys]
constexpr int kLrMaxSlots = 6, kLrMaxRest = 4, kLrSmem = 232448, kLrTail = 2048;
constexpr uint32_t kLrTmO = 32;                // TMEM columns: two score buffers of 16, then 32 per 128 value columns

struct LrParams {
  const float* q;
  const int32_t* block_table;
  const int32_t* row_to_seq;
  const int32_t* ctx_lens;
  const float* sink;
  __nv_bfloat16* out;
  float* part;         // n_splits > 1: unnormalised sums [pair][split][rank | maximum | denominator], merged by another launch
  uint32_t* status;
  int bt_stride, heads, groups, krow, rank, block_size, window, vpairs, rest, slots, rest_slots, cluster, n_splits;   // groups: of up to 16 heads
  float scale;
  LatentShare share;
};

__device__ __forceinline__ uint32_t lr_idesc(int n, int a_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// one step of the maxima (sums) over a group of lanes: 2 H values become H
template <int H, bool MAX>
__device__ __forceinline__ void lr_halve(float* x, int lane) {
  const bool up = (lane & H) != 0;
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const float keep = up ? x[i + H] : x[i], other = __shfl_xor_sync(0xffffffffu, up ? x[i] : x[i + H], H);
    x[i] = MAX ? fmaxf(keep, other) : keep + other;
  }
}
// over the warp, of value i of 16, to lanes i and i + 16
template <bool MAX>
__device__ __forceinline__ float lr_reduce(float (&x)[16], int lane) {
  lr_halve<8, MAX>(x, lane);
  lr_halve<4, MAX>(x, lane);
  lr_halve<2, MAX>(x, lane);
  lr_halve<1, MAX>(x, lane);
  const float other = __shfl_xor_sync(0xffffffffu, x[0], 16);
  return MAX ? fmaxf(x[0], other) : x[0] + other;
}

__global__ void __launch_bounds__(kLrThreads, 1) latent_rows_kernel(const __grid_constant__ CUtensorMap map, const LrParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (p.krow + 63) >> 6, ksteps = p.krow >> 4, vchunks = min(2 * p.vpairs, chunks);
  unsigned char* ring = smem;                                  // [slots][2][128][64] value columns of a tile, in pairs of chunks
  unsigned char* rest_ring = ring + p.slots * 2 * kLrChunk;    // [rest_slots][128][64] its other chunks
  unsigned char* qs = rest_ring + p.rest_slots * kLrChunk;     // [chunks][16][64]
  unsigned char* ps = qs + chunks * kLrQChunk;
  uint64_t* full = reinterpret_cast<uint64_t*>(ps + kLrP);
  uint64_t* empty = full + kLrMaxSlots;
  uint64_t* rest_full = empty + kLrMaxSlots;
  uint64_t* rest_empty = rest_full + kLrMaxRest;
  uint64_t* s_full = rest_empty + kLrMaxRest;    // [2]
  uint64_t* p_ready = s_full + 2;
  uint64_t* o_full = p_ready + 1;
  uint64_t* q_ready = o_full + 1;
  uint64_t* last = q_ready + 1;                  // the MMAs in flight when a wait ran out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(last + 1);   // and, behind it, the mark of a wait that ran out
  float* wmax = reinterpret_cast<float*>(tmem_slot + 4);         // [2][4 warps][16]
  float* stat = wmax + 2 * 4 * kLrPairs;                         // [maximum (log2), denominator][16] of this CTA
  float* lred = stat + 2 * kLrPairs;                             // [4 warps][16]
  float* fac = lred + 4 * kLrPairs;                              // [16 heads][8 CTAs] what their sums are weighted with
  const Waits wait(tmem_slot + 1, p.status);
  if (p.share.plan) {
    pdl_wait();
    if (!latent_by_rows(p.share)) return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.slots; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int s = 0; s < p.rest_slots; ++s) {
      mbar_init(rest_full + s, 1);
      mbar_init(rest_empty + s, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_full + 1, 1);
    mbar_init(p_ready, 4);
    mbar_init(o_full, 1);
    mbar_init(q_ready, 4);
    mbar_init(last, 1);
    tmem_slot[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();
  const int part = blockIdx.x % p.cluster, split = blockIdx.x / p.cluster % p.n_splits, item = blockIdx.x / (p.cluster * p.n_splits);
  const int t = item / p.groups, h0 = item % p.groups * kLrPairs, shares = p.cluster * p.n_splits, share0 = split * p.cluster + part;
  const int n_heads = min(p.heads - h0, kLrPairs);
  const int ctx = p.ctx_lens[t], lo = p.window > 0 ? max(ctx - p.window, 0) : 0;
  // tiles from the 64 keys that hold the oldest visible one: a cache block is whole 64s, so none is read that lies before the window
  const int first = lo & ~63, tiles = max((ctx - first + kLrKeys - 1) / kLrKeys, 0), per = (tiles + shares - 1) / shares;
  const int tile_lo = min(tiles, share0 * per), tile_hi = min(tiles, (share0 + 1) * per);

  const int fh = threadIdx.x >> 3, fz = threadIdx.x & 7;   // the factor that the thread works out at the end
  const float sk = threadIdx.x < 8 * kLrPairs && fh < n_heads && p.sink && p.n_splits == 1 ? p.sink[h0 + fh] * 1.4426950408889634f : -INFINITY;

  if (warp == 0) {
    // ===== TMA: per tile the value columns two chunks a slot, then the other chunks; 64 keys a box, those past the context's last box left out =====
    const bool issuer = elect_one();
    if (issuer) asm volatile("prefetch.tensormap [%0];" ::"l"(&map) : "memory");
    const int32_t* bt = p.block_table + (int64_t)(p.row_to_seq ? p.row_to_seq[t] : t) * p.bt_stride;
    int st = 0, rs = 0;
    uint32_t st_ph = 1, rs_ph = 1;   // parity of the release that a slot's next load waits for (the first round finds it free)
    for (int i = tile_lo; i < tile_hi && !wait.stop(); ++i) {
      const int tok = first + i * kLrKeys, halves = ctx - tok > 64 ? 2 : 1;
      int row[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int k = tok + (x < halves ? x * 64 : 0);
        row[x] = __shfl_sync(0xffffffffu, bt[k / p.block_size], 0) * p.block_size + k % p.block_size;
      }
      auto load = [&](unsigned char* dst, int c, uint64_t* bar) {
        for (int x = 0; x < halves; ++x) tma_load_2d(dst + x * 8192, &map, c * 64, row[x], bar);
      };
      for (int j = 0; j < p.vpairs; ++j) {
        wait(empty + st, st_ph);
        if (issuer) {
          const int n = min(2, vchunks - 2 * j);
          mbar_expect_tx(full + st, n * halves * 8192);
          for (int c = 0; c < n; ++c) load(ring + (st * 2 + c) * kLrChunk, 2 * j + c, full + st);
        }
        __syncwarp();
        if (++st == p.slots) st = 0, st_ph ^= 1;
      }
      for (int c = 0; c < p.rest; ++c) {
        wait(rest_empty + rs, rs_ph);
        if (issuer) {
          mbar_expect_tx(rest_full + rs, halves * 8192);
          load(rest_ring + rs * kLrChunk, vchunks + c, rest_full + rs);
        }
        __syncwarp();
        if (++rs == p.rest_slots) rs = 0, rs_ph ^= 1;
      }
    }
    if (wait.stop()) {   // the loads in flight: a slot's last one filled it in this round of the ring or in the one before
      for (int s = 0; s < p.slots; ++s) wait.drain(full + s, s < st ? st_ph ^ 1 : st_ph);
      for (int s = 0; s < p.rest_slots; ++s) wait.drain(rest_full + s, s < rs ? rs_ph ^ 1 : rs_ph);
    }
  } else if (warp == 1) {
    // ===== MMA: the whole warp walks the loops; with room for two tiles the scores of the next are issued before the weights of this one =====
    const uint32_t one = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t desc_k = make_desc(smem_u32(ring), 16, 1024), desc_r = make_desc(smem_u32(rest_ring), 16, 1024),
                   desc_q = make_desc(smem_u32(qs), 16, 1024), desc_v = make_desc(smem_u32(ring), kLrChunk, 1024), desc_p = make_desc(smem_u32(ps), 16, 1024);
    const uint32_t id_s = lr_idesc(kLrPairs, 0), id_o = lr_idesc(2 * kLrPairs, 1);
    const bool ahead = p.slots >= 2 * p.vpairs && p.rest_slots >= 2 * p.rest;
    const int nt = __shfl_sync(0xffffffffu, tile_hi - tile_lo, 0), keys = __shfl_sync(0xffffffffu, ctx - first - tile_lo * kLrKeys, 0);
    int st = 0, rs = 0, pv_st = 0;
    uint32_t st_ph = 0, rs_ph = 0;
    auto chunk = [&](uint32_t d, uint64_t da, int c) {
      const uint64_t dq = desc_q + (uint64_t)((c * kLrQChunk) >> 4);
      const int ks = min(4, ksteps - 4 * c);
      const uint32_t acc = c ? 1u : 0u;
      if (ks == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_ss(one, d, da + j * 2, dq + j * 2, id_s, j ? 1u : acc);
      } else {
        for (int j = 0; j < ks; ++j) mma_ss(one, d, da + j * 2, dq + j * 2, id_s, j ? 1u : acc);
      }
    };
    auto scores = [&](int n) {
      const uint32_t d = tm + (n & 1) * kLrPairs;
      for (int j = 0; j < p.vpairs; ++j) {
        wait(full + st, st_ph);
        fence_after();
        for (int c = 0; c < min(2, vchunks - 2 * j); ++c) chunk(d, desc_k + (uint64_t)(((st * 2 + c) * kLrChunk) >> 4), 2 * j + c);
        if (++st == p.slots) st = 0, st_ph ^= 1;
      }
      for (int c = 0; c < p.rest; ++c) {
        wait(rest_full + rs, rs_ph);
        fence_after();
        chunk(d, desc_r + (uint64_t)((rs * kLrChunk) >> 4), vchunks + c);
        commit(one, rest_empty + rs);
        if (++rs == p.rest_slots) rs = 0, rs_ph ^= 1;
      }
      commit(one, s_full + (n & 1));
    };
    if (nt > 0) {
      wait(q_ready, 0);
      fence_after();
      scores(0);
    }
    for (int n = 0; n < nt; ++n) {
      if (ahead && n + 1 < nt) scores(n + 1);
      wait(p_ready, n & 1);
      fence_after();
      const int steps = min(8, (keys - n * kLrKeys + 15) >> 4);   // 16 keys each
      for (int j = 0; j < p.vpairs; ++j) {
        const uint64_t dv = desc_v + (uint64_t)((pv_st * 2 * kLrChunk) >> 4);
        const uint32_t o = tm + kLrTmO + j * 32, acc = n ? 1u : 0u;
        if (steps == 8) {
#pragma unroll
          for (int s = 0; s < 8; ++s) mma_ss(one, o, dv + (uint64_t)(s * 128), desc_p + (uint64_t)((s >> 2) * 256 + (s & 3) * 2), id_o, s ? 1u : acc);
        } else {
          for (int s = 0; s < steps; ++s) mma_ss(one, o, dv + (uint64_t)(s * 128), desc_p + (uint64_t)((s >> 2) * 256 + (s & 3) * 2), id_o, s ? 1u : acc);
        }
        commit(one, empty + pv_st);
        if (++pv_st == p.slots) pv_st = 0;
      }
      commit(one, o_full);
      if (!ahead && n + 1 < nt) scores(n + 1);
    }
    if (wait.stop()) {
      commit(one, last);
      wait.drain(last, 0);
    }
  } else {
    // ===== softmax: a thread owns a key of the tile =====
    const int quad = warp & 3, m = quad * 32 + lane, tid = threadIdx.x - 64;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    // the row's queries, fp32 -> bf16 chunks of 64 columns: eight lanes a row of a chunk (16-byte pieces)
    const float* qrow = p.q + ((int64_t)t * p.heads + h0) * p.krow;
    for (int c0 = 0; c0 < chunks; c0 += 5) {   // a thread's piece of five chunks requested before the first is used
      const int r = tid >> 3, col = (tid & 7) * 8;
      float4 v[5][2];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const bool ok = r < n_heads && (c0 + i) * 64 + col < p.krow;
        const float4* src = reinterpret_cast<const float4*>(qrow + (int64_t)r * p.krow + (c0 + i) * 64 + col);
        v[i][0] = ok ? src[0] : make_float4(0.f, 0.f, 0.f, 0.f);
        v[i][1] = ok ? src[1] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < 5; ++i)
        if (c0 + i < chunks)
          *reinterpret_cast<uint4*>(qs + (c0 + i) * kLrQChunk + (r >> 3) * 1024 + (r & 7) * 128 + (((tid & 7) ^ (r & 7)) << 4)) =
              make_uint4(pack_bf16(v[i][0].x, v[i][0].y), pack_bf16(v[i][0].z, v[i][0].w), pack_bf16(v[i][1].x, v[i][1].y), pack_bf16(v[i][1].z, v[i][1].w));
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(q_ready);
    const float sc2 = p.scale * 1.4426950408889634f;   // scores in the log2 domain
    float mu = -INFINITY;                              // of head lane % 16
    float mus[16], l[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) mus[i] = 0.f, l[i] = 0.f;
    int n = 0;
    for (int i = tile_lo; i < tile_hi; ++i, ++n) {
      const int key = first + i * kLrKeys + m;
      const bool live = key >= lo && key < ctx;
      wait(s_full + (n & 1), (n >> 1) & 1);
      fence_after();
      uint32_t raw[16];
      ld16(tmem + lane_off + (n & 1) * kLrPairs, raw);
      ld_wait<16>(raw);
      float x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = live ? __uint_as_float(raw[j]) : -INFINITY;
      const float wm = lr_reduce<true>(x, lane) * sc2;
      float* wx = wmax + (n & 1) * 4 * kLrPairs;
      if (lane < 16) wx[quad * kLrPairs + lane] = wm;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const int h = lane & 15;
      const float mx = fmaxf(fmaxf(wx[h], wx[kLrPairs + h]), fmaxf(wx[2 * kLrPairs + h], wx[3 * kLrPairs + h]));
      const bool jump = mx > mu + 8.f;   // also the first live key (mu = -inf)
      if (n > 0) {   // the second product of the tile before has taken the weights (and may be rescaled)
        wait(o_full, (n - 1) & 1);
        fence_after();
      }
      if (__any_sync(0xffffffffu, jump)) {   // the same answer in all four warps
        const float mn = jump ? mx : mu, f = jump && mu != -INFINITY ? exp2_fast(mu - mn) : 1.f;
        float fs[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          mus[j] = __shfl_sync(0xffffffffu, mn > -INFINITY ? mn : 0.f, j);
          fs[j] = __shfl_sync(0xffffffffu, f, j);
          l[j] *= fs[j];
        }
        mu = mn;
        if (n > 0)
          for (int j = 0; j < p.vpairs; ++j) {
            uint32_t o[32];
            ld32(tmem + lane_off + kLrTmO + j * 32, o);
            ld_wait<32>(o);
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * fs[c & 15]);
            st32(tmem + lane_off + kLrTmO + j * 32, o);
          }
      }
      // weights: row h the bf16 term, row 16 + h what that rounding took; key m of the tile is column m % 64 of chunk m / 64
      unsigned char* pw = ps + (m >> 6) * 4096 + (m & 7) * 2;
      const int piece = (m & 63) >> 3;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float w = live ? exp2_fast(fmaf(__uint_as_float(raw[j]), sc2, -mus[j])) : 0.f;
        l[j] += w;
        const uint32_t hi = __float_as_uint(w) & 0xffff0000u;
        unsigned char* at = pw + (j >> 3) * 1024 + (j & 7) * 128 + ((piece ^ (j & 7)) << 4);
        *reinterpret_cast<uint16_t*>(at) = (uint16_t)(hi >> 16);
        *reinterpret_cast<__nv_bfloat16*>(at + 2048) = __float2bfloat16_rn(w - __uint_as_float(hi));
      }
      const int n_valid = min(ctx - first - i * kLrKeys, kLrKeys), n_read = (n_valid + 15) & ~15;
      if (n_valid < n_read) {
        // value rows past the context may hold anything, and 0 * NaN = NaN: zero those that the last step of 16 keys reads
        const int units = (n_read - n_valid) * 8;
        for (int c = 0; c < vchunks; ++c) {
          unsigned char* vb = ring + (((n * p.vpairs + (c >> 1)) % p.slots) * 2 + (c & 1)) * kLrChunk + n_valid * 128;
          for (int e = tid; e < units; e += 128) *reinterpret_cast<uint4*>(vb + e * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      st_wait();
      fence_async_smem();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
    }
    // this CTA's sums: [head][rank] floats where the ring was, maxima and denominators beside them
    const float ls = lr_reduce<false>(l, lane);
    if (lane < 16) lred[quad * kLrPairs + lane] = ls;
    if (n > 0) {
      wait(o_full, (n - 1) & 1);
      fence_after();
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (tid < kLrPairs) {
      stat[tid] = mu;
      stat[kLrPairs + tid] = lred[tid] + lred[kLrPairs + tid] + lred[2 * kLrPairs + tid] + lred[3 * kLrPairs + tid];
    }
    float* sums = reinterpret_cast<float*>(ring);
    for (int j = 0; j < p.vpairs; ++j) {
      uint32_t o[32];
      if (n > 0) {
        ld32(tmem + lane_off + kLrTmO + j * 32, o);
        ld_wait<32>(o);
      }
      const int d = j * 128 + m;
      if (d < p.rank)
#pragma unroll
        for (int h = 0; h < 16; ++h) sums[h * p.rank + d] = n > 0 ? __uint_as_float(o[h]) + __uint_as_float(o[16 + h]) : 0.f;
    }
    fence_before();
  }
  __syncthreads();
  if (p.cluster > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  // every CTA finishes its share of the columns: the cluster's sums brought to one maximum (the sink's included), added and normalised
  {
    auto peer = [&](const void* a, int c) {
      uint32_t r;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(a)), "r"(c));
      return r;
    };
    if (threadIdx.x < 8 * kLrPairs) {
      float mc = -INFINITY, lc = 0.f;
      if (fz < p.cluster) {
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(mc) : "r"(peer(stat + fh, fz)) : "memory");
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(lc) : "r"(peer(stat + kLrPairs + fh, fz)) : "memory");
      }
      float mn = mc;
#pragma unroll
      for (int o = 4; o >= 1; o >>= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mn = fmaxf(mn, sk);
      const float ec = mc != -INFINITY ? exp2_fast(mc - mn) : 0.f;
      float den = lc * ec;
#pragma unroll
      for (int o = 4; o >= 1; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
      if (p.n_splits > 1) {
        fac[threadIdx.x] = ec;
        if (fz == 0 && part == 0 && fh < n_heads) {   // the maximum in natural units
          float* dst = p.part + (((int64_t)t * p.heads + h0 + fh) * p.n_splits + split) * (p.rank + 2) + p.rank;
          dst[0] = mn * 0.6931471805599453f;
          dst[1] = den;
        }
      } else {
        if (p.sink) den += exp2_fast(sk - mn);
        fac[threadIdx.x] = den > 0.f ? ec / den : 0.f;
      }
    }
    __syncthreads();
    // units of four columns; a thread's loads of four units and all CTAs are requested together
    const int wide = p.rank / 4, share = (wide + p.cluster - 1) / p.cluster, u0 = part * share, cols = max(min(share, wide - u0), 0), units = n_heads * cols;
    const float* sums = reinterpret_cast<const float*>(ring);
    __nv_bfloat16* dst = p.out + ((int64_t)t * p.heads + h0) * p.rank;
    constexpr int U = 4;
    for (int e0 = threadIdx.x; e0 < units; e0 += U * kLrThreads) {
      float4 a[U];
      int at[U], hh[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = min(e0 + u * kLrThreads, units - 1);
        hh[u] = e / cols;
        at[u] = hh[u] * p.rank + (u0 + e % cols) * 4;
        a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      auto add = [&](float4& to, const float4& v, float f) { to.x = fmaf(v.x, f, to.x), to.y = fmaf(v.y, f, to.y), to.z = fmaf(v.z, f, to.z), to.w = fmaf(v.w, f, to.w); };
      if (p.cluster == 1) {
#pragma unroll
        for (int u = 0; u < U; ++u) add(a[u], *reinterpret_cast<const float4*>(sums + at[u]), fac[hh[u] * 8]);
      } else {
        for (int z = 0; z < p.cluster; z += 2) {   // (a power of two)
          float4 v[2][U];
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int u = 0; u < U; ++u)
              asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[x][u].x), "=f"(v[x][u].y), "=f"(v[x][u].z), "=f"(v[x][u].w) : "r"(peer(sums + at[u], z + x)) : "memory");
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int u = 0; u < U; ++u) add(a[u], v[x][u], fac[hh[u] * 8 + z + x]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (e0 + u * kLrThreads < units) {
          if (p.n_splits > 1) {
            float2* d2 = reinterpret_cast<float2*>(p.part + (((int64_t)t * p.heads + h0 + hh[u]) * p.n_splits + split) * (p.rank + 2) + at[u] - hh[u] * p.rank);
            d2[0] = make_float2(a[u].x, a[u].y);   // (rank + 2 is even: 8-byte aligned rows)
            d2[1] = make_float2(a[u].z, a[u].w);
          } else {
            *reinterpret_cast<uint2*>(dst + at[u]) = make_uint2(pack_bf16(a[u].x, a[u].y), pack_bf16(a[u].z, a[u].w));
          }
        }
    }
  }
  if (p.cluster > 1) {   // nobody leaves while a peer reads its sums
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u));
  }
}

// false: key rows whose tile and queries do not fit beside each other
bool lr_shape(int krow, int rank, LrParams& p) {
  if (krow % 16 || rank % 16 || rank < 16 || rank > 512 || rank > krow) return false;
  const int chunks = (krow + 63) / 64;
  p.vpairs = (rank + 127) / 128;
  p.rest = std::max(chunks - 2 * p.vpairs, 0);
  p.rest_slots = 2 * p.rest;
  if (p.rest_slots > kLrMaxRest) return false;
  const int room = kLrSmem - 1024 - kLrTail - chunks * kLrQChunk - kLrP - p.rest_slots * kLrChunk;
  p.slots = std::min(room / (2 * kLrChunk), kLrMaxSlots);
  return p.slots >= p.vpairs;
}

}  // namespace

bool latent_attn_rows_supported(int heads, int krow, int rank, int block_size) {
  LrParams p;
  return heads > 0 && block_size > 0 && block_size % 64 == 0 && lr_shape(krow, rank, p);
}
int latent_attn_rows_items(int T, int heads) { return T * ((heads + kLrPairs - 1) / kLrPairs); }
int latent_attn_rows_cluster(int items) { return items <= 15 ? 8 : items <= 33 ? 4 : items <= 74 ? 2 : 1; }   // clusters of whole SMs that the device holds at a time

// every row by itself (row t of sequence row_to_seq[t], or t); scale > 0.  n_splits: at most so many shares of the context beyond the cluster's; how many were
// taken (more than one: unmerged sums in part).  share: whether the step is this kernel's
int latent_attn_rows(const float* q, const __nv_bfloat16* kc, const int32_t* block_table, int bt_stride, const int32_t* row_to_seq, const int32_t* ctx_lens,
                     __nv_bfloat16* out, int T, int heads, int krow, int rank, int block_size, float scale, const float* sink, cudaStream_t s, int window, float* part,
                     int64_t longest, const LatentShare& share, int* n_splits) {
  LrParams p = {};
  B200_REQUIRE(latent_attn_rows_supported(heads, krow, rank, block_size) && lr_shape(krow, rank, p), B200_ERR_UNSUPPORTED,
               "latent_attn_rows: shape %d / %d / %d", heads, krow, rank);
  if (const int e = wait_status()) return e;
  CUtensorMap map;
  const int rc = get_tensor_map_2d(kc, 1ull << 31, krow, krow, 64, &map);   // rows touched come from the block table
  if (rc) return rc;
  p.q = q;
  p.block_table = block_table;
  p.row_to_seq = row_to_seq;
  p.ctx_lens = ctx_lens;
  p.sink = sink;
  p.out = out;
  p.status = wait_status_word();
  p.bt_stride = bt_stride;
  p.heads = heads;
  p.groups = (heads + kLrPairs - 1) / kLrPairs;
  p.krow = krow;
  p.rank = rank;
  p.block_size = block_size;
  p.window = window;
  p.scale = scale;
  const int items = T * p.groups;
  p.cluster = latent_attn_rows_cluster(items);
  p.share = share;
  // One to seven rows leave SMs for more shares, whose merge is a launch of its own and pays at long contexts only (one row of 3 000 tokens 21 us without, 39 with
  // all of them; of 16 000 58 and 43, of 60 000 about 180 and 53; 50, 77 and 158 on attn_latent_tc.cu).
  p.n_splits = part && !share.plan && p.cluster == 8 && longest > 32768 ? std::max(std::min(*n_splits, 15 / items), 1) : 1;
  p.part = part;
  *n_splits = p.n_splits;
  static bool done[64] = {};
  B200_CUDA(ensure_dynamic_smem(latent_rows_kernel, kLrSmem, done));
  B200_CUDA(launch_cluster(latent_rows_kernel, dim3((unsigned)(items * p.cluster * p.n_splits)), dim3(kLrThreads), (size_t)kLrSmem, s, dim3(p.cluster, 1, 1), map, p));
  return B200_OK;
}

}  // namespace b200
