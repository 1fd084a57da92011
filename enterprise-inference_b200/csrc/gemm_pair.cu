// tcgen05 linear for more than 128 tokens on pairs of SMs: y[T][n_out] = x[T][k] . w[n_out][k]^T with 256 weight rows and up to 256
// tokens a tile (tcgen05.mma.cta_group::2), and the grouped form of the same for routed experts.
//
// What bounds it: the tensor pipe, if the operands arrive.  A CTA by itself (gemm_tc.cu, 128 weight rows x 256 tokens) fetches 48 KiB per 64 of
// k for 512 cycles of MMAs, 96 bytes a cycle of the 64 that an SM gets from L2.  A pair shares the token rows: each CTA fetches its own 128
// weight rows and half of the tokens, 32 KiB for the same 512 cycles.
//
// A CTA pair per two SMs, persistent.  Per CTA: a warp fetches weights and one token rows (TMA, rings of seven and five times 16 KiB; both CTAs' bytes
// complete on the leader's barriers), warp 1 of the leader issues the MMAs of both, eight warps turn the accumulator into the launch's output.  The 512 columns of tensor memory hold two
// accumulators, so a tile's epilogue runs beside the next tile's MMAs; it goes through shared memory of its own, 32 tokens at a time per
// four warps.  Launches with few tiles share a tile's k between up to four pairs of one cluster, which add up through distributed shared memory.
//
// Against 128 x 256 tiles of single CTAs with k split over clusters (us, before -> now; five calls in a row after the L2 was overwritten): 2000 tokens, k 14336,
// 4096 features 177 -> 158 (among other calls, under the power cap, 208 -> 194); 2048, 4096, 28672 472 -> 337; 2048, 4096, 6144 142 -> 94; 1000, 4096, 4096 72 -> 41;
// 300, 2048, 2048 32 -> 18; 200, 14336, 4096 67 -> 45; 130, 2048, 2048 29 -> 17.
// Routed experts (the table of token tiles is moe.cu's): 32 experts of 1024, width 2048, 4 of them a row, router and grouping included, tiles of
// 128 x 128 before: 2048 rows 264 -> 175 (among other calls 280 -> 192), 1200 rows 222 -> 135, 700 rows 164 -> 124; 64 of 512, width 4096, 8 a row, 2048 rows
// 582 -> 363.  Their weights come from HBM (1000 rows: 402 MB), and whole waves of tiles decide the rest (2048 rows: 5.2 waves of gate|up).
// 128 tokens and fewer stay on gemm_tc.cu's tiles: their launches stream W, and 148 CTAs with two of them to an SM keep more of it in flight
// (64 tokens, 4096, 28672: 42 there, 49 here; 128, 14336, 4096: 33 and 34).
#include <algorithm>
#include <type_traits>

#include "gemm_epilogue.cuh"
#include "pair_drain.h"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int kPairWarps = 11, kPairThreads = kPairWarps * 32;
// Weights come from HBM, token rows (which other pairs read too) mostly from L2: a ring and a fetching warp for each, the one that waits longer deeper.  Against six
// stages of both and one warp (us, graph): 383 x 5120 x 7168 34.3 -> 25.1, 700 rows 59.6 -> 47.2, 1500 x 2048 x 8192 43 -> 37.6, 1000 x 4096 x 4096 31 -> 27; 16
// experts of 1024, width 1024, 2048 rows 93 -> 77.  Rings of 8 and 4 gain as much there, but lose where tokens come late (2000 x 14336 x 4096 157 -> 165, 32
// experts 155 -> 167); 6 and 6 leave the first group at 30, 56, 43 and 31.
constexpr int kPairWStages = 7, kPairXStages = 5;
constexpr int kPairABytes = kBlockM * kBlockK * 2;          // this CTA's weight rows of a stage; the token rows (at most 128) take as much
constexpr int kPairRings = (kPairWStages + kPairXStages) * kPairABytes;
constexpr int kPairStgTok = 32;                             // tokens of a staged piece of the epilogue
constexpr int kPairSplits = 4;                              // shares of k at most: clusters of eight CTAs
constexpr int kPairStgBytes = kPairStgTok * kBlockM * 4;
constexpr int kPairSmem = 1024 + kPairRings + 2 * kPairStgBytes + 512;
constexpr uint64_t kKeepNormal = 0x1000000000000000ull, kKeepLast = 0x14F0000000000000ull;

__device__ __forceinline__ uint32_t smem_of(const void* p, int cta) {   // the same shared-memory address in another CTA of the cluster
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(tc::smem_u32(p)), "r"(cta));
  return r;
}
// A wait that runs out marks every CTA of the cluster: each serves another's loads, MMAs or sums.  What follows is out of the loops' way, in
// functions of its own, and the loops' predicates stay what they were (an MMA predicate that a wait may clear: 187 us instead of 196).
constexpr uint32_t kPairRunning = 0xffffffffu;   // Waits::mark[1] (weights), [2] (tokens) until the CTA's fetching warp has ended, then the fills it issued
__device__ __noinline__ void pair_gave_up(uint32_t* mark, uint32_t* status, int ctas) {
  *reinterpret_cast<volatile uint32_t*>(mark) = 1;
  for (int c = 0; c < ctas; ++c) asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(smem_of(mark, c)), "r"(1u) : "memory");
  if (status) *reinterpret_cast<volatile uint32_t*>(status) = 1;
}
__device__ __forceinline__ uint32_t pair_issued(uint32_t* mark, int ring, int cta) {
  uint32_t v;
  asm volatile("ld.relaxed.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(smem_of(mark + 1 + ring, cta)) : "memory");
  return v;
}
// before the MMA warp commits anything for a fill that did not land: all fetching warps have ended (they see the mark), so nothing is issued on it
__device__ __noinline__ void pair_await_ends(uint32_t* mark, int lead, int limit) {
  for (int i = 0; i < limit && (pair_issued(mark, 0, lead) == kPairRunning || pair_issued(mark, 0, lead + 1) == kPairRunning ||
                                pair_issued(mark, 1, lead) == kPairRunning || pair_issued(mark, 1, lead + 1) == kPairRunning); ++i)
    __nanosleep(1000);
}
struct PairWaits : tc::Waits {
  int ctas;
  __device__ __forceinline__ PairWaits(uint32_t* m, uint32_t* st, int n) : tc::Waits(m, st), ctas(n) {}
  template <typename F>
  __device__ __forceinline__ void operator()(uint64_t* bar, uint32_t parity, F&& gave_up) const {
    for (int i = 0; !tc::mbar_try(bar, parity); ++i)
      if ((i & 63) == 63 && (marked() || i > limit)) {
        if (!marked()) pair_gave_up(mark, status, ctas);
        gave_up();
        return;
      }
  }
  __device__ __forceinline__ void operator()(uint64_t* bar, uint32_t parity) const { (*this)(bar, parity, [] {}); }
  // for the whole warp; false: it ran out
  __device__ __forceinline__ bool all(uint64_t* bar, uint32_t parity) const {
    if (__all_sync(0xffffffffu, tc::mbar_try(bar, parity))) return true;
    (*this)(bar, parity);
    return !stop();
  }
};
__device__ __forceinline__ void pair_load(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(
          tc::smem_u32(dst)),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
// two boxes of rows, c2 and the slab behind it
__device__ __forceinline__ void pair_load3(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(
          tc::smem_u32(dst)),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t one, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 q, %5, 0;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(one)
      : "memory");
}
// arrives at this barrier of the CTAs in `ctas` (one bit each) once the MMAs issued so far are done
__device__ __forceinline__ void pair_commit(uint32_t one, uint64_t* bar, uint16_t ctas) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %1, 0;\n"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n"
      "}\n" ::"r"(tc::smem_u32(bar)),
      "r"(one), "h"(ctas)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
        "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The token rows in boxes of 16, 32, .. 128 rows: a CTA's half of any tile in one load (a load more a stage costs the fetching warp more than the
// ring can hide: 2 048 rows of 32 experts in boxes of 64 and 16 180 us, so 174)
struct PairMaps {
  CUtensorMap x[8];
};

struct PairTile {
  int m, row0, n, expert;   // 256-row tile of W, first token row, tokens (a multiple of 32)
};
__device__ __forceinline__ PairTile pair_tile(const TcParams& p, int t) {
  PairTile r;
  if (p.pair_tile) {   // an expert's slabs follow each other: its tokens stay in L2
    const int4 e = __ldg(p.pair_tile + 1 + t / p.pair_m);
    r.m = t % p.pair_m;
    r.expert = e.x;
    r.row0 = e.y;
    r.n = min(max(e.z & ~31, 32), 256);   // (whatever has become of the caller's workspace, never an MMA of an undefined shape)
  } else {             // tokens fast: the tiles in flight share a few slabs and pair_group token tiles
    const int per = p.pair_group * p.pair_m, g = t / per, gs = min(p.pair_group, p.pair_tok - g * p.pair_group), i = t - g * per;
    r.m = i / gs;
    r.expert = 0;
    r.row0 = (g * p.pair_group + i % gs) * p.pair_n;
    r.n = p.pair_n;
  }
  return r;
}

// After a wait that ran out, with both CTAs' roles at their ends: the loads in flight (of either ring) land before either gives its shared memory up.
__device__ __forceinline__ void pair_land(const PairWaits& wait, uint64_t* full_w, uint64_t* full_x, const TcParams& p, uint32_t* mark, int lead, int kbs, int first,
                                          int step) {
#pragma unroll 1
  for (int i = 0; i < kPairWStages + kPairXStages; ++i) {
    const int ring = i >= kPairWStages, s = ring ? i - kPairWStages : i;
    uint64_t* full = ring ? full_x + s : full_w + s;
    const PairOwed o = pair_owed(s, ring ? kPairXStages : kPairWStages, (int)pair_issued(mark, ring, lead), (int)pair_issued(mark, ring, lead + 1));
    if (o.parity < 0) continue;
    const uint32_t half = ring ? (uint32_t)pair_tile(p, first + o.fill / kbs * step).n * kBlockK : kPairABytes;   // a CTA's bytes of the fill
    if (o.announce > 0) tc::mbar_expect_tx(full, half);
    if (o.announce < 0) asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(tc::smem_u32(full)), "r"(half) : "memory");
    wait.drain(full, (uint32_t)o.parity);
  }
}

__device__ __forceinline__ void pair_bias(const TcParams& p, int m_tile, int r4, float (&bb)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int row = m_tile * kBlockM + r4 + e;
    bb[e] = p.bias && row < p.n_out ? __bfloat162float(p.bias[row]) : 0.f;
  }
}

template <int MODE>
__global__ void __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ PairMaps maps, const TcParams p, uint32_t* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* stg_all = reinterpret_cast<float*>(smem + kPairRings);
  uint64_t* full_w = reinterpret_cast<uint64_t*>(smem + kPairRings + 2 * kPairStgBytes);   // the leader's: both CTAs' bytes
  uint64_t* full_x = full_w + kPairWStages;
  uint64_t* empty_w = full_x + kPairXStages;
  uint64_t* empty_x = empty_w + kPairWStages;
  uint64_t* acc_full = empty_x + kPairXStages;   // [2]
  uint64_t* acc_free = acc_full + 2;           // [2] the leader's: both CTAs' epilogue warps
  uint64_t* last = acc_free + 2;               // after a wait that ran out: the MMAs issued before
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(last + 1);
  uint32_t* mark = tmem_slot + 1;              // and, behind it, how many fills of either ring the CTA issued
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a cluster: the CTA pairs of one tile, each with its share of k
  const int cta = blockIdx.x % (2 * p.splits), rank = cta & 1, split = cta >> 1, lead = cta - rank;
  const int first = blockIdx.x / (2 * p.splits), step = gridDim.x / (2 * p.splits);
  const int kb_base = p.n_kblocks / p.splits, kb_rem = p.n_kblocks % p.splits;
  const int kb0 = split * kb_base + min(split, kb_rem), kb1 = kb0 + kb_base + (split < kb_rem ? 1 : 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * (kPairWStages + kPairXStages); ++s) tc::mbar_init(&full_w[s], 1);   // full and empty of both rings
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(&acc_full[s], 1);
      tc::mbar_init(&acc_free[s], 16);
    }
    tc::mbar_init(last, 1);
    mark[0] = 0;
    mark[1] = mark[2] = kPairRunning;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc::smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc::fence_before();
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;
  const PairWaits wait(mark, status, 2 * p.splits);
  pdl_wait();
  pdl_launch_dependents();
  const int tiles = (p.pair_tile ? __ldg(&p.pair_tile[0].x) : p.pair_tok) * p.pair_m;

  if (warp == 0 || warp == kPairWarps - 1) {
    // ===== fetch weights (warp 0), tokens (the last one): the whole warp walks the loop, one lane issues =====
    const bool issuer = elect_one();
    auto fetch = [&](auto ring) {
      constexpr int RING = decltype(ring)::value, STAGES = RING ? kPairXStages : kPairWStages;
      uint64_t *full = RING ? full_x : full_w, *empty = RING ? empty_x : empty_w;
      unsigned char* slots = smem + RING * kPairWStages * kPairABytes;
      if (issuer) {
        if (RING == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        else if (!p.pair_tile) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x[(p.pair_n >> 5) - 1]) : "memory");
      }
      int it = 0;
      for (int t = first; t < tiles; t += step) {
        const PairTile tile = pair_tile(p, t);
        const int half = tile.n >> 1, x0 = tile.row0 + rank * half, m = 2 * tile.m + rank;
        const int w0 = tile.expert * p.n_out + m * kBlockM;
        const CUtensorMap* map_x = &maps.x[(tile.n >> 5) - 1];
        const uint32_t bytes = RING ? (uint32_t)(tile.n * kBlockK * 2) : (uint32_t)(2 * kPairABytes);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int st = it % STAGES;
          if (it >= STAGES && !wait.all(&empty[st], (it / STAGES - 1) & 1)) break;
          if (issuer) {
            unsigned char* dst = slots + st * kPairABytes;
            const uint32_t bar = smem_of(&full[st], lead);
            if (rank == 0) tc::mbar_expect_tx(&full[st], bytes);
            if (RING) pair_load(dst, map_x, kb * kBlockK, x0, bar, kKeepLast);
            else if (p.gu_ff) pair_load3(dst, &map_w, kb * kBlockK, m * (kBlockM / 2), 2 * tile.expert, bar, kKeepNormal);   // 64 gate rows, then the matching up rows
            else pair_load(dst, &map_w, kb * kBlockK, w0, bar, kKeepNormal);
          }
          __syncwarp();
          if (wait.stop()) {
            ++it;   // (this fill too)
            break;
          }
        }
        if (wait.stop()) break;
      }
      if (issuer) *reinterpret_cast<volatile uint32_t*>(mark + 1 + RING) = (uint32_t)it;
    };
    if (warp == 0) fetch(std::integral_constant<int, 0>());
    else fetch(std::integral_constant<int, 1>());
  } else if (warp == 1) {
    // ===== the leader's MMA warp: instructions predicated to one lane in convergent code =====
    if (rank == 0) {
      const uint32_t one = elect_one();
      const uint16_t both = (uint16_t)(3 << lead);
      const uint64_t desc0 = tc::make_desc(tc::smem_u32(smem), 16, 1024);
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const int n_tiles = __shfl_sync(0xffffffffu, tiles, 0);
      int i = 0, sw = 0, sx = 0;
      uint32_t ph_w = 0, ph_x = 0;
      for (int t = first; t < n_tiles; t += step, ++i) {
        const int n = __shfl_sync(0xffffffffu, pair_tile(p, t).n, 0);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(2 * kBlockM >> 4) << 24);
        const uint32_t acc = tm + (uint32_t)((i & 1) * 256);
        if (i >= 2) wait(&acc_free[i & 1], ((i >> 1) - 1) & 1);
        tc::fence_after();
        for (int kb = kb0; kb < kb1; ++kb) {
          wait(&full_x[sx], ph_x, [&] { pair_await_ends(mark, lead, wait.limit); });
          wait(&full_w[sw], ph_w, [&] { pair_await_ends(mark, lead, wait.limit); });
          tc::fence_after();
          const uint64_t da = desc0 + (uint64_t)((sw * kPairABytes) >> 4), db = desc0 + (uint64_t)(((kPairWStages + sx) * kPairABytes) >> 4);
          const uint32_t more = kb > kb0 ? 1u : 0u;
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)   // 16 of k are 32 bytes inside the swizzle's span
            pair_mma(one, acc, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, k ? 1u : more);
          pair_commit(one, &empty_w[sw], both);
          pair_commit(one, &empty_x[sx], both);
          if (++sw == kPairWStages) sw = 0, ph_w ^= 1;
          if (++sx == kPairXStages) sx = 0, ph_x ^= 1;
        }
        pair_commit(one, &acc_full[i & 1], both);
        if (wait.stop()) break;
      }
      if (wait.stop()) {
        pair_commit(one, last, (uint16_t)(1 << lead));
        wait.drain(last, 0);
      }
    }
  } else {
    // ===== epilogue: two groups of four warps take pieces of 32 tokens in turn =====
    const int quad = warp & 3, grp = (warp - 2) >> 2, wq = (warp - 2) & 3, srow = quad * 32 + lane, r4 = lane * 4;
    float* stg = stg_all + grp * (kPairStgBytes / 4);
    float* whole = reinterpret_cast<float*>(smem);   // with k split: the pair's sums of the tile, [token][128]
    const int barrier = 1 + grp;
    int i = 0, turn = 0;   // turn: the half of the staging area that the next straight piece takes
    for (int t = first; t < tiles; t += step, ++i) {
      const PairTile tile = pair_tile(p, t);
      const int m_tile = 2 * tile.m + rank;
      const int n_rows = p.pair_tile ? tile.n : min(tile.n, p.T - tile.row0);
      const bool live = (p.gu_ff ? m_tile * (kBlockM / 2) < p.gu_ff : m_tile * kBlockM < p.n_out) && !wait.marked();
      float bb[4], gate_bias[4], up_bias[4];
      pair_bias(p, m_tile, r4, bb);
      if constexpr (MODE == kSiluMul) {   // of the features that the lane finishes
        pair_bias(p, m_tile, (quad & 1) * 32 + (lane & 7) * 4, gate_bias);
        pair_bias(p, m_tile, 64 + (quad & 1) * 32 + (lane & 7) * 4, up_bias);
      }
      // A whole slab of plain outputs in rows of 16-byte pieces: rounded by the thread that reads them from tensor memory and staged as they are written, 32 tokens in
      // either half of the staging area in turn (one barrier a piece).  A quarter of the instructions that four features at a time take, which is what launches over
      // short k are bound by: 2048 tokens, 4096 features, k 512 24.9 us, so 16.9 (20.8 in tiles of 128 x 256, two CTAs to an SM); k 64 24.9, 18.7 (16.7); 1000 tokens
      // of 8192 features, k 256 23.9, 16.9 (18.7); and 2048 tokens, 28672 features, k 4096 349, 340.
      // (squared: the activation of two-matrix experts)
      const bool squared = MODE == kPlain && p.post_act == 1 + B200_ACT_RELU2;
      const bool straight = MODE == kPlain && p.splits == 1 && (p.post_act == 0 || squared) && (m_tile + 1) * kBlockM <= p.n_out && p.ldy % 8 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
      const float bias = straight && p.bias ? __bfloat162float(p.bias[m_tile * kBlockM + srow]) : 0.f;
      __nv_bfloat16* const y0 = straight ? p.y + (int64_t)tile.row0 * p.ldy + m_tile * kBlockM + (lane & 15) * 8 : nullptr;
      if (MODE == kRopeKv) {   // a token's cos|sin row is a dependent load: ask for the tile's rows while its MMAs run
        const int tt = (warp - 2) * 32 + lane;
        if (tt < n_rows) {
          const char* row = reinterpret_cast<const char*>(p.cos_sin + (int64_t)p.positions[tile.row0 + tt] * kHeadDim);
          asm volatile("prefetch.global.L1 [%0];" ::"l"(row));
          asm volatile("prefetch.global.L1 [%0];" ::"l"(row + 128));
        }
      }
      wait(&acc_full[i & 1], (i >> 1) & 1);
      tc::fence_after();
      const uint32_t taddr = tmem + (uint32_t)((i & 1) * 256) + ((uint32_t)(quad * 32) << 16);
      if (MODE == kPlain && p.splits == 1 && !straight) asm volatile("bar.sync %0, 128;" ::"r"(barrier) : "memory");   // (the tile before may have been)
      for (int c = grp * kPairStgTok; c < tile.n; c += 2 * kPairStgTok) {
        int pair = -1;   // kScatter: lane l holds the destination and weight of the piece's token l
        float wt = 1.0f;
        if (MODE == kScatter && c + lane < n_rows) {
          pair = p.grp_pair ? __ldg(p.grp_pair + tile.row0 + c + lane) : tile.row0 + c + lane;
          if (pair >= 0 && p.grp_wt) wt = __ldg(p.grp_wt + pair);
        }
        uint32_t r[32];
        tmem_ld32(taddr + c, r);
        if (p.splits > 1) {   // one tile a pair: its stages are free by now
#pragma unroll
          for (int j = 0; j < 32; ++j) whole[(c + j) * kBlockM + srow] = __uint_as_float(r[j]);
          continue;
        }
        if (MODE == kPlain && straight) {
          __nv_bfloat16* half = reinterpret_cast<__nv_bfloat16*>(stg) + turn * kPairStgTok * kBlockM;
          turn ^= 1;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float v = __uint_as_float(r[j]) + bias, o = squared ? fmaxf(v, 0.f) * fmaxf(v, 0.f) : v;
            half[j * kBlockM + srow] = __float2bfloat16_rn(o);
          }
          asm volatile("bar.sync %0, 128;" ::"r"(barrier) : "memory");
#pragma unroll
          for (int j = wq * 8 + (lane >> 4); j < wq * 8 + 8; j += 2)   // two tokens a warp and step
            if (live && c + j < n_rows) *reinterpret_cast<uint4*>(y0 + (int64_t)(c + j) * p.ldy) = *reinterpret_cast<const uint4*>(half + j * kBlockM + (lane & 15) * 8);
          continue;
        }
        // Products with an activation and scattered rows: a warp turns its 32 features x 32 tokens in 4 KiB of its own (a token's 16-byte pieces swapped by its number),
        // eight lanes a token, and every lane's values are worked out side by side, with the stores alone depending on the token.  (Four warps' features together behind two
        // barriers, token after token with a branch each: 21 000 cycles a tile of gate|up and 12 000 of scattered rows, more than the tile's MMAs take;
        // 2 048 rows of 32 experts, router and
        // grouping included, 167 us, so 154; 1 527 rows of 64 without a gate 229, 218.)
        float4* const own = reinterpret_cast<float4*>(stg_all) + (grp * 4 + quad) * (kPairStgTok * 8);
        const int tok_of = lane >> 3, piece = lane & 7;
        if constexpr (MODE == kScatter || MODE == kSiluMul) {
          float* const cell = reinterpret_cast<float*>(own) + (lane & 3);
#pragma unroll
          for (int j = 0; j < 32; ++j) cell[(j * 8 + ((lane >> 2) ^ (j & 7))) * 4] = __uint_as_float(r[j]);
        }
        if constexpr (MODE == kScatter) {
          __syncwarp();
          const int row = m_tile * kBlockM + quad * 32 + piece * 4;
          const bool wide = row + 3 < p.n_out && p.n_out % 4 == 0;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int j = 4 * i + tok_of, to = __shfl_sync(0xffffffffu, pair, j);
            const float w = __shfl_sync(0xffffffffu, wt, j);
            const float4 a = own[j * 8 + (piece ^ (j & 7))];
            const float o[4] = {a.x * w, a.y * w, a.z * w, a.w * w};
            float* dst = p.grp_out + (int64_t)to * p.n_out + row;
            if (!live || to < 0) continue;   // (rows past the run's end have no destination)
            if (wide) {
              *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (row + e < p.n_out) dst[e] = o[e];
            }
          }
          __syncwarp();
          continue;
        }
        if constexpr (MODE == kSiluMul) {
          // gate rows with one warp, the matching up rows with another: each finishes half of the tokens
          const int feat = quad & 1, shared_by = 1 + 2 * grp + feat;
          asm volatile("bar.sync %0, 64;" ::"r"(shared_by) : "memory");
          const float4 *gates = reinterpret_cast<const float4*>(stg_all) + (grp * 4 + feat) * (kPairStgTok * 8), *ups = gates + 2 * kPairStgTok * 8;
          const int f = m_tile * 64 + feat * 32 + piece * 4;
          const bool wide = p.ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0;
          float o[4][4];
          auto finish = [&](auto kind) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int j = (quad >> 1) * 16 + 4 * i + tok_of;
              const float4 ga = gates[j * 8 + (piece ^ (j & 7))], ua = ups[j * 8 + (piece ^ (j & 7))];
              const float gv[4] = {ga.x, ga.y, ga.z, ga.w}, uv[4] = {ua.x, ua.y, ua.z, ua.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float g = round_bf16(gv[e] + gate_bias[e]), u = round_bf16(uv[e] + up_bias[e]);
                o[i][e] = kind == 0 ? silu_to_bf16(g) * u : gate_combine(g, u, kind, p.act_limit);
              }
            }
          };
          if (p.act == 0) finish(std::integral_constant<int, 0>());   // (the choice outside the loops)
          else finish(p.act);
          asm volatile("bar.sync %0, 64;" ::"r"(shared_by) : "memory");
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int t = c + (quad >> 1) * 16 + 4 * i + tok_of;
            if (!live || t >= n_rows) continue;
            __nv_bfloat16* dst = p.y + (int64_t)(tile.row0 + t) * p.ldy + f;
            if (wide) {
              *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(o[i][0], o[i][1]), pack_bf16(o[i][2], o[i][3]));
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16_rn(o[i][e]);
            }
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) stg[j * kBlockM + srow] = __uint_as_float(r[j]);
        asm volatile("bar.sync %0, 128;" ::"r"(barrier) : "memory");
        if (live) {
#pragma unroll 4
          for (int j = wq; j < kPairStgTok; j += 4) {
            if (c + j >= n_rows) break;   // warp-uniform
            const float4 a = *reinterpret_cast<const float4*>(stg + j * kBlockM + r4);
            finalize4<MODE>(p, m_tile, lane, tile.row0 + c + j, a, bb);
          }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(barrier) : "memory");
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(smem_of(&acc_free[i & 1], lead)) : "memory");
    }
  }
  if (p.splits > 1) {
    // every pair has the tile's sums over its share of k in shared memory: of the tokens, CTA `split` of a slab adds up and finishes
    // split, split + splits, ..., the shares in their order
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp >= 2 && warp < kPairWarps - 1) {
      const PairTile tile = pair_tile(p, first);
      const int m_tile = 2 * tile.m + rank, r4 = lane * 4, n_rows = min(tile.n, p.T - tile.row0);
      if (m_tile * kBlockM < p.n_out && !wait.marked()) {
        float bb[4];
        pair_bias(p, m_tile, r4, bb);
        constexpr int U = 4;   // tokens whose loads are in flight together
        for (int t0 = split + p.splits * (warp - 2); t0 < n_rows; t0 += U * 8 * p.splits) {
          float4 v[U][kPairSplits];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int t = min(t0 + u * 8 * p.splits, n_rows - 1);
#pragma unroll
            for (int s = 0; s < kPairSplits; ++s)
              if (s < p.splits)
                asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                             : "=f"(v[u][s].x), "=f"(v[u][s].y), "=f"(v[u][s].z), "=f"(v[u][s].w)
                             : "r"(smem_of(smem, 2 * s + rank) + (uint32_t)(t * kBlockM + r4) * 4u)
                             : "memory");
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int t = t0 + u * 8 * p.splits;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int s = 0; s < kPairSplits; ++s)
              if (s < p.splits) a.x += v[u][s].x, a.y += v[u][s].y, a.z += v[u][s].z, a.w += v[u][s].w;
            if (t < n_rows) finalize4<MODE>(p, m_tile, lane, tile.row0 + t, a, bb, tile.row0 + t);   // warp-uniform
          }
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // a CTA's shared and tensor memory serve the other's MMAs
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (wait.marked()) {   // the same answer in all CTAs of the cluster, whose waits have ended
    if (rank == 0 && threadIdx.x == 0) pair_land(wait, full_w, full_x, p, mark, lead, kb1 - kb0, first, step);
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  tc::fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

template <int MODE>
int launch_pair(const CUtensorMap& mw, const PairMaps& mx, const TcParams& p, int clusters, cudaStream_t s) {
  static bool attr_set[64] = {};
  B200_CUDA(ensure_dynamic_smem(linear_pair_kernel<MODE>, kPairSmem, attr_set));
  B200_CUDA(launch_cluster(linear_pair_kernel<MODE>, dim3(clusters * 2 * p.splits), dim3(kPairThreads), (size_t)kPairSmem, s, dim3(2 * p.splits, 1, 1), mw, mx, p, wait_status_word()));
  return B200_OK;
}

}  // namespace

// Tokens a tile and shares of k by an estimate of the launch's cycles: whole waves of tiles over the clusters that fit the GPU at a time, a tile per 64
// of k its MMAs (2 cycles a token) or its loads (256 + tokens rows of 128 bytes at 64 bytes a cycle and SM, two SMs), the last tile's epilogue and,
// where k is shared, the exchange.
PairPlan linear_pair_plan(int T, int n_out, int k) {
  constexpr int kActive[kPairSplits + 1] = {0, 74, 33, 22, 15};   // clusters of 2, 4, 6, 8 such CTAs that run at a time (cudaOccupancyMaxActiveClusters)
  const int m = (n_out + 2 * kBlockM - 1) / (2 * kBlockM), kbs = (k + kBlockK - 1) / kBlockK;
  PairPlan best = {0, 1};
  int64_t best_cost = 0;
  for (int n = 256; n >= 32; n -= 32) {
    const int64_t tiles = (int64_t)m * ((T + n - 1) / n);
    for (int s = 1; s <= kPairSplits; ++s) {
      if (s > 1 && (tiles > kActive[s] || kbs / s < 4)) continue;
      const int64_t c = (tiles + kActive[s] - 1) / kActive[s] * ((kbs + s - 1) / s) * std::max(2 * n, 256 + n) + 20 * std::min(n, T) + (s > 1 ? 800 + 800 * s : 0);
      if (best.n == 0 || c < best_cost) best = {n, s}, best_cost = c;
    }
  }
  return best;
}

int linear_pair(int mode, TcParams p, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int k, PairPlan pl, cudaStream_t s) {
  if (const int e = wait_status()) return e;
  p.pair_n = pl.n;
  p.splits = pl.splits;
  p.pair_tok = (p.T + pl.n - 1) / pl.n;
  p.pair_m = (p.n_out + 2 * kBlockM - 1) / (2 * kBlockM);
  p.pair_group = (p.pair_tok + (p.pair_tok + 8) / 9 - 1) / ((p.pair_tok + 8) / 9);
  CUtensorMap mw;
  PairMaps mx = {};
  int rc = get_tensor_map_2d(w, (uint64_t)p.n_out, (uint64_t)k, (uint64_t)k, kBlockM, &mw);
  if (rc) return rc;
  rc = get_tensor_map_2d(x, (uint64_t)p.T, (uint64_t)k, (uint64_t)ldx, (uint32_t)pl.n / 2, &mx.x[pl.n / 32 - 1]);
  if (rc) return rc;
  const int clusters = (int)std::min<int64_t>((int64_t)p.pair_tok * p.pair_m, kNumSMs / 2);
  switch (mode) {
    case kScatter: return launch_pair<kScatter>(mw, mx, p, clusters, s);
    case kSiluMul: return launch_pair<kSiluMul>(mw, mx, p, clusters, s);
    case kRopeKv: return launch_pair<kRopeKv>(mw, mx, p, clusters, s);
    default: return launch_pair<kPlain>(mw, mx, p, clusters, s);
  }
}

// ---- grouped form ----------------------------------------------------------------------------------------------------------
static int launch_grouped_pair(int mode, TcParams p, const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int k,
                               cudaStream_t s) {
  B200_REQUIRE(x && w && g.tiles && k > 0 && k % 8 == 0 && ldx % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0,
               B200_ERR_INVALID, "grouped linear: operands in rows of 16-byte pieces");
  if (const int e = wait_status()) return e;
  p.T = (int)g.rows;
  p.n_kblocks = (k + kBlockK - 1) / kBlockK;
  p.splits = 1;
  p.pair_tile = g.tiles;
  CUtensorMap mw;
  PairMaps mx;
  int rc = p.gu_ff ? get_tensor_map_3d(w, 2u * (uint32_t)g.experts, (uint64_t)p.gu_ff, (uint64_t)k, kBlockM / 2, &mw)
                   : get_tensor_map_2d(w, (uint64_t)g.experts * p.n_out, (uint64_t)k, (uint64_t)k, kBlockM, &mw);
  for (int i = 0; i < 8 && !rc; ++i) rc = get_tensor_map_2d(x, (uint64_t)g.rows, (uint64_t)k, (uint64_t)ldx, 16 * (i + 1), &mx.x[i]);
  if (rc) return rc;
  const int clusters = (int)std::min<int64_t>((int64_t)g.max_tiles * p.pair_m, kNumSMs / 2);
  switch (mode) {
    case kScatter: return launch_pair<kScatter>(mw, mx, p, clusters, s);
    case kSiluMul: return launch_pair<kSiluMul>(mw, mx, p, clusters, s);
    default: return launch_pair<kPlain>(mw, mx, p, clusters, s);
  }
}

int linear_pair_grouped(const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int n_out, int k, __nv_bfloat16* y, int64_t ldy,
                        cudaStream_t s, int post_act) {
  TcParams p = {};
  p.y = y;
  p.ldy = ldy;
  p.n_out = n_out;
  p.post_act = post_act;
  p.pair_m = (n_out + 2 * kBlockM - 1) / (2 * kBlockM);
  return launch_grouped_pair(kPlain, p, g, x, ldx, w, k, s);
}

int linear_pair_gate_up(const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int ff, int k, __nv_bfloat16* y, cudaStream_t s,
                        int act, float act_limit) {
  B200_REQUIRE(ff > 0 && ff % (kBlockM / 2) == 0, B200_ERR_UNSUPPORTED, "grouped gate|up: ff=%d must be a multiple of 64", ff);
  TcParams p = {};
  p.y = y;
  p.ldy = ff;
  p.n_out = 2 * ff;
  p.gu_ff = ff;
  p.act = act;
  p.act_limit = act_limit;
  p.pair_m = (ff + kBlockM - 1) / kBlockM;
  return launch_grouped_pair(kSiluMul, p, g, x, ldx, w, k, s);
}

int linear_pair_scatter(const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int n_out, int k, const int32_t* row_pair,
                        const float* wts, float* out, cudaStream_t s) {
  B200_REQUIRE(row_pair && wts && out && reinterpret_cast<uintptr_t>(out) % 16 == 0, B200_ERR_INVALID, "grouped linear: no destination");
  TcParams p = {};
  p.n_out = n_out;
  p.grp_pair = row_pair;
  p.grp_wt = wts;
  p.grp_out = out;
  p.pair_m = (n_out + 2 * kBlockM - 1) / (2 * kBlockM);
  return launch_grouped_pair(kScatter, p, g, x, ldx, w, k, s);
}

}  // namespace b200
