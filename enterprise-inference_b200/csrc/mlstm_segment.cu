// The matrix-memory recurrence of mlstm.cu over longer portions on tcgen05 (bf16 rows), cut in time over the CTAs of a cluster.
//
// With F_t the sum of the log forget gates up to row t of a segment, M_t = max_{s<=t} (i_s - F_s) and m_t = F_t + max(m_0, M_t), which is the running maximum
// of the row-by-row walk,
//   S_t = exp(F_t + m_0 - m_t) S_0 + exp(F_t + M_t - m_t) sum_{s<=t} exp(i_s - F_s - M_t) k_s v_s^T          (n_t likewise with v = 1)
// so a segment needs S_0, n_0 and m_0 of the rows before it, and neither what it adds to them nor its own sums depend on them.
//
// A cluster of four CTAs takes (sequence, head, 64 value columns), up to 1 024 rows at a time, each CTA a segment of up to 256:
//   1. sums F and maxima M of its gates; D = K^T (w V) with w_s = exp(i_s - F_s - M_L), the segment's own part of the state (M: dimensions, N: columns);
//   2. outputs as attention within the segment: scores Q K^T in blocks of 128 rows x 128 keys, weighted by the exponentials under the diagonal, times V;
//   3. every CTA reads the earlier segments' D from the output rows where they left it (their own, not written yet; it stays in L2) and adds up its S_0 (the last one
//      the state after all): Q S_0.
// Nothing walks from chunk to chunk.  Everything that was fp32 in the walk stays so in effect: sums F are taken in 64 bits (differences of large
// sums), an fp32 operand (weights, w V, S_0) enters the bf16 MMA as three bf16 terms (24 bits) against rows that are bf16 to begin with, the small
// terms first, accumulators are fp32 and short: D has two, of every other 64 rows each (128 at most), outputs one for every 128 keys, scores one for either half of the dimensions.
// Weights of a row on 32 keys that all lie before it are the product of two exponentials around the keys' maximum, one a row and one a key; only blocks on the diagonal take
// one a pair (there a later row's key may be the maximum, and the product overflow).
// A value that is not finite is taken out of V before the products (0 times it would reach earlier rows); its column is NaN from its row on.
//
// Why tcgen05, and segments: in chunks of 64 rows on mma.sync (mlstm_chunk.cuh) 2 048 rows of 8 heads, 128 x 256, are 32 dependent chunks of 4.4 us; the same
// segments on mma.sync took 103 us, because m16n8k16 takes 16 cycles of a scheduler here (three terms of everything: 92 000 cycles).
// What bounds it now: the instructions of a round (45 000 issue slots a scheduler for two rounds, a third of the stalls are instruction fetches,
// hence loops that stay loops, one copy of each phase), and the phases' latency, one CTA an SM.  2 048 rows of 8 heads, 128 x 256: 142 -> 57 us; 1 024: 73 -> 31;
// 512: 38 -> 21; 8 000 rows 545 -> 220; 64 x 128: 114 -> 54.
// Error of the results against 64 bits, over 32 cases: 5.1e-7 (chunks 5.6e-7), of the state 6.8e-8 (7.8e-8); scores in one accumulator would
// make it 6.0e-7 (eight truncated sums of 16 dimensions), weights by expf 6.4e-7.
// Tried: eight warps instead of sixteen 68 us; D over the cluster's shared memory 12 000 cycles a round instead of 4 000; the MMAs issued by a warp with rows 65 us.
#include <algorithm>

#include "exp2_of_double.h"
#include "mlstm_chunk.cuh"
#include "tc.cuh"

namespace b200 {

uint32_t* wait_status_word();
int wait_status();

namespace {

using namespace tc;

constexpr int kSgCluster = 4, kSgRows = 256, kSgCols = 64;   // CTAs of a cluster; rows of a segment; value columns
constexpr int kSgResident = 33;   // clusters of four CTAs, one an SM, that run at a time (cudaOccupancyMaxActiveClusters: 132 of the 148 SMs)
constexpr int kSgThreads = 512, kSgAll = kSgThreads + 128;   // sixteen warps, and a group of four of which one issues the MMAs
// registers a thread: 640 threads are launched with 96 each; four warps give what the sixteen others take (16 x 104 + 4 x 64 = 20 x 96)
constexpr int kSgRegs = 104, kSgRegsMma = 64;
static_assert(16 * kSgRegs + 4 * kSgRegsMma <= 20 * 96, "registers of the launch");
constexpr int kSgRegsChunks = 184, kSgRegsGate = 64, kSgRegsRest = 24;   // portions in chunks: eight warps with rows, four of which one has the gates, eight others
static_assert(8 * kSgRegsChunks + 4 * kSgRegsGate + 8 * kSgRegsRest <= 20 * 96, "registers of the launch");
static_assert(kSgThreads >= kScanThreads && 2 * kScanCols == kSgCols, "the walk takes a cluster's columns with two of its CTAs");
constexpr int kSgPanel = kSgRows * 128, kSgTile = 128 * 128;   // bytes of 64 dimensions (columns) of a segment's rows; of 128 rows of them
// Tensor memory columns: a block's scores on either half of the dimensions; in the first one's place its weights (32 keys: 16 columns of first
// terms, 16 of second ones) and later Q S_0 of either row tile; third terms; O of the first row tile and of the second one's two key blocks, in the
// latter's place D's two accumulators before.
constexpr int kTmHalf = 128, kTmE = 256, kTmO = 320, kTmD = 384;

// Staged rows as SWIZZLE_128B has them: panels of 64 dimensions (columns), rows of 128 bytes whose 16-byte pieces are swapped by the row's number.
__device__ __forceinline__ unsigned char* sg_at(unsigned char* x, int row, int piece) {
  return x + (piece >> 3) * kSgPanel + row * 128 + (((piece ^ row) & 7) << 4);
}
// barriers (what an MMA reads from shared memory is behind one whose arrivals follow the writes, copies included, and a fence to the async proxy).  By the MMA warp: scores of a block, D of a half's rows, weights of a block multiplied, the last ones, Q S_0
// (sixteen warps wait); by those: a half of w V is there, weights of a block are, S_0 is there
enum { kScores, kD, kPv, kPvLast, kQs, kEnd, kWeighed, kWeights, kTerms, kBars };   // kEnd: after a wait that ran out, every MMA issued
constexpr double kLog2e = 1.4426950408889634;
struct SgSmall {
  double F[kSgRows], M[kSgRows], G[kSgRows];   // sums, running maxima of G, i - F (M and G times log2 e)
  double gm[8];                                // the largest G of 32 rows
  double part[2][8], fl[kSgCluster], ml[kSgCluster];   // F and M of the segments' last rows
  float w[kSgRows], c[kSgRows];                // exp(G - ml), exp(G - gm)
  float psum[4][kSgRows], qn[2][kSgRows];      // of the weights; q . n_0 on either half of the dimensions
  float dn[kSgCluster][128], n[128];           // the segments' parts of n; n_0
  int odd_from[kSgCols], odd;                  // first row whose value in the column is not finite; any
  uint64_t bar[kBars];
  uint32_t tmem, mark;
};
template <int KS>
struct SgSmem {   // offsets from a 1 024-byte boundary
  static constexpr int k = 0, q = k + (KS / 4) * kSgPanel, v = q + (KS / 4) * kSgPanel, r = v + kSgPanel;
  static constexpr int small = r + 3 * kSgTile, bytes = small + (int)sizeof(SgSmall) + 1024;
};
static_assert(SgSmem<8>::bytes <= 232448, "shared memory");

__device__ __forceinline__ void sg_st4(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void sg_ld8(uint32_t taddr, float* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ uint32_t sg_remote(const void* p, uint32_t rank) {
  uint32_t to;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(p)), "r"(rank));
  return to;
}
__device__ __forceinline__ void sg_put(uint32_t at, float x) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(x) : "memory"); }
__device__ __forceinline__ void sg_put(uint32_t at, double x) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(x) : "memory"); }
__device__ __forceinline__ void sg_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void sg_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// KS: 16-wide steps over the (zero padded) key dimensions
template <int KS>
__global__ void __launch_bounds__(kSgAll, 1) mlstm_segment_kernel(const MlstmArgs a, uint32_t* status) {
  extern __shared__ __align__(16) unsigned char raw[];
  using L = SgSmem<KS>;
  constexpr int PIECES = KS * 2;   // 16-byte pieces of a q or k row
  unsigned char* smem = raw + (-smem_u32(raw) & 1023);   // (an offset: rounded as an address it would be a generic one, 64 bits and a slower load each time)
  SgSmall& sm = *reinterpret_cast<SgSmall*>(smem + L::small);

  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, rank = blockIdx.z % kSgCluster, cb = blockIdx.z / kSgCluster, jb = cb * kSgCols;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int heads = a.heads, dim = a.dim, vd = a.vd, nz = (vd + kScanCols - 1) / kScanCols;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows < kChunkFrom) {   // (nothing to do at all among them) two CTAs take the cluster's columns
    if (rank < 2 && 2 * cb + rank < nz && tid < kScanThreads)
      mlstm_walk<__nv_bfloat16, KS / 4>(a, reinterpret_cast<float*>(raw), 2 * cb + rank, nz);
    return;
  }
  if (n_rows < kSegmentFrom) {   // every CTA sixteen columns
    if (warp < kMcGate) {
      asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSgRegsChunks));
      mlstm_chunks<KS, 1>(a, raw, blockIdx.z);
    } else if (warp < kMcGate + 4) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSgRegsGate));
      if (warp == kMcGate) mlstm_chunks<KS, 2>(a, raw, blockIdx.z);
    } else {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSgRegsRest));
    }
    return;
  }
  const Waits mbar_wait(&sm.mark, status);
  if (tid == 0) {
    for (int i = 0; i < kBars; ++i) mbar_init(sm.bar + i, i < kWeighed ? 1 : kSgThreads / 32);
    sm.mark = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kSgThreads / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  sg_arrive();   // (the others' shared memory is written to from here on)
  sg_wait();
  fence_after();
  const uint32_t tm = __shfl_sync(0xffffffffu, sm.tmem, 0);
  uint32_t phases = 0;
  auto wait = [&](int b) {
    mbar_wait(sm.bar + b, (phases >> b) & 1);
    phases ^= 1u << b;
    fence_after();
  };
  // segments of equal length (128 rows at least: a row tile's time does not depend on its rows), rounds of four of them
  const int rounds = (n_rows - 1) / (kSgCluster * kSgRows) + 1, per_round = (n_rows + rounds - 1) / rounds;
  const int SL = max(128, (per_round + kSgCluster * 16 - 1) / (kSgCluster * 16) * 16);

  if (warp >= kSgThreads / 32) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSgRegsMma));
    if (warp > kSgThreads / 32) return;
    // ===== MMAs =====
    const uint32_t one = elect_one() ? 1u : 0u;
    // descriptors (groups of eight rows 1 024 bytes apart; the next 64 of M or N, where they run along the rows, a panel away) of what starts at an
    // offset; the address's higher bits, which have the CTA of the cluster, are not theirs
    const uint32_t desc0 = ((smem_u32(smem) & 0x3ffff) >> 4) + ((kSgPanel >> 4) << 16);
    auto desc = [&](uint32_t at) { return (uint64_t)(desc0 + (at >> 4)) | ((uint64_t)((1024 >> 4) | (1u << 14) | (2u << 29)) << 32); };
    constexpr uint32_t kIdS = idesc_bf16(128, 0), kIdO = idesc_bf16(kSgCols, 1), kIdD = kIdO | (1u << 15);   // (K^T: M runs along the rows)
    auto scores = [&](int tile, int block) {
#pragma unroll
      for (int j = 0; j < KS; ++j)
        mma_ss(one, tm + (j < KS / 2 ? 0 : kTmHalf), desc(L::q + (j >> 2) * kSgPanel + tile * kSgTile + (j & 3) * 32),
               desc(L::k + (j >> 2) * kSgPanel + block * kSgTile + (j & 3) * 32), kIdS, j % (KS / 2) ? 1u : 0u);
      commit(one, sm.bar + kScores);
    };
    const int first = a.positions[start];
    for (int base = 0; base < n_rows; base += kSgCluster * SL) {
      const int n16 = (max(0, min(SL, n_rows - base - rank * SL)) + 15) & ~15;
      const bool two = n16 > 128;
      sg_arrive();   // (nothing to show: the others do not wait for the last products' issue)
#pragma unroll 1
      for (int step = 0; step < (n16 ? two ? 3 : 1 : 0); ++step) {   // the first tile, the second on the first block of keys, on its own
        if (step < 2) {
          wait(kWeighed);
          if (step == 0) scores(0, 0);
          // D of up to 128 rows, an accumulator for every other 64
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int steps = (n16 - step * 128 - x * 64) >> 4;
#pragma unroll
            for (int i = 2; i >= 0; --i)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                mma_ss(j < steps ? one : 0u, tm + kTmD + x * 64, desc(L::k + (step * 128 + x * 64 + j * 16) * 128),
                       desc(L::r + i * kSgTile + (x * 64 + j * 16) * 128), kIdD, step || i < 2 || j ? 1u : 0u);
          }
          commit(one, sm.bar + kD);
        }
        wait(kWeights);
        const int steps = (n16 - (step >> 1) * 128) >> 4;
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          const uint32_t weights = tm + (i == 2 ? kTmE : i * 16), next = i == 2 ? 16 : 32;   // 32 keys of a term
#pragma unroll
          for (int j = 0; j < 8; ++j)
            mma_ts(j < steps ? one : 0u, tm + kTmO + step * 64, weights + (j >> 1) * next + (j & 1) * 8, desc(L::v + ((step >> 1) * 128 + j * 16) * 128), kIdO,
                   i < 2 || j ? 1u : 0u);
        }
        commit(one, sm.bar + (step == (two ? 2 : 0) ? kPvLast : kPv));
        if (two && step < 2) scores(1, step);
      }
      sg_wait();
      sg_arrive();
      sg_wait();
      if (n16 && !(first == 0 && base == 0 && rank == 0)) {
        wait(kTerms);
#pragma unroll 1
        for (int tile = 0; tile <= (two ? 1 : 0); ++tile)
#pragma unroll
          for (int i = 2; i >= 0; --i)
#pragma unroll
            for (int j = 0; j < KS; ++j)
              mma_ss(one, tm + tile * 64, desc(L::q + (j >> 2) * kSgPanel + tile * kSgTile + (j & 3) * 32), desc(L::r + i * kSgTile + j * 2048), kIdO,
                     i < 2 || j ? 1u : 0u);
        commit(one, sm.bar + kQs);
      }
    }
    __syncthreads();
    if (mbar_wait.stop()) {   // a wait ran out (all roles are at their ends): what is in flight finishes before tensor and shared memory are given up
      commit(one, sm.bar + kEnd);
      mbar_wait.drain(sm.bar + kEnd, 0);
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(512u));
    return;
  }

  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSgRegs));
  // ===== sixteen warps: rows, gates, weights, state, outputs =====
  auto sync = [] { asm volatile("bar.sync 1, 512;" ::: "memory"); };
  auto arrive = [&](int b) {
    __syncwarp();
    if (lane == 0) mbar_arrive(sm.bar + b);
  };
  const int first = a.positions[start], slot = a.seq_slots[s];
  // a thread's place in tensor memory: lane 32 quad + lane (a row of a tile, a dimension of the state), sixteen columns from 16 part on
  const int quad = warp & 3, part = warp >> 2, ml = quad * 32 + lane;
  const uint32_t tl = tm + ((uint32_t)(quad * 32) << 16);
  const int width = min(vd - jb, kSgCols), cols = min(width - part * 16, 16);   // columns that exist, of the CTA and the thread (multiples of 8, or none)
  const bool wide = a.vec_out && width == kSgCols;

  for (int base = 0; base < n_rows; base += kSgCluster * SL) {
    const int r0 = base + rank * SL, nl = max(0, min(SL, n_rows - r0)), n16 = (nl + 15) & ~15;   // this CTA's rows
    const int last = (min(kSgCluster * SL, n_rows - base) - 1) / SL;                              // the last CTA with rows
    const bool two = n16 > 128;
    if (nl == 0) {
      sg_arrive();
      sg_wait();
      sg_arrive();
      sg_wait();
      continue;
    }
    // ---- rows: k and v of the first 128, of the others, q ----
    float ig = -INFINITY, fg = 0.f;   // rows past the end: no weight, no decay
    if (tid < nl) {
      const float* p = a.gates + (int64_t)(start + r0 + tid) * 2 * heads + h;
      ig = p[0];
      fg = p[heads];
    }
    if (tid < kSgCols) sm.odd_from[tid] = kSgRows;
    if (tid == 0) sm.odd = 0;
    {
      const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.qkv) + (int64_t)(start + r0) * a.ld;
      const int p = tid % PIECES, r_of = tid / PIECES, pv = tid & 7, rv_of = tid >> 3;
      const bool live = p * 8 < dim, live_v = jb + pv * 8 < vd;
      const __nv_bfloat16* row = src + h * dim + (live ? p * 8 : 0);
      auto fetch = [&](int at, int off, int from, int to) {
#pragma unroll 4
        for (int r = from + r_of; r < to; r += kSgThreads / PIECES) {
          const bool ok = live && r < nl;
          cp16z(sg_at(smem + at, r, p), row + (ok ? (int64_t)r * a.ld : 0) + off, ok);
        }
      };
      const __nv_bfloat16* row_v = src + a.v_off + h * vd + (live_v ? jb + pv * 8 : 0);
      auto fetch_v = [&](int from, int to) {
#pragma unroll 2
        for (int r = from + rv_of; r < to; r += kSgThreads / 8) {
          const bool ok = live_v && r < nl;
          cp16z(sg_at(smem + L::v, r, pv), row_v + (ok ? (int64_t)r * a.ld : 0), ok);
        }
      };
#pragma unroll 1
      for (int from = 0; from < 256; from += 128) {   // (groups without rows among them)
        const int to = min(n16, from + 128);
        fetch_v(from, to);
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 1
        for (int x = 0; x < 2; ++x) fetch(x ? L::q : L::k, x ? a.q_off : a.k_off, from, to);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
    }
    // ---- gates: a thread a row ----
    if (warp < 8) {
      double F = fg < -1e5f ? -1e5f : fg;   // (a gate below -1e5 leaves nothing in fp32 either way; NaN stays)
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, F, d);
        if (lane >= d) F += v;
      }
      if (lane == 31) sm.part[0][warp] = F;
      asm volatile("bar.sync 2, 256;" ::: "memory");
      double before = 0.0;
#pragma unroll
      for (int i = 0; i < 7; ++i)
        if (i < warp) before += sm.part[0][i];
      F += before;
      const double G = (double)ig - F;
      double M = G;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, M, d);
        if (lane >= d) M = fmax(M, v);
      }
      const double own = __shfl_sync(0xffffffffu, M, 31);
      if (lane == 31) sm.part[1][warp] = M;
      asm volatile("bar.sync 2, 256;" ::: "memory");
      double all = sm.part[1][0];
#pragma unroll
      for (int i = 1; i < 8; ++i) {
        if (i <= warp) M = fmax(M, sm.part[1][i - 1]);
        all = fmax(all, sm.part[1][i]);
      }
      sm.F[tid] = F;
      const double g2 = G * kLog2e, own2 = own * kLog2e;
      sm.M[tid] = M * kLog2e;
      sm.G[tid] = g2;
      sm.w[tid] = all == -INFINITY ? 0.f : exp2_of_double(g2 - all * kLog2e);
      sm.c[tid] = own == -INFINITY ? 0.f : exp2_of_double(g2 - own2);
      if (lane == 31) sm.gm[warp] = own2;
      if (tid == 255) {
#pragma unroll
        for (int i = 0; i < kSgCluster; ++i) {   // (nobody reads them before the cluster has met)
          sg_put(sg_remote(sm.fl + rank, i), F);
          sg_put(sg_remote(sm.ml + rank, i), all);
        }
      }
    }
    // ---- w V in three terms, 128 rows at a time ----
    auto weigh = [&](int from, int to) {
      const int p = tid & 7;
#pragma unroll 2
      for (int r = from + (tid >> 3); r < to; r += kSgThreads / 8) {
        uint4* at = reinterpret_cast<uint4*>(sg_at(smem + L::v, r, p));
        uint4 v = *at;
        if (odd2(v.x) || odd2(v.y) || odd2(v.z) || odd2(v.w)) {
          auto clean = [&](uint32_t& x, int col) {
            if ((x & 0x7f80u) == 0x7f80u) x &= 0xffff0000u, atomicMin(&sm.odd_from[col], r);
            if ((x & 0x7f800000u) == 0x7f800000u) x &= 0xffffu, atomicMin(&sm.odd_from[col + 1], r);
          };
          sm.odd = 1;
          clean(v.x, p * 8);
          clean(v.y, p * 8 + 2);
          clean(v.z, p * 8 + 4);
          clean(v.w, p * 8 + 6);
          *at = v;
        }
        const float w = sm.w[r];
        uint4 t[3];
        split3(w * bf16lo(v.x), w * bf16hi(v.x), t[0].x, t[1].x, t[2].x);
        split3(w * bf16lo(v.y), w * bf16hi(v.y), t[0].y, t[1].y, t[2].y);
        split3(w * bf16lo(v.z), w * bf16hi(v.z), t[0].z, t[1].z, t[2].z);
        split3(w * bf16lo(v.w), w * bf16hi(v.w), t[0].w, t[1].w, t[2].w);
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(sg_at(smem + L::r + i * kSgTile, r - from, p)) = t[i];
      }
      fence_async_smem();
      arrive(kWeighed);
    };
    asm volatile("cp.async.wait_group 3;" ::: "memory");
    sync();   // the first rows' values, and the gates
    asm volatile("cp.async.wait_group 2;" ::: "memory");   // (k and q too, which the products wait for)
    // ---- outputs within the segment: a warp the weights of 32 rows (quad) on a quarter (part) of each 32 keys of a block ----
    // (the sum of the weights decides how large an output becomes, and may be far below its terms: 64 bits)
    auto weights = [&](int tile, int block, bool wait_e) {
      const double M = sm.M[tile * 128 + ml], mt = (M == -INFINITY ? 0.0 : M) - a.log2_qscale;   // weights times q's scale
      float s[4][8];
      double sum = 0.0;
#pragma unroll
      for (int x = 0; x < 4; x += 2) {
        float s2[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          sg_ld8(tl + (x + i) * 32 + part * 8, s[x + i]);
          sg_ld8(tl + kTmHalf + (x + i) * 32 + part * 8, s2[i]);
        }
        ld_wait<16>(reinterpret_cast<uint32_t*>(s[x]));
        ld_wait<16>(reinterpret_cast<uint32_t*>(s2[0]));
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) s[x + i][j] += s2[i][j];
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int sb = block * 4 + x;   // the keys' group of 32
        if (tile == block && x >= quad) continue;
        const double gm = sm.gm[sb];
        const float w = gm == -INFINITY ? 0.f : exp2_of_double(gm - mt);
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
          const float4 c = *reinterpret_cast<const float4*>(sm.c + sb * 32 + part * 8 + j);
          float* y = s[x] + j;
          y[0] *= w * c.x, y[1] *= w * c.y, y[2] *= w * c.z, y[3] *= w * c.w;
          sum += (double)((y[0] + y[1]) + (y[2] + y[3]));
        }
      }
      if (tile == block) {   // (selected, above the diagonal and on it: a later row's key may be anything)
        float y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float z = quad == 0 ? s[0][j] : quad == 1 ? s[1][j] : quad == 2 ? s[2][j] : s[3][j];
          const float w = exp2_of_double(sm.G[(block * 4 + quad) * 32 + part * 8 + j] - mt);
          y[j] = part * 8 + j <= lane ? z * w : 0.f;
        }
        sum += (double)((y[0] + y[1]) + (y[2] + y[3])) + (double)((y[4] + y[5]) + (y[6] + y[7]));
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int j = 0; j < 8; ++j) s[x][j] = x == quad ? y[j] : x > quad ? 0.f : s[x][j];
      }
      asm volatile("bar.sync %0, 128;" ::"r"(3 + quad) : "memory");   // the four warps of these rows have their scores: weights take their place
      if (wait_e) wait(kPv);   // the block before has been multiplied: its third terms' place is free
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        uint32_t t[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split3(s[x][2 * j], s[x][2 * j + 1], t[0][j], t[1][j], t[2][j]);
        sg_st4(tl + x * 32 + part * 4, t[0]);
        sg_st4(tl + x * 32 + 16 + part * 4, t[1]);
        sg_st4(tl + kTmE + x * 16 + part * 4, t[2]);
      }
      if (tile == 1 && block == 1) sum += (double)sm.psum[part][128 + ml];
      sm.psum[part][tile * 128 + ml] = (float)sum;
      st_wait();
      fence_before();
    };
    // the segment's part of n: a warp eight dimensions, a lane every 32nd row
    auto part_of_n = [&]() {
      if (warp >= PIECES) return;
      float x[8] = {};
#pragma unroll 2
      for (int r = lane; r < nl; r += 32) {
        const uint4 k = *reinterpret_cast<const uint4*>(sg_at(smem + L::k, r, warp));
        const float w = sm.w[r];
        const uint32_t y[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[2 * i] = fmaf(w, bf16lo(y[i]), x[2 * i]);
          x[2 * i + 1] = fmaf(w, bf16hi(y[i]), x[2 * i + 1]);
        }
      }
#pragma unroll
      for (int half = 4; half >= 1; half >>= 1) {   // the lane keeps one half of what it holds
        const bool up = (lane & half) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
          const float keep = up ? x[i + half] : x[i], give = up ? x[i] : x[i + half];
          x[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
      }
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], 8);
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], 16);
      if (lane < 8) {
#pragma unroll
        for (int i = 0; i < kSgCluster; ++i) sg_put(sg_remote(&sm.dn[rank][warp * 8 + lane], i), x[0]);
      }
    };
    float4* X = reinterpret_cast<float4*>(smem + L::r);
    float* scratch = a.out + ((int64_t)(start + base) * heads + h) * vd + jb;   // of the round's first segment
    const int64_t segment = (int64_t)SL * heads * vd;
    auto place = [&](int j) { return (int64_t)(j * 32 + (tid >> 4)) * heads * vd + (tid & 15) * 4; };
    auto place_of = [&](int j) {   // the same of `width` columns (a multiple of 8), whose 128 rows hold what 128 dimensions of them take
      const int pieces = width >> 2, at = (part * 4 + j) * 128 + ml;
      return (int64_t)(at / pieces) * heads * vd + at % pieces * 4;
    };
#pragma unroll 1
    for (int step = 0; step < (two ? 3 : 1); ++step) {
      if (step < 2) {
        if (step) wait(kD);
        weigh(step * 128, min(n16, step * 128 + 128));
      }
      wait(kScores);
      weights(step ? 1 : 0, step >> 1, step > 0);
      if (step == 0) {   // q's second tile too, whose scores are issued behind these weights (k's and v's: kWeighed of the second 128 rows)
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        fence_async_smem();
      }
      if (step != 1) arrive(kWeights);
      if (step == 0) {
        sync();   // all rows
        part_of_n();
      }
      if (step == (two ? 1 : 0)) {
        wait(kD);
        float D[16];
        {
          uint32_t y[2][16];
          ld16(tl + kTmD + part * 16, y[0]);
          ld16(tl + kTmD + 64 + part * 16, y[1]);
          ld_wait<32>(y[0]);
#pragma unroll
          for (int j = 0; j < 16; ++j) D[j] = n16 > 64 ? __uint_as_float(y[0][j]) + __uint_as_float(y[1][j]) : __uint_as_float(y[0][j]);
        }
        fence_before();
        if (step == 1) arrive(kWeights);   // (the products go where D was)
        if (sm.odd) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (sm.odd_from[part * 16 + j] < kSgRows) D[j] = NAN;
        }
        // D: kept in shared memory and, for the segments behind, where this segment's first outputs will be (all 128 rows are there then; a cluster's
        // shared memory is read at 8 bytes a cycle, L2 at 30).  In pieces of four values, a warp's side by side (value by value, in rows far apart, one portion of 300
        // rows, 8 heads of 40 columns, 33.7 us, so 20.8); value by value only where outputs do not start at 16-byte addresses
        if (rank == last) {
#pragma unroll
          for (int j = 0; j < 4; ++j) X[j * kSgThreads + tid] = make_float4(D[4 * j], D[4 * j + 1], D[4 * j + 2], D[4 * j + 3]);
        } else if (wide) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(scratch + rank * segment + place(j)) = make_float4(D[4 * j], D[4 * j + 1], D[4 * j + 2], D[4 * j + 3]);
        } else if (a.vec_out) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (4 * j < cols) *reinterpret_cast<float4*>(scratch + rank * segment + place_of(j)) = make_float4(D[4 * j], D[4 * j + 1], D[4 * j + 2], D[4 * j + 3]);
        } else if (ml < dim) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < cols) scratch[rank * segment + (int64_t)ml * heads * vd + part * 16 + j] = D[j];
        }
        sg_arrive();   // D is there, and (from the second round on) the state that the round before left in the slot
      }
    }
    sg_wait();
    const auto S_at = [&] { return a.state + (int64_t)slot * a.slot_stride; };                                    // S [heads][vd][dim]
    const auto n_st = [&] { return S_at() + (int64_t)heads * vd * dim + ((int64_t)h * nz + 2 * cb) * dim; };      // n [heads][nz][dim]
    const auto m_st = [&] { return S_at() + (int64_t)heads * (vd + nz) * dim + (int64_t)h * nz + 2 * cb; };       // m [heads][nz]
    const auto S_st = [&] { return S_at() + ((int64_t)h * vd + jb + part * 16) * dim + ml; };
    const bool empty = first == 0 && base == 0, zero = empty && rank == 0;   // S_0 is zeros
    // ---- S_0, n_0, m_0: the state before the round, then segment after segment ----
    double m0 = empty ? 0.0 : (double)__ldcg(m_st());
    float S[16], n0 = 0.f;
    if (empty) {
#pragma unroll
      for (int j = 0; j < 16; ++j) S[j] = 0.f;
    } else {
      if (tid < dim) n0 = __ldcg(n_st() + tid);
#pragma unroll
      for (int j = 0; j < 16; ++j) S[j] = ml < dim && j < cols ? __ldcg(S_st() + (int64_t)j * dim) : 0.f;
    }
    {
      float4 x[4];
      auto get = [&](int i, float4 (&x)[4]) {
        if (wide) {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = __ldcg(reinterpret_cast<const float4*>(scratch + i * segment + place(j)));
        } else if (a.vec_out) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            x[j] = 4 * j < cols ? __ldcg(reinterpret_cast<const float4*>(scratch + i * segment + place_of(j))) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
          float y[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) y[j] = ml < dim && j < cols ? __ldcg(scratch + i * segment + (int64_t)ml * heads * vd + part * 16 + j) : 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
        }
      };
#pragma unroll 1
      for (int i = 0; i < rank; ++i) {
        get(i, x);
        const double fl = sm.fl[i], gl = sm.ml[i], m1 = (double)(float)(fl + fmax(m0, gl));
        const float gamma = expf((float)(fl + m0 - m1)), beta = expf((float)(fl + gl - m1));
        m0 = m1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          S[4 * j] = fmaf(gamma, S[4 * j], beta * x[j].x);
          S[4 * j + 1] = fmaf(gamma, S[4 * j + 1], beta * x[j].y);
          S[4 * j + 2] = fmaf(gamma, S[4 * j + 2], beta * x[j].z);
          S[4 * j + 3] = fmaf(gamma, S[4 * j + 3], beta * x[j].w);
        }
        if (tid < dim) n0 = fmaf(gamma, n0, beta * sm.dn[i][tid]);
      }
    }
    if (tid < KS * 16) sm.n[tid] = n0;
    sg_arrive();
    float D[16];
    if (rank == last) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 x = X[j * kSgThreads + tid];
        D[4 * j] = x.x, D[4 * j + 1] = x.y, D[4 * j + 2] = x.z, D[4 * j + 3] = x.w;
      }
      sync();   // X has been read
    }
    if (!zero) {   // S_0 in three terms, rows of dimensions
      if (ml < KS * 16) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint4 t[3];
          split3(S[8 * j], S[8 * j + 1], t[0].x, t[1].x, t[2].x);
          split3(S[8 * j + 2], S[8 * j + 3], t[0].y, t[1].y, t[2].y);
          split3(S[8 * j + 4], S[8 * j + 5], t[0].z, t[1].z, t[2].z);
          split3(S[8 * j + 6], S[8 * j + 7], t[0].w, t[1].w, t[2].w);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(sg_at(smem + L::r + i * kSgTile, ml, part * 2 + j)) = t[i];
        }
      }
      fence_async_smem();
      arrive(kTerms);
    }
    sg_wait();   // everybody has read the slot and the others' parts
    if (rank == last) {
      const double m1 = (double)(float)(sm.fl[rank] + fmax(m0, sm.ml[rank]));
      const float gamma = expf((float)(sm.fl[rank] + m0 - m1)), beta = expf((float)(sm.fl[rank] + sm.ml[rank] - m1));
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (ml < dim && j < cols) S_st()[(int64_t)j * dim] = fmaf(gamma, S[j], beta * D[j]);
      for (int i = 0; i < min(2, nz - 2 * cb); ++i) {   // the copies of n and m beside these columns
        if (tid < dim) n_st()[(int64_t)i * dim + tid] = fmaf(gamma, n0, beta * sm.dn[rank][tid]);
        if (tid == 0) m_st()[i] = (float)m1;
      }
    }
    if (!zero) {   // q . n_0: two threads a row
      sync();      // (n_0)
      const int r = tid & 255, half = tid >> 8;
      if (r < nl) {
        float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < KS; ++i) {
          const int p = half * KS + i;
          const uint4 q = *reinterpret_cast<const uint4*>(sg_at(smem + L::q, r, p));
          const float4 n_lo = *reinterpret_cast<const float4*>(sm.n + p * 8), n_hi = *reinterpret_cast<const float4*>(sm.n + p * 8 + 4);
          x[0] = fmaf(bf16lo(q.x), n_lo.x, x[0]);
          x[1] = fmaf(bf16hi(q.x), n_lo.y, x[1]);
          x[2] = fmaf(bf16lo(q.y), n_lo.z, x[2]);
          x[3] = fmaf(bf16hi(q.y), n_lo.w, x[3]);
          x[0] = fmaf(bf16lo(q.z), n_hi.x, x[0]);
          x[1] = fmaf(bf16hi(q.z), n_hi.y, x[1]);
          x[2] = fmaf(bf16lo(q.w), n_hi.z, x[2]);
          x[3] = fmaf(bf16hi(q.w), n_hi.w, x[3]);
        }
        sm.qn[half][r] = (x[0] + x[1]) + (x[2] + x[3]);
      }
    }
    wait(kPvLast);
    if (!zero) wait(kQs);
    sync();   // sums of the weights, q . n_0
    // ---- outputs, by way of shared memory (k and q are done with): a row's 256 bytes leave together ----
    float4* stage = reinterpret_cast<float4*>(smem + L::k);
#pragma unroll 1
    for (int tile = 0; tile <= (two ? 1 : 0); ++tile) {
      const int t = tile * 128 + ml;
      uint32_t o[16], o1[16], qs[16];
      ld16(tl + kTmO + tile * 64 + part * 16, o);
      ld16(tl + kTmO + 128 + part * 16, o1);
      ld16(tl + tile * 64 + part * 16, qs);
      const double F = sm.F[t], M = sm.M[t] * 0.6931471805599453, m = (double)(float)(F + fmax(m0, M));
      const float in = M == -INFINITY ? 0.f : expf((float)(F + M - m)), ahead = zero ? 0.f : expf((float)(F + m0 - m)) * a.qscale;
      float nq = in * ((sm.psum[0][t] + sm.psum[1][t]) + (sm.psum[2][t] + sm.psum[3][t]));
      if (!zero) nq = fmaf(ahead, sm.qn[0][t] + sm.qn[1][t], nq);
      const float den = fmaxf(fabsf(nq), expf(-(float)m)) + 1e-6f;
      ld_wait<16>(o);
      ld_wait<16>(o1);
      ld_wait<16>(qs);
      // x / den by the reciprocal and one step of Newton's (rounded as the division is, but for its last bit at most)
      const float inv = 1.0f / den;
      float y[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float x = tile ? __uint_as_float(o[j]) + __uint_as_float(o1[j]) : __uint_as_float(o[j]);
        x = zero ? in * x : fmaf(in, x, ahead * __uint_as_float(qs[j]));
        const float z = x * inv, rest = fmaf(-z, den, x);
        y[j] = rest == rest ? fmaf(rest, inv, z) : z;
      }
      if (sm.odd) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (t >= sm.odd_from[part * 16 + j]) y[j] = NAN;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) stage[t * 16 + ((part * 4 + j) ^ (t & 7))] = make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
    }
    fence_before();
    sync();
    float* dst = a.out + ((int64_t)(start + r0) * heads + h) * vd + jb;
#pragma unroll 1
    for (int e = tid; e < nl * 16; e += kSgThreads) {
      const int r = e >> 4, c = e & 15;
      const float4 y = stage[r * 16 + (c ^ (r & 7))];
      float* to = dst + (int64_t)r * heads * vd + c * 4;
      if (wide) {
        *reinterpret_cast<float4*>(to) = y;
      } else if (c * 4 < width) {   // (a multiple of 8)
        to[0] = y.x, to[1] = y.y, to[2] = y.z, to[3] = y.w;
      }
    }
    sync();   // rows, tensor memory and sums have been read
  }
  __syncthreads();
}

}  // namespace

// Are all clusters of a launch on the device at a time?
bool mlstm_segments_fit(const MlstmArgs& a, int S) { return (int64_t)S * a.heads * ((a.vd + kSgCols - 1) / kSgCols) <= kSgResident; }

int mlstm_segments(MlstmArgs a, int S, cudaStream_t s) {
  if (const int e = wait_status()) return e;
  a.vec_out = reinterpret_cast<uintptr_t>(a.out) % 16 == 0;
  const dim3 grid(S, a.heads, kSgCluster * ((a.vd + kSgCols - 1) / kSgCols)), block(kSgAll), cluster(1, 1, kSgCluster);
#define SEGMENTS(K)                                                                                            \
  do {                                                                                                         \
    static bool done[64] = {};                                                                                 \
    constexpr size_t smem = std::max({(size_t)SgSmem<K>::bytes, sizeof(McSmem<K>), (size_t)ml_floats(K / 4) * 4});   \
    B200_CUDA(ensure_dynamic_smem(mlstm_segment_kernel<K>, (int)smem, done));                                  \
    B200_CUDA(launch_cluster(mlstm_segment_kernel<K>, grid, block, smem, s, cluster, a, wait_status_word()));  \
  } while (0)
  if (a.dim <= 64) SEGMENTS(4);
  else SEGMENTS(8);
#undef SEGMENTS
  return B200_OK;
}

}  // namespace b200
