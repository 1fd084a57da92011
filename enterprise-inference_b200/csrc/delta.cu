// Delta-rule recurrence with one decay per head and key channel (B200_MIXER_DELTA).  Per head and sequence the state is
// S [dim][vdim], fp32, kept in the sequence's state slot between steps together with the last taps - 1 inputs of the
// q | k | v convolution:
//   x_t   = silu(sum_j w[:, j] raw_{t - taps + 1 + j})         per channel of the q | k | v projection, zeros before position 0
//   q_t   = x_q / sqrt(|x_q|^2 + 1e-6) * dim^-1/2              k_t = x_k / sqrt(|x_k|^2 + 1e-6)       per q/k head
//   b_t   = sigmoid(w_b . h_t)                                 per head
//   g_t   = exp(-exp(a_log) * softplus(W_a2 (W_a1 h_t) + dt_bias))          per head and key channel
//   S_t   = diag(g_t) S_{t-1};   u = b_t (v_t - S_t^T k_t);   S_t += k_t u^T;   o_t = S_t^T q_t
// Head h reads q/k head h / (heads / kv_heads).
//
//  * delta_prep: two CTAs per row (one for beta and the decays): convolution taps from the step's own rows or, before the portion's first row, from the
//    slot's tail; silu; the unit vectors; beta; the decays.  Everything leaves in fp32.
//  * delta_tails: CTAs of 256 channels per sequence, after prep: the last taps - 1 raw rows of the portion (or what is left of the old tail
//    when the portion is shorter) become the slot's tail.
//  * delta_scan: the recurrence.  The columns of S do not interact, so a CTA takes (sequence, head, 16 value columns) and walks the
//    sequence's rows of the step with the state in registers (stored [head][vdim][dim]).
//    A sequence whose first row of the step is at position 0 starts from zeros, whatever the slot held.
//
// Two parameters widen the kernels to other recurrences of the same shape.  The decay of (row, head, key channel) is read at
// decay[t * g_row + h * g_head + d * g_chan]: channel decays are (heads*dim, dim, 1), ONE decay per head is (heads, 1, 0), and
// delta_prep then takes the decay's pre-activation straight from the fused row (one column per head, decay_dim 1) instead of a
// second-step projection.  DELTA false drops the correction: u = beta v, which is the state-space recurrence
// S = g S + dt B x^T, y = S^T C of ssd.cu with keys B, queries C, values x and beta = dt.
#include <algorithm>

#include "common.cuh"
#include "f32x2.cuh"

namespace b200 {
namespace {

template <typename AT> __device__ __forceinline__ float ldx(const AT* p, int64_t i);
template <> __device__ __forceinline__ float ldx<float>(const float* p, int64_t i) { return p[i]; }
template <> __device__ __forceinline__ float ldx<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }

__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }

constexpr int kPrepThreads = 256;

template <typename AT>
__global__ void __launch_bounds__(kPrepThreads)
delta_prep_kernel(const AT* __restrict__ fused, int64_t ld, const AT* __restrict__ a2, int64_t a2_ld, int decay_dim, const float* __restrict__ conv_w,
                  const float* __restrict__ dt_bias, const float* __restrict__ a_log, const int32_t* __restrict__ positions,
                  const int32_t* __restrict__ row_to_seq, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_slots,
                  const float* __restrict__ tails, int64_t slot_stride, float* __restrict__ qn, float* __restrict__ kn,
                  float* __restrict__ vn, float* __restrict__ beta, float* __restrict__ decay, int heads, int kv_heads, int dim, int vdim,
                  int taps, int off_b) {
  extern __shared__ float xs[];   // [C] convolved and activated channels
  const int64_t t = blockIdx.x;
  const int qk = kv_heads * dim, C = 2 * qk + heads * vdim;
  if (gridDim.x <= 128) {   // short steps wait on latency: weights and the sequence's tail go to L2 while the launch before runs
    if (blockIdx.y == 0) {
      prefetch_l2_span(conv_w, (size_t)C * taps * 4);
      if (tails) prefetch_l2_span(tails + (int64_t)seq_slots[row_to_seq ? row_to_seq[t] : (int)t] * slot_stride, (size_t)(taps - 1) * C * 4);
    } else {
      prefetch_l2_span(dt_bias, (size_t)heads * decay_dim * 4);
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  if (blockIdx.y == 1) {   // the second CTA of a row: beta and the decays (nothing of the convolution enters them)
    const int hd = heads * decay_dim;   // decay_dim: dim (one decay per key channel) or 1 (one per head)
    for (int h = threadIdx.x; h < heads; h += kPrepThreads) beta[t * heads + h] = sigmoid_f(ldx<AT>(fused, t * ld + off_b + h));
    for (int c = threadIdx.x; c < hd; c += kPrepThreads) {
      const float z = ldx<AT>(a2, t * a2_ld + c) + dt_bias[c];
      decay[t * hd + c] = expf(-expf(a_log[c / decay_dim]) * softplus_f(z));
    }
    return;
  }
  const int s = row_to_seq ? row_to_seq[t] : (int)t;
  const int start = seq_start[s], r = (int)t - start, pos = positions[t];
  const float* tail = tails ? tails + (int64_t)seq_slots[s] * slot_stride : nullptr;   // [taps - 1][C]
  for (int c = threadIdx.x; c < C; c += kPrepThreads) {
    float a = 0.f;
    for (int j = 0; j < taps; ++j) {   // lag j: the input of position pos - j
      if (pos - j < 0) break;
      const float x = r - j >= 0 ? ldx<AT>(fused, (t - j) * ld + c) : tail[(int64_t)(taps - 1 + r - j) * C + c];
      a = fmaf(conv_w[(int64_t)c * taps + taps - 1 - j], x, a);
    }
    xs[c] = a * sigmoid_f(a);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = kPrepThreads / 32;
  const float qscale = rsqrtf((float)dim);
  for (int v = warp; v < 2 * kv_heads; v += nw) {   // q heads, then k heads
    const float* src = xs + (int64_t)v * dim;
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32) ss = fmaf(src[d], src[d], ss);
    ss = warp_sum(ss);
    const float inv = (1.0f / sqrtf(ss + 1e-6f)) * (v < kv_heads ? qscale : 1.0f);
    float* dst = v < kv_heads ? qn + t * qk + (int64_t)v * dim : kn + t * qk + (int64_t)(v - kv_heads) * dim;
    for (int d = lane; d < dim; d += 32) dst[d] = src[d] * inv;
  }
  const int hv = heads * vdim;
  for (int c = threadIdx.x; c < hv; c += kPrepThreads) vn[t * hv + c] = xs[2 * qk + c];
}

template <typename AT>
__global__ void __launch_bounds__(256)
delta_tails_kernel(const AT* __restrict__ fused, int64_t ld, const int32_t* __restrict__ positions, const int32_t* __restrict__ seq_start,
                   const int32_t* __restrict__ seq_slots, float* __restrict__ tails, int64_t slot_stride, int C, int taps) {
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x;
  const int start = seq_start[s], n = seq_start[s + 1] - start;
  if (n <= 0) return;
  const bool fresh = positions[start] == 0;
  float* tail = tails + (int64_t)seq_slots[s] * slot_stride;
  // entry i holds the input of the position (taps - 2 - i) before the portion's last one.  A thread owns a channel and
  // walks i upwards: what it reads of the old tail lies above everything it has written.
  const int c = blockIdx.y * 256 + threadIdx.x;
  if (c < C)
    for (int i = 0; i < taps - 1; ++i) {
      const int ri = n - taps + 1 + i;   // row of the portion, negative: before it
      float v;
      if (ri >= 0) v = ldx<AT>(fused, (int64_t)(start + ri) * ld + c);
      else v = fresh ? 0.f : tail[(int64_t)(taps - 1 + ri) * C + c];
      tail[(int64_t)i * C + c] = v;
    }
}

// The walk.  A lane holds a few neighbouring key channels of four value columns (one shared-memory read of k, q and the decays per row
// serves all four), a warp owns those four columns, a CTA's four warps sixteen; the state lives in registers as pairs for the packed
// fp32 arithmetic.  The step's rows are staged 16 at a time in shared memory by cp.async, the next stage travelling while this one is
// walked.
// What bounds it: one long sequence fills one warp per scheduler, so a row costs its instructions' latency.  Of the chain from row to row
// only S^T k needs other lanes.  The delta rule takes two rows per turn: with S' = S diag(g1), S'' = S' diag(g2)
//   u1 = b1 (v1 - S'^T k1)         u2 = b2 (v2 - S''^T k2 - (sum_d k1 g2 k2) u1)
//   o1 = S'^T q1 + (k1 . q1) u1    S = S'' + (g2 k1) u1 + k2 u2         o2 = S^T q2
// so the eight sums of two rows and four columns are reduced together (a lane keeps half of what it holds at every step: 9 shuffles
// instead of 40), and the two dot products of inputs alone are taken once per stage for all columns.  The read-out leaves per-lane sums in
// shared memory, added for the whole stage after its walk.
// 1 900 rows of three sequences, 16 heads of 128 x 128, channel decays: 295 us (one row per turn, unpacked, eight warps a CTA: 457 us).
constexpr int kDsWarps = 4, kDsCols = 4 * kDsWarps, kDsStage = 16, kDsThreads = kDsWarps * 32;
constexpr int kDsFlush = 8;       // rows whose read-out sums are kept (with all 16 of a stage only two CTAs fit an SM: 342 us instead)
constexpr int kDsPartRow = 144;   // floats of a row of read-out sums: 32 lanes x 4 columns, rows 64 bytes apart in the banks

struct ScanArgs {
  const float* qn;
  const float* kn;
  const float* vn;
  const float* beta;
  const float* decay;
  const int32_t* positions;
  const int32_t* seq_start;
  const int32_t* seq_slots;
  float* state;
  float* out;
  int64_t g_row, slot_stride;
  int g_head, g_chan, heads, kv_heads, dim, vd;
  int vec;   // rows of q, k (and channel decays) can be copied 16 bytes, state columns moved 8 bytes at a time
};

// NP: pairs of channels per lane (1, 2, 4: dim up to 64, 128, 256).  A staged row holds 64 NP floats, zero beyond dim.
__host__ __device__ constexpr int ds_row(int np) { return 64 * np; }
// floats of one stage buffer: q | k | (g) rows, then per row the CTA's 16 values, beta and (head decays) g
__host__ __device__ constexpr int ds_buf(int np, bool chan) { return kDsStage * ((chan ? 3 : 2) * ds_row(np) + kDsCols + 2); }
__host__ __device__ constexpr int ds_floats(int np, bool chan) { return 2 * ds_buf(np, chan) + kDsStage + kDsWarps * kDsFlush * kDsPartRow; }

// the lane's pairs of a staged row; pair i starts at channel 2 x (NP 1), 4 x + 2 (i & 1) + 128 (i >> 1) (else) for lane x
template <int NP>
__device__ __forceinline__ void ds_pairs(const float* row, int lane, uint64_t (&x)[NP]) {
  if constexpr (NP == 1) {
    x[0] = *reinterpret_cast<const uint64_t*>(row + 2 * lane);
  } else {
#pragma unroll
    for (int v = 0; v < NP / 2; ++v) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + 128 * v + 4 * lane);
      x[2 * v] = t.x;
      x[2 * v + 1] = t.y;
    }
  }
}
template <int NP>
__device__ __forceinline__ int ds_chan(int lane, int i) {
  return NP == 1 ? 2 * lane : 4 * lane + 2 * (i & 1) + 128 * (i >> 1);
}
// sums over the warp of N (a power of two) values at once, all of them to every lane
template <int N>
__device__ __forceinline__ void ds_reduce(float (&v)[N], int lane) {
  int bit = 16;
  float x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = v[i];
#pragma unroll
  for (int half = N / 2; half >= 1; half >>= 1, bit >>= 1) {   // keep one half of the values, hand over the other
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = up ? x[i + half] : x[i], give = up ? x[i] : x[i + half];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
  }
#pragma unroll
  for (; bit >= 1; bit >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], bit);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __shfl_sync(0xffffffffu, x[0], i * (32 / N));   // value i ended with the lanes i * 32 / N ..
}

// One row by itself: the four columns' state (pairs of channels, as ds_chan has them) is decayed, corrected, added to and read.  (The walk below has
// the same in line: with this function there instead its registers fell differently, 1 900 rows 294 -> 319 us.)  The row's q, k and
// decays (g_chan apart) start at the head, v and out at the warp's first column, `cols` of which exist.
template <int NP, bool DELTA, bool CHAN>
__device__ __forceinline__ void ds_row_alone(const float* q, const float* k, const float* g, int g_chan, const float* v, float b, float* out, int dim, int cols,
                                             int lane, uint64_t (&S)[4][NP]) {
  uint64_t kk[NP], qq[NP];
  const float gs = CHAN ? 0.f : g[0];
  float d4[4] = {0.f, 0.f, 0.f, 0.f}, o4[4], v4[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) v4[c] = c < cols ? v[c] : 0.f;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int d = ds_chan<NP>(lane, i);
    auto pair = [&](const float* p, int64_t st) { return f2::pack(d < dim ? p[d * st] : 0.f, d + 1 < dim ? p[(d + 1) * st] : 0.f); };
    kk[i] = pair(k, 1);
    qq[i] = pair(q, 1);
    const uint64_t gg = CHAN ? pair(g, g_chan) : f2::both(gs);
#pragma unroll
    for (int c = 0; c < 4; ++c) S[c][i] = f2::mul(S[c][i], gg);
  }
  if (DELTA) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint64_t acc = f2::mul(S[c][0], kk[0]);
#pragma unroll
      for (int i = 1; i < NP; ++i) acc = f2::fma(S[c][i], kk[i], acc);
      d4[c] = f2::sum(acc);
    }
    ds_reduce<4>(d4, lane);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint64_t u = f2::both(b * (v4[c] - d4[c]));
    uint64_t acc = 0;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      S[c][i] = f2::fma(kk[i], u, S[c][i]);
      acc = f2::fma(S[c][i], qq[i], acc);
    }
    o4[c] = f2::sum(acc);
  }
  ds_reduce<4>(o4, lane);
  const float mine = lane == 0 ? o4[0] : lane == 1 ? o4[1] : lane == 2 ? o4[2] : o4[3];
  if (lane < cols) out[lane] = mine;   // (cols <= 4)
}
template <int NP>
__device__ __forceinline__ void ds_load(const float* S_st, int dim, int cols, int vec, bool fresh, int lane, uint64_t (&S)[4][NP]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      const float* p = S_st + (int64_t)c * dim + d;
      S[c][i] = 0;
      if (!fresh && c < cols && d < dim) S[c][i] = vec ? *reinterpret_cast<const uint64_t*>(p) : f2::pack(p[0], d + 1 < dim ? p[1] : 0.f);
    }
}
template <int NP>
__device__ __forceinline__ void ds_store(float* S_st, int dim, int cols, int vec, int lane, const uint64_t (&S)[4][NP]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      float* p = S_st + (int64_t)c * dim + d;
      if (c >= cols || d >= dim) continue;
      if (vec) {
        *reinterpret_cast<uint64_t*>(p) = S[c][i];
      } else {
        p[0] = f2::lo(S[c][i]);
        if (d + 1 < dim) p[1] = f2::hi(S[c][i]);
      }
    }
}

// Steps of decode rows (one row per sequence): the walk without its stages' shared memory, which leaves three or four CTAs to an SM.
// 64 sequences, 16 heads of 128 x 128, channel decays: 37 us in the walk, 23 here; the uncorrected rule, 64 heads of 128 x 64: 4 sequences 8.4
// and 6.4 (7.0 at the unpacked walk, whose CTAs were fewer), 200 sequences 180 and 105.
template <int NP, bool DELTA, bool CHAN>
__global__ void __launch_bounds__(kDsThreads) delta_rows_kernel(const ScanArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int start = a.seq_start[s], end = a.seq_start[s + 1];
  if (end <= start) return;
  const int j0 = blockIdx.z * kDsCols + warp * 4, cols = min(a.vd - j0, 4), g = h / (a.heads / a.kv_heads), dim = a.dim;
  float* S_st = a.state + (int64_t)a.seq_slots[s] * a.slot_stride + ((int64_t)h * a.vd + j0) * dim;
  const int64_t qk = (int64_t)a.kv_heads * dim, hv = (int64_t)a.heads * a.vd;
  uint64_t S[4][NP];
  ds_load<NP>(S_st, dim, cols, a.vec, a.positions[start] == 0, lane, S);
  for (int64_t t = start; t < end; ++t)
    ds_row_alone<NP, DELTA, CHAN>(a.qn + t * qk + (int64_t)g * dim, a.kn + t * qk + (int64_t)g * dim, a.decay + t * a.g_row + (int64_t)h * a.g_head, a.g_chan,
                                  a.vn + t * hv + (int64_t)h * a.vd + j0, a.beta[t * a.heads + h], a.out + t * hv + (int64_t)h * a.vd + j0, dim, cols, lane, S);
  ds_store<NP>(S_st, dim, cols, a.vec, lane, S);
}

// CHAN: a decay per key channel, else one per row and head.
template <int NP, bool DELTA, bool CHAN>
__global__ void __launch_bounds__(kDsThreads) delta_scan_kernel(const ScanArgs a) {
  extern __shared__ __align__(16) float stage[];
  constexpr int ROW = ds_row(NP), BUF = ds_buf(NP, CHAN);
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, jb = blockIdx.z * kDsCols;
#define DS_SYNC() __syncthreads()
#include "delta_walk.cuh"
#undef DS_SYNC
}
// the same by the first kDsThreads threads of a larger CTA
template <int NP, bool DELTA, bool CHAN>
__device__ __forceinline__ void ds_walk(const ScanArgs& a, float* stage, int s, int h, int jb) {
  constexpr int ROW = ds_row(NP), BUF = ds_buf(NP, CHAN);
#define DS_SYNC() asm volatile("bar.sync 1, 128;" ::: "memory")
#include "delta_walk.cuh"
#undef DS_SYNC
}

// Portions of several rows in blocks of eight.  With L_i the product of the decays up to row i of a block, u the corrected values and S the state before it
//   u_i = b_i (v_i - S^T (L_i k_i) - sum_{j<i} (k_i . (L_i / L_j) k_j) u_j)
//   o_i = S^T (L_i q_i) + sum_{j<=i} (q_i . (L_i / L_j) k_j) u_j          S' = L_8 S + sum_j (L_8 / L_j) k_j u_j^T
// so with w_i = b_i (v_i - S^T (L_i k_i)) the rows of a block meet in two 8 x 8 triangles that depend on its inputs alone: u = T w, o = S^T (L q) + B w
// (the ratios are products of the decays between the rows: nothing is divided, a decay may be 0).
// A CTA per (sequence, head, 16 value columns), those of a head in clusters.  Its main warps own four columns per LG lanes and reduce a block's sums over
// these lanes together (a lane keeps half of what it holds at every step); two warps turn the rows of the blocks ahead into L q, L k and
// (L_8 / L) k; one or two work out the triangles of every C-th block for the C CTAs of the cluster, a round of blocks ahead.
// LG 32 (four main warps) where one or two CTAs share an SM, LG 16 (two warps, a third fewer instructions a column) for three and for keys of at most 64.
// What bounds them: a block's chain of about 2 100 cycles (dots 840, their reduction 400, triangles and u 500, update 210, waiting for the
// cluster 230), and issue slots where CTAs share an SM: a shuffle takes four cycles of a scheduler, a packed fma two.
// A reduction's first two steps go over the rows: a lane takes the rows of a set in an order of its own, so that every lane keeps the same registers and
// hands over the same others.  Choosing them by lane was two selections a shuffle: without, one sequence of 2 000 rows 310 -> 274 us, two of 1 000
// together 163 -> 147, three of 1 900 244 -> 228, keys of 64 239 -> 205 (same sums, same bits).
// Against the walk (us, 16 heads of 128 x 128, channel decays): one sequence of 1 900 rows 406 -> 245, two of 1 000 together 182 -> 114, three of 1 900
// 295 -> 186, four of 1 200 315 -> 145; one decay per head, four of 2 048 554 -> 211; keys of 64, four of 2 000 349 -> 129; 150 rows 37 -> 26.  The walk keeps
// short portions (a block needs its triangles before it starts, about 5 us) and the uncorrected rule (in CTAs of 32 columns three sequences of 64 heads
// 282 -> 251, but four short ones 11 -> 17).
constexpr int kDbRows = 8, kDbScale = 2, kDbSlots = 4, kDbCluster = 4;   // (clusters of eight such CTAs do not fit the device sixteen at a time)
constexpr int kDbTri = 2 * kDbRows * kDbRows;   // T, B
constexpr int db_main(int lg) { return lg == 32 ? 4 : 2; }   // warps with columns; warps that work out triangles
constexpr int db_tri_warps(int ctas) { return ctas <= 2 ? 2 : 1; }   // (ctas: that share an SM)
constexpr int db_threads(int lg, int ctas) { return (db_main(lg) + kDbScale + db_tri_warps(ctas)) * 32; }
// rows from which a portion goes in blocks: where the two meet for one sequence, and for two to four
constexpr int db_from(int lg) { return lg == 32 ? 64 : 128; }
// CTAs that share an SM.  Two where the launch then fills its places twice over (four sequences, 16 heads of 128 x 128: 1 200 rows 145 us, at three 173),
// three where that leaves a third of a wave alone (three sequences of 1 900 rows 186, at two 247) and from four launches' worth on (eight of 2 048 206, at two 213).
constexpr int db_share(int64_t ctas) { return ctas <= kNumSMs ? 1 : ctas <= 2 * kNumSMs || (ctas > 3 * kNumSMs && ctas <= 4 * kNumSMs) ? 2 : 3; }
// lanes of four columns
constexpr int db_lanes(int np, int share) { return np == 2 && share <= 2 ? 32 : 16; }
// Sequences of a launch in blocks whose rows the host does not know: with more of them most are likely short, and these are walked faster by the walk's own CTAs
// (eight sequences of three rows 9.2 us, from the block kernel 10.2; six 9.2 and 8.5).  Where it knows them, up to as many as db_sequence orders, of at
// least kDbMean rows on average (eight of 125 rows 146 us, in blocks 111; 32 of 25 rows 122 and 111, of three 28 and 36).
constexpr int kDbSeqs = 6, kDbOrdered = 32, kDbMean = 32;
// floats of a slot: L q | L k | (L_8 / L) k, L_8
__host__ __device__ constexpr int db_slot(int np) { return (3 * kDbRows + 1) * ds_row(np); }
// slots; three rounds of triangles; per main warp 8 x 8 pairs (u, u)
constexpr int db_floats(int np, int lg, int ctas) { return kDbSlots * db_slot(np) + 3 * db_tri_warps(ctas) * kDbCluster * kDbTri + db_main(lg) * kDbRows * 16; }
template <int N>
__device__ __forceinline__ void db_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ void db_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory"); }
__device__ __forceinline__ void db_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void db_cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }   // (nothing to show)
__device__ __forceinline__ void db_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The sum over the warp of value i of 32, to lane i.
__device__ __forceinline__ float db_reduce(float (&x)[32], int lane) {
#pragma unroll
  for (int half = 16; half >= 1; half >>= 1) {
    const bool up = (lane & half) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = up ? x[i + half] : x[i], give = up ? x[i] : x[i + half];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
    }
  }
  return x[0];
}

// One step of the sums over a group of lanes: 2 H values become H, the lane keeps one half of them and hands over the other.
template <int H>
__device__ __forceinline__ void db_halve(float* x, int lane) {
  const bool up = (lane & H) != 0;
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const float keep = up ? x[i + H] : x[i], give = up ? x[i] : x[i + H];
    x[i] = keep + __shfl_xor_sync(0xffffffffu, give, H);
  }
}

// The same where every lane has laid its values out so that the first half is the one it keeps.
template <int H>
__device__ __forceinline__ void db_fold(float* x) {
#pragma unroll
  for (int i = 0; i < H; ++i) x[i] += __shfl_xor_sync(0xffffffffu, x[i + H], H);
}

// The k-th longest of n portions: the grid goes over the sequences last and the longest first.  The CTAs of an SM are then of several sequences, and
// what waits for a place is short.  With the sequences first in the grid those of an SM were mostly of one, and the longest one's SMs the last: three of 1 900 rows
// together 228 us, 186 now, two of 1 000 147 and 114, one decay per head 372 and 254.
__device__ __forceinline__ int db_sequence(const ScanArgs& a, int n, int k) {
  static_assert(kDbOrdered == 32, "a lane a sequence");
  const int lane = threadIdx.x & 31, rows = lane < n ? a.seq_start[lane + 1] - a.seq_start[lane] : -1;
  int rank = 0;
  for (int i = 0; i < n; ++i) {
    const int other = __shfl_sync(0xffffffffu, rows, i);
    rank += other > rows || (other == rows && i < lane);
  }
  return __ffs(__ballot_sync(0xffffffffu, lane < n && rank == k)) - 1;
}

template <int NP, bool CHAN, int LG, int CTAS>
__global__ void __launch_bounds__(db_threads(LG, CTAS), CTAS) delta_block_kernel(const ScanArgs a) {
  extern __shared__ __align__(16) float stage[];
  constexpr int ROW = ds_row(NP), R = kDbRows, SLOT = db_slot(NP), MAIN = db_main(LG), BAR = 32 * (MAIN + 1);   // BAR: threads of the main warps and one other
  // named barriers: slot ready; slot read; triangles of an even (odd) round read, from the main warps to those that work triangles out
  constexpr int kFull = 1, kEmpty = 1 + kDbSlots, kRead = 1 + 2 * kDbSlots, READ = 32 * (MAIN + db_tri_warps(CTAS));
  static_assert(NP <= 2, "a preparing lane's channels are one piece of at most 16 bytes");
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.y, jb = blockIdx.x * kDsCols, s = db_sequence(a, gridDim.z, blockIdx.z);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows <= 0) return;
  const int g = h / (a.heads / a.kv_heads), dim = a.dim, vd = a.vd;
  const bool fresh = a.positions[start] == 0;
  const int64_t qk = (int64_t)a.kv_heads * dim, hv = (int64_t)a.heads * vd;
  const float* qsrc = a.qn + (int64_t)start * qk + (int64_t)g * dim;
  const float* ksrc = a.kn + (int64_t)start * qk + (int64_t)g * dim;
  const float* gsrc = a.decay + (int64_t)start * a.g_row + (int64_t)h * a.g_head;
  const float* vsrc = a.vn + (int64_t)start * hv + (int64_t)h * vd + jb;
  const float* bsrc = a.beta + (int64_t)start * a.heads + h;
  float* out = a.out + (int64_t)start * hv + (int64_t)h * vd + jb;
  float* state = a.state + (int64_t)a.seq_slots[s] * a.slot_stride + ((int64_t)h * vd + jb) * dim;
  if (n_rows < db_from(LG)) {
    if (warp < kDsWarps) ds_walk<NP, true, CHAN>(a, stage, s, h, jb);
    return;
  }
  const int n_blocks = (n_rows + R - 1) / R;
  uint32_t C, rank;   // CTAs of the cluster, all of one sequence and head
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int per_round = db_tri_warps(CTAS) * (int)C, rounds = (n_blocks + per_round - 1) / per_round;
  float* tris = stage + kDbSlots * SLOT;   // [3][blocks of a round][T | B]
  // cluster barriers: all CTAs run; then, for every round p, its triangles are there and those of round p - 3 have been read
  db_cluster_arrive_relaxed();

  if (warp >= MAIN + kDbScale) {
    // ===== triangles: lane l takes the sums of the pair (pi, pj), 28 below the diagonal row by row; lanes from 28 on the diagonal's halves =====
    int pi = 1;
    while (pi < R - 1 && lane >= (pi + 1) * pi / 2) ++pi;
    const int d = 2 * NP * lane;
    using Rows = uint64_t[R];
    Rows k0, g0, q0;
    auto pieces = [&](int b, int i, Rows& k, Rows& g, Rows& q, float gs = 0.f) {   // the lane's i-th pairs of the block's rows
      const int nb = min(n_rows - b * R, R);
      auto pair = [&](const float* src, int64_t st, int r, uint64_t none) {
        return r < nb && d < dim ? *reinterpret_cast<const uint64_t*>(src + (int64_t)(b * R + r) * st + d + 2 * i) : none;
      };
#pragma unroll
      for (int r = 0; r < R; ++r) {
        k[r] = pair(ksrc, qk, r, 0);
        q[r] = pair(qsrc, qk, r, 0);
        g[r] = CHAN ? pair(gsrc, a.g_row, r, f2::both(1.f)) : f2::both(__shfl_sync(0xffffffffu, gs, r));
      }
    };
    // what a block starts with; where a CTA has an SM's registers to itself it is asked for before the wait for the round before (2 000 rows alone 275 -> 258 us; at the
    // 128 registers of two or three CTAs an SM warps spill for it, three sequences of 1 900 rows 184 -> 232)
    constexpr bool AHEAD = CTAS == 1 && NP == 2;
    float bs0, gs0;   // of row `lane`
    auto scalars = [&](int b, float& bs, float& gs) {
      const int nb = min(n_rows - b * R, R);
      bs = lane < nb ? bsrc[(int64_t)(b * R + lane) * a.heads] : 0.f;
      gs = !CHAN && lane < nb ? gsrc[(int64_t)(b * R + lane) * a.g_row] : 1.f;
    };
    auto fetch = [&](int b) {
      if (b >= n_blocks) return;
      scalars(b, bs0, gs0);
      pieces(b, 0, k0, g0, q0);
    };
    if (AHEAD) fetch((warp - MAIN - kDbScale) * (int)C + (int)rank);
    db_cluster_wait();
    for (int p = 0; p < rounds; ++p) {
      const int own = (warp - MAIN - kDbScale) * (int)C + (int)rank, b = p * per_round + own;
      if (b < n_blocks) {
        float bs, gs;
        if (AHEAD) bs = bs0, gs = gs0;
        else scalars(b, bs, gs);
        float x[2][32];   // k with k and the diagonal's first half; q with k and its second
#pragma unroll
        for (int i = 0; i < NP; ++i) {   // channels in NP passes, for the registers
          Rows k, g, q;
          if (AHEAD && !i) {
#pragma unroll
            for (int r = 0; r < R; ++r) k[r] = k0[r], q[r] = q0[r], g[r] = CHAN ? g0[r] : f2::both(__shfl_sync(0xffffffffu, gs, r));
          } else {
            pieces(b, i, k, g, q, gs);
          }
          auto add = [&](float& to, uint64_t a, uint64_t b) {
            const float sum = f2::sum(f2::mul(a, b));
            to = i ? to + sum : sum;
          };
#pragma unroll
          for (int j = 0; j < R - 1; ++j) {
            uint64_t z = k[j];
#pragma unroll
            for (int r = j + 1; r < R; ++r) {
              z = f2::mul(z, g[r]);
              add(x[0][r * (r - 1) / 2 + j], z, k[r]);
              add(x[1][r * (r - 1) / 2 + j], z, q[r]);
            }
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            add(x[0][28 + r], k[r], q[r]);
            add(x[1][28 + r], k[4 + r], q[4 + r]);
          }
        }
        const float kk = db_reduce(x[0], lane), qq = db_reduce(x[1], lane);
        // T = (1 + diag(b) (k with k))^-1 and B = (q with k) T, a column a lane
        float* tri = tris + (p % 3 * per_round + own) * kDbTri;
        float t[R];
#pragma unroll
        for (int i = 0; i < R; ++i) t[i] = lane == i ? 1.f : 0.f;
        const float bl = __shfl_sync(0xffffffffu, bs, pi) * kk;
#pragma unroll
        for (int m = 0; m < R - 1; ++m)
#pragma unroll
          for (int i = m + 1; i < R; ++i) {
            const float c = __shfl_sync(0xffffffffu, bl, i * (i - 1) / 2 + m);
            if (lane <= m) t[i] = fmaf(-c, t[m], t[i]);   // (not beyond the column's first row: there is nothing to multiply)
          }
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float c = __shfl_sync(0xffffffffu, i < 4 ? kk : qq, 28 + (i & 3));
          float y = lane <= i ? c * t[i] : 0.f;
#pragma unroll
          for (int m = 0; m < i; ++m) {
            const float e = __shfl_sync(0xffffffffu, qq, i * (i - 1) / 2 + m);
            if (lane <= m) y = fmaf(e, t[m], y);
          }
          if (lane < R) {
            tri[i * R + lane] = t[i];
            tri[(R + i) * R + lane] = y;
          }
        }
        __syncwarp();
        const float4 quad = *reinterpret_cast<const float4*>(tri + 4 * lane);
        for (uint32_t c = 0; c < C; ++c) {
          if (c == rank) continue;
          uint32_t to;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"((uint32_t)__cvta_generic_to_shared(tri + 4 * lane)), "r"(c));
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(quad.x), "f"(quad.y), "f"(quad.z), "f"(quad.w) : "memory");
        }
      }
      // Round p + 1's triangles go where those of round p - 2 were: this CTA's main warps have read them, which this warp's release hands on to the CTAs that
      // write there.  (A release of the main warps' own waits for their outputs' stores: one sequence of 2 000 rows, keys of 64, 280 us instead of 254.)
      if (p >= 2 && p + 1 < rounds) db_sync<READ>(kRead + (p & 1));
      db_cluster_arrive();
      if (AHEAD) fetch(b + per_round);
      db_cluster_wait();
    }
    return;
  }

  if (warp >= MAIN) {
    // ===== rows times their decays: a warp a block, a lane NP neighbouring pairs of channels =====
    const int w = warp - MAIN, d = 2 * NP * lane;
    const bool live = d < dim;
    auto store = [&](float* row, const uint64_t (&x)[NP]) {
      if constexpr (NP == 1) *reinterpret_cast<uint64_t*>(row + d) = x[0];
      else *reinterpret_cast<ulonglong2*>(row + d) = make_ulonglong2(x[0], x[1]);
    };
    uint64_t k[R][NP], q[R][NP], gg[R][NP];
    float gs = 1.f;   // of row `lane`
    auto fetch = [&](int b) {   // channels beyond dim and rows past the last one: no weight, no decay
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int64_t t = (int64_t)b * R + r;
        const bool there = live && t < n_rows;
        auto get = [&](const float* p, uint64_t none, uint64_t (&x)[NP]) {
#pragma unroll
          for (int i = 0; i < NP; ++i) x[i] = none;
          if (!there) return;
          if constexpr (NP == 1) {
            x[0] = *reinterpret_cast<const uint64_t*>(p + d);
          } else {
            const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(p + d);
            x[0] = y.x;
            x[1] = y.y;
          }
        };
        get(qsrc + t * qk, 0, q[r]);
        get(ksrc + t * qk, 0, k[r]);
        if (CHAN) get(gsrc + t * a.g_row, f2::both(1.f), gg[r]);
      }
      if (!CHAN) gs = lane < R && b * R + lane < n_rows ? gsrc[(int64_t)(b * R + lane) * a.g_row] : 1.f;
    };
    if (w < n_blocks) fetch(w);
    db_cluster_wait();
    db_cluster_arrive_relaxed();
    int round = 0;   // whose barrier this warp has arrived at
    for (int b = w; b < n_blocks; b += kDbScale) {
      while (b >= (round + 1) * per_round) {
        db_cluster_wait();
        db_cluster_arrive_relaxed();
        ++round;
      }
      if (b >= kDbSlots) db_sync<BAR>(kEmpty + b % kDbSlots);   // block b - kDbSlots has been read
      float* slot = stage + (b % kDbSlots) * SLOT;
      uint64_t L[NP], rest[NP], x[NP];
      if (!CHAN) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint64_t y = f2::both(__shfl_sync(0xffffffffu, gs, r));
#pragma unroll
          for (int i = 0; i < NP; ++i) gg[r][i] = y;
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int i = 0; i < NP; ++i) L[i] = r ? f2::mul(L[i], gg[r][i]) : gg[0][i];
#pragma unroll
        for (int i = 0; i < NP; ++i) x[i] = f2::mul(q[r][i], L[i]);
        store(slot + r * ROW, x);
#pragma unroll
        for (int i = 0; i < NP; ++i) x[i] = f2::mul(k[r][i], L[i]);
        store(slot + (R + r) * ROW, x);
      }
      store(slot + 3 * R * ROW, L);
#pragma unroll
      for (int r = R - 1; r >= 0; --r) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          x[i] = r == R - 1 ? k[r][i] : f2::mul(k[r][i], rest[i]);
          rest[i] = r == R - 1 ? gg[r][i] : f2::mul(rest[i], gg[r][i]);
        }
        store(slot + (2 * R + r) * ROW, x);
      }
      __syncwarp();
      db_arrive<BAR>(kFull + b % kDbSlots);
      if (b + kDbScale < n_blocks) fetch(b + kDbScale);
    }
    while (++round < rounds) {
      db_cluster_wait();
      db_cluster_arrive_relaxed();
    }
    db_cluster_wait();
    return;
  }

  // ===== LG lanes four columns, a lane x of them the channels 4 x + 4 LG v =====
  constexpr int CW = 128 / LG, V = ROW / (4 * LG);   // columns of a warp; pieces of four channels a lane
  const int xl = lane & (LG - 1), x16 = lane & 15, grp = lane / LG, j0 = warp * CW + grp * 4, cols = min(vd - jb - j0, 4);
  float* us = tris + 3 * db_tri_warps(CTAS) * kDbCluster * kDbTri + warp * R * 16;   // [8 rows][CW columns] pairs (u, u)
  uint64_t S[4][2 * V];
  float* S_st = state + (int64_t)j0 * dim;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = 4 * xl + 4 * LG * i;
      ulonglong2 y = make_ulonglong2(0, 0);
      if (!fresh && c < cols && d < dim) y = *reinterpret_cast<const ulonglong2*>(S_st + (int64_t)c * dim + d);
      S[c][2 * i] = y.x;
      S[c][2 * i + 1] = y.y;
    }
  // the lane's two places in a block's small sums: rows rr and rr + 4 of one of its half's columns
  const int rr = x16 >> 2, col = x16 & 3, from = grp * 16 + col;
  const bool have = col < cols;
  float v[2], bt[2];
  auto fetch_v = [&](int b) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int64_t t = (int64_t)b * R + rr + 4 * i;
      const bool ok = t < n_rows;
      v[i] = ok && have ? vsrc[t * hv + j0 + col] : 0.f;
      bt[i] = ok ? bsrc[t * a.heads] : 0.f;
    }
  };
  auto row_of = [&](const float* row, uint64_t (&y)[2 * V]) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + 4 * xl + 4 * LG * i);
      y[2 * i] = t.x;
      y[2 * i + 1] = t.y;
    }
  };
  // a lane takes the rows of a set in the order that leaves its own row of the four first: what it hands over is then the same half in every lane
  int own[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) own[r] = (r ^ rr) * ROW;
  fetch_v(0);
  db_cluster_wait();
  db_cluster_arrive_relaxed();
  int in_round = per_round - 1, round = -1;   // block of the round, the round
  for (int b = 0; b < n_blocks; ++b) {
    if (++in_round == per_round) {
      in_round = 0;
      db_cluster_wait();
      if (++round + 1 < rounds) db_cluster_arrive_relaxed();
      if (round >= 1 && round + 2 < rounds) db_arrive<READ>(kRead + ((round - 1) & 1));
    }
    db_sync<BAR>(kFull + b % kDbSlots);
    const float* in = stage + (b % kDbSlots) * SLOT;
    const float* tri = tris + (round % 3 * per_round + in_round) * kDbTri + rr * R;
    float m[2][3][4];   // T and B: row rr up to column 3, row rr + 4
    auto triangles = [&]() {
#pragma unroll
      for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float4 e = *reinterpret_cast<const float4*>(tri + z * R * R + (i ? 4 * R + 4 * (i - 1) : 0));
          m[z][i][0] = e.x, m[z][i][1] = e.y, m[z][i][2] = e.z, m[z][i][3] = e.w;
        }
    };
    // sets of four rows times four columns: of L k (rows 0..3, 4..7), of L q.  JOINT sets are reduced together, a step of one covers the others' latency
    constexpr int JOINT = LG == 32 ? 4 : 2;
    float sum[2][2];   // of L k, of L q; of rows rr and rr + 4
#pragma unroll
    for (int s0 = 0; s0 < 4; s0 += JOINT) {
      float part[JOINT][16];
#pragma unroll
      for (int s1 = 0; s1 < JOINT; ++s1) {
        const int set = s0 + s1;
        uint64_t y[4][2 * V];
#pragma unroll
        for (int r = 0; r < 4; ++r) row_of(in + ((set < 2 ? R : 0) + 4 * (set & 1)) * ROW + own[r], y[r]);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint64_t acc = f2::mul(S[c][0], y[r][0]);
#pragma unroll
            for (int i = 1; i < 2 * V; ++i) acc = f2::fma(S[c][i], y[r][i], acc);
            part[s1][4 * r + c] = f2::sum(acc);
          }
      }
      auto all = [&](auto&& f) {
#pragma unroll
        for (int s1 = 0; s1 < JOINT; ++s1) f(part[s1]);
      };
      all([&](float* x) { db_fold<8>(x); });
      if (s0 + JOINT == 4) triangles();
      all([&](float* x) { db_fold<4>(x); });
      all([&](float* x) { db_halve<2>(x, lane); });
      all([&](float* x) { db_halve<1>(x, lane); });
#pragma unroll
      for (int s1 = 0; s1 < JOINT; ++s1)
        sum[(s0 + s1) >> 1][s1 & 1] = part[s1][0] + (LG == 32 ? __shfl_xor_sync(0xffffffffu, part[s1][0], 16) : 0.f);
    }
    const float w[2] = {bt[0] * (v[0] - sum[0][0]), bt[1] * (v[1] - sum[0][1])};
    fetch_v(b + 1);
    // u = T w, o = S^T (L q) + B w: the rows up to the lane's own
    float y[2][2] = {{0.f, 0.f}, {sum[1][0], sum[1][1]}};
    uint64_t G[2 * V], kx[LG == 32 ? R : 1][2 * V];   // (a lane of 32 has room for the rows that the update takes)
    row_of(in + 3 * R * ROW, G);
    if (LG == 32) {
#pragma unroll
      for (int r = 0; r < R; ++r) row_of(in + (2 * R + r) * ROW, kx[r]);
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const float wj = __shfl_sync(0xffffffffu, w[j >> 2], from + 4 * (j & 3));
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        if (j < 4) {
          if (j <= rr) y[z][0] = fmaf(m[z][0][j], wj, y[z][0]);   // (selected: a later row may be anything)
          y[z][1] = fmaf(m[z][1][j], wj, y[z][1]);
        } else if (j - 4 <= rr) {
          y[z][1] = fmaf(m[z][2][j - 4], wj, y[z][1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = b * R + rr + 4 * i;
      const float u = t < n_rows ? y[0][i] : 0.f;
      *reinterpret_cast<float2*>(us + (rr + 4 * i) * 2 * CW + grp * 8 + 2 * col) = make_float2(u, u);
      if (t < n_rows && have && (LG == 16 || lane < 16)) out[(int64_t)t * hv + j0 + col] = y[1][i];
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int i = 0; i < 2 * V; ++i) S[c][i] = f2::mul(S[c][i], G[i]);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint64_t x[2 * V];
      if (LG == 32) {
#pragma unroll
        for (int i = 0; i < 2 * V; ++i) x[i] = kx[r][i];
      } else {
        row_of(in + (2 * R + r) * ROW, x);
      }
      const ulonglong2* up = reinterpret_cast<const ulonglong2*>(us + r * 2 * CW + grp * 8);
      const ulonglong2 u01 = up[0], u23 = up[1];
      const uint64_t uu[4] = {u01.x, u01.y, u23.x, u23.y};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 2 * V; ++i) S[c][i] = f2::fma(x[i], uu[c], S[c][i]);
    }
    if (b + kDbSlots < n_blocks) db_arrive<BAR>(kEmpty + b % kDbSlots);
    __syncwarp();   // u has been read
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = 4 * xl + 4 * LG * i;
      if (c < cols && d < dim) *reinterpret_cast<ulonglong2*>(S_st + (int64_t)c * dim + d) = make_ulonglong2(S[c][2 * i], S[c][2 * i + 1]);
    }
}

// CTAs of a head that share triangles: the largest divisor of its column blocks up to kDbCluster
int db_cluster(int blocks) {
  int c = kDbCluster;
  while (blocks % c) --c;
  return c;
}
template <int NP, bool CHAN, int LG, int CTAS>   // CTAS: that share an SM
int delta_block(const ScanArgs& a, int S, cudaStream_t s) {
  static bool done[64] = {};
  const dim3 grid((a.vd + kDsCols - 1) / kDsCols, a.heads, S);
  // shared memory for CTAS an SM, so that no more meet there: the CTAs of a cluster are packed onto as few SMs as hold them
  constexpr int need = std::max(db_floats(NP, LG, CTAS), ds_floats(NP, CHAN)) * 4, bytes = CTAS == 1 ? 120 * 1024 : CTAS == 2 ? 80 * 1024 : need;
  static_assert(need <= bytes && CTAS * (bytes + 1024) <= 228 * 1024, "CTAs an SM");
  B200_CUDA(ensure_dynamic_smem(delta_block_kernel<NP, CHAN, LG, CTAS>, bytes, done));
  B200_CUDA(launch_cluster(delta_block_kernel<NP, CHAN, LG, CTAS>, grid, dim3(db_threads(LG, CTAS)), (size_t)bytes, s, dim3(db_cluster((int)grid.x), 1, 1), a));
  return B200_OK;
}

template <int NP, bool CHAN>
int delta_blocks(const ScanArgs& a, int S, int64_t ctas, cudaStream_t s) {
  switch (db_share(ctas)) {
    case 1: return delta_block<NP, CHAN, db_lanes(NP, 1), 1>(a, S, s);
    case 2: return delta_block<NP, CHAN, db_lanes(NP, 2), 2>(a, S, s);
    default: return delta_block<NP, CHAN, db_lanes(NP, 3), 3>(a, S, s);
  }
}

}  // namespace

static int up8(int v) { return (v + 7) / 8 * 8; }

// rows of the fused projection; offsets of q, k, v, a1, g1, b
int delta_fused_rows(int heads, int kv_heads, int dim, int vdim, int decay_rank, int gate_rank, int* off) {
  int o[6];
  o[0] = 0;
  o[1] = kv_heads * dim;
  o[2] = 2 * kv_heads * dim;
  o[3] = up8(o[2] + heads * vdim);
  o[4] = up8(o[3] + decay_rank);
  o[5] = up8(o[4] + gate_rank);
  if (off)
    for (int i = 0; i < 6; ++i) off[i] = o[i];
  return up8(o[5] + heads);
}

int64_t delta_state_floats(int heads, int dim, int vd) { return (int64_t)heads * vd * dim; }
int64_t delta_tail_floats(int heads, int kv_heads, int dim, int vd, int taps) {
  return (int64_t)(taps > 1 ? taps - 1 : 0) * (2 * kv_heads * dim + heads * vd);
}

int delta_prep(bool f32, const void* fused, int64_t ld, const void* a2, const float* conv_w, const float* dt_bias, const float* a_log,
               const int32_t* positions, const int32_t* row_to_seq, const int32_t* seq_start, const int32_t* seq_slots, const float* tails,
               int64_t slot_stride, float* qn, float* kn, float* vn, float* beta, float* decay, int T, int heads, int kv_heads, int dim,
               int vdim, int taps, int decay_rank, int gate_rank, cudaStream_t s, bool head_decay) {
  if (T == 0) return B200_OK;
  B200_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && taps >= 1, B200_ERR_INVALID, "delta_prep: %d heads over %d, %d taps", heads,
               kv_heads, taps);
  B200_REQUIRE(taps == 1 || (tails && seq_slots), B200_ERR_INVALID, "delta_prep: the convolution needs its tails");
  int off[6];
  delta_fused_rows(heads, kv_heads, dim, vdim, decay_rank, gate_rank, off);
  int64_t a2_ld = (int64_t)heads * dim;
  int decay_dim = dim;
  if (head_decay) {   // fused rows q | k | v | gate | b | a without padding: the decay's pre-activation is the row's last group
    off[5] = 2 * kv_heads * dim + 2 * heads * vdim;
    a2 = static_cast<const char*>(fused) + (int64_t)(off[5] + heads) * (f32 ? 4 : 2);
    a2_ld = ld;
    decay_dim = 1;
  }
  const size_t smem = (size_t)(2 * kv_heads * dim + heads * vdim) * 4;
  B200_REQUIRE(smem <= 200 * 1024, B200_ERR_UNSUPPORTED, "delta_prep: %zu bytes of channels do not fit shared memory", smem);
  static bool done[2][64] = {};
  if (f32) {
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(delta_prep_kernel<float>, 200 * 1024, done[0]));
    B200_CUDA(launch(delta_prep_kernel<float>, dim3(T, 2), dim3(kPrepThreads), smem, s, (const float*)fused, ld, (const float*)a2, a2_ld, decay_dim, conv_w, dt_bias,
                     a_log, positions, row_to_seq, seq_start, seq_slots, tails, slot_stride, qn, kn, vn, beta, decay, heads, kv_heads, dim, vdim,
                     taps, off[5]));
  } else {
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(delta_prep_kernel<__nv_bfloat16>, 200 * 1024, done[1]));
    B200_CUDA(launch(delta_prep_kernel<__nv_bfloat16>, dim3(T, 2), dim3(kPrepThreads), smem, s, (const __nv_bfloat16*)fused, ld,
                     (const __nv_bfloat16*)a2, a2_ld, decay_dim, conv_w, dt_bias, a_log, positions, row_to_seq, seq_start, seq_slots, tails, slot_stride, qn, kn,
                     vn, beta, decay, heads, kv_heads, dim, vdim, taps, off[5]));
  }
  return B200_OK;
}

int delta_tails(bool f32, const void* fused, int64_t ld, const int32_t* positions, const int32_t* seq_start, const int32_t* seq_slots,
                float* tails, int64_t slot_stride, int S, int channels, int taps, cudaStream_t s) {
  if (S == 0 || taps <= 1) return B200_OK;
  B200_REQUIRE(tails && seq_slots && seq_start && positions, B200_ERR_INVALID, "delta_tails: null argument");
  if (f32)
    B200_CUDA(launch(delta_tails_kernel<float>, dim3(S, (channels + 255) / 256), dim3(256), (size_t)0, s, (const float*)fused, ld, positions, seq_start, seq_slots, tails,
                     slot_stride, channels, taps));
  else
    B200_CUDA(launch(delta_tails_kernel<__nv_bfloat16>, dim3(S, (channels + 255) / 256), dim3(256), (size_t)0, s, (const __nv_bfloat16*)fused, ld, positions, seq_start,
                     seq_slots, tails, slot_stride, channels, taps));
  return B200_OK;
}

int delta_scan(const float* qn, const float* kn, const float* vn, const float* beta, const float* decay, const int32_t* positions,
               const int32_t* seq_start, const int32_t* seq_slots, float* state, int64_t slot_stride, float* out, int S, int heads,
               int kv_heads, int dim, int vd, cudaStream_t s, int rows) {
  return linear_scan(true, qn, kn, vn, beta, decay, (int64_t)heads * dim, dim, 1, positions, seq_start, seq_slots, state, slot_stride, out, S,
                     heads, kv_heads, dim, vd, s, rows);
}

int linear_scan(bool delta_rule, const float* qn, const float* kn, const float* vn, const float* beta, const float* decay, int64_t g_row,
                int g_head, int g_chan, const int32_t* positions, const int32_t* seq_start, const int32_t* seq_slots, float* state,
                int64_t slot_stride, float* out, int S, int heads, int kv_heads, int dim, int vd, cudaStream_t s, int rows) {
  if (S == 0) return B200_OK;
  B200_REQUIRE(dim > 0 && dim <= 256 && vd > 0, B200_ERR_UNSUPPORTED, "delta_scan: key size %d outside (0, 256]", dim);
  B200_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0, B200_ERR_INVALID, "delta_scan: %d heads over %d", heads, kv_heads);
  B200_REQUIRE(positions && seq_start && seq_slots && state, B200_ERR_INVALID, "delta_scan: null argument");
  const bool chan = g_chan != 0;
  ScanArgs a = {qn, kn, vn, beta, decay, positions, seq_start, seq_slots, state, out, g_row, slot_stride, g_head, g_chan, heads, kv_heads, dim, vd, 0};
  const auto at = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr); };
  // wide pieces: every row and state column starts at a multiple of four floats
  a.vec = dim % 4 == 0 && slot_stride % 4 == 0 && ((at(qn) | at(kn) | at(state)) & 15) == 0 &&
          (!chan || (g_chan == 1 && g_row % 4 == 0 && g_head % 4 == 0 && at(decay) % 16 == 0));
  const dim3 grid(S, heads, (vd + kDsCols - 1) / kDsCols), block(kDsThreads);
  const int64_t ctas = (int64_t)S * heads * grid.z;
  const bool single_rows = rows == S;
  // Blocks where a portion may be long enough for them; where the rows of the step are known to be too few its walk is launched by itself (one portion of 63 rows, 16
  // heads of 128 x 128: 19.0 us from the block kernel, 18.2; of two rows 5.5 and 5.1)
  const bool few = S <= kDbSeqs && ctas <= kDbSeqs * kNumSMs, many = S <= kDbOrdered && ctas <= kDbOrdered * kNumSMs && rows >= kDbMean * S;
  const bool blocks = a.vec && (few || many) && (rows <= 0 || rows - S + 1 >= db_from(db_lanes(dim > 64 ? 2 : 1, db_share(ctas))));
#define SCAN3(D, R, CH)                                                                                       \
  do {                                                                                                        \
    static bool done[64] = {};                                                                                \
    const size_t smem = (size_t)ds_floats(D, CH) * 4;                                                         \
    if (single_rows) {                                                                                        \
      B200_CUDA(launch(delta_rows_kernel<D, R, CH>, grid, block, (size_t)0, s, a));                           \
      break;                                                                                                  \
    }                                                                                                         \
    if constexpr (D <= 2 && R)                                                                                \
      if (blocks) {                                                                                           \
        if (const int e = delta_blocks<D, CH>(a, S, ctas, s)) return e;                                       \
        break;                                                                                                \
      }                                                                                                       \
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(delta_scan_kernel<D, R, CH>, (int)smem, done));       \
    B200_CUDA(launch(delta_scan_kernel<D, R, CH>, grid, block, smem, s, a));                                  \
  } while (0)
#define SCAN(D)                                          \
  do {                                                   \
    if (delta_rule && chan) SCAN3(D, true, true);        \
    else if (delta_rule) SCAN3(D, true, false);          \
    else if (chan) SCAN3(D, false, true);                \
    else SCAN3(D, false, false);                         \
  } while (0)
  if (dim <= 64) SCAN(1);
  else if (dim <= 128) SCAN(2);
  else SCAN(4);
#undef SCAN
#undef SCAN3
  return B200_OK;
}

}  // namespace b200
