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
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows <= 0) return;
  const bool fresh = a.positions[start] == 0;
  const int g = h / (a.heads / a.kv_heads), dim = a.dim, vd = a.vd;
  const int j0 = jb + warp * 4;   // the warp's first value column
  float* S_st = a.state + (int64_t)a.seq_slots[s] * a.slot_stride + ((int64_t)h * vd + j0) * dim;
  const int64_t qk = (int64_t)a.kv_heads * dim, hv = (int64_t)a.heads * vd;
  const float* qsrc = a.qn + (int64_t)start * qk + (int64_t)g * dim;
  const float* ksrc = a.kn + (int64_t)start * qk + (int64_t)g * dim;
  const float* gsrc = a.decay + (int64_t)start * a.g_row + (int64_t)h * a.g_head;
  const float* vsrc = a.vn + (int64_t)start * hv + (int64_t)h * vd + jb;
  const float* bsrc = a.beta + (int64_t)start * a.heads + h;
  uint64_t S[4][NP];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      const float* p = S_st + (int64_t)c * dim + d;
      S[c][i] = 0;
      if (!fresh && j0 + c < vd && d < dim) S[c][i] = a.vec ? *reinterpret_cast<const uint64_t*>(p) : f2::pack(p[0], d + 1 < dim ? p[1] : 0.f);
    }
  if (n_rows == 1) {
    // a decode row: nothing to stage; the row's inputs are fetched beside the state
    const float b = bsrc[0], gs = CHAN ? 0.f : gsrc[0];
    uint64_t k[NP], q[NP];
    float d4[4] = {0.f, 0.f, 0.f, 0.f}, o4[4];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      auto pair = [&](const float* p, int64_t st) { return f2::pack(d < dim ? p[d * st] : 0.f, d + 1 < dim ? p[(d + 1) * st] : 0.f); };
      k[i] = pair(ksrc, 1);
      q[i] = pair(qsrc, 1);
      const uint64_t gg = CHAN ? pair(gsrc, a.g_chan) : f2::both(gs);
#pragma unroll
      for (int c = 0; c < 4; ++c) S[c][i] = f2::mul(S[c][i], gg);
    }
    if (DELTA) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint64_t acc = f2::mul(S[c][0], k[0]);
#pragma unroll
        for (int i = 1; i < NP; ++i) acc = f2::fma(S[c][i], k[i], acc);
        d4[c] = f2::sum(acc);
      }
      ds_reduce<4>(d4, lane);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint64_t u = f2::both(b * ((j0 + c < vd ? vsrc[warp * 4 + c] : 0.f) - d4[c]));
      uint64_t acc = 0;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        S[c][i] = f2::fma(k[i], u, S[c][i]);
        acc = f2::fma(S[c][i], q[i], acc);
      }
      o4[c] = f2::sum(acc);
    }
    ds_reduce<4>(o4, lane);
    const float mine = lane == 0 ? o4[0] : lane == 1 ? o4[1] : lane == 2 ? o4[2] : o4[3];
    if (lane < 4 && j0 + lane < vd) a.out[(int64_t)start * hv + (int64_t)h * vd + j0 + lane] = mine;
  } else {
    float* kq = stage + 2 * BUF;                                          // [kDsStage] per pair of rows: k1 g2 k2, k1 . q1
    float* part = kq + kDsStage + warp * kDsFlush * kDsPartRow;
    if (dim < ROW) {   // zeros beyond dim, once: the copies leave them alone
      for (int e = tid; e < 2 * BUF; e += kDsThreads) stage[e] = 0.f;
      __syncthreads();
    }
    auto fetch = [&](int b0, float* buf) {
      const int nb = min(kDsStage, n_rows - b0);
      float* sq = buf;
      float* sk = sq + kDsStage * ROW;
      float* sg = sk + kDsStage * ROW;
      float* sv = sq + kDsStage * (CHAN ? 3 : 2) * ROW;
      float* sb = sv + kDsStage * kDsCols;
      if (a.vec) {
#pragma unroll
        for (int e0 = 0; e0 < kDsStage * ROW / 4; e0 += kDsThreads) {
          const int e = e0 + tid, r = e / (ROW / 4), c = (e % (ROW / 4)) * 4;
          if (r < nb && c < dim) {
            f2::cp16(sq + r * ROW + c, qsrc + (b0 + r) * qk + c);
            f2::cp16(sk + r * ROW + c, ksrc + (b0 + r) * qk + c);
            if (CHAN) f2::cp16(sg + r * ROW + c, gsrc + (b0 + r) * a.g_row + c);
          }
        }
      } else {
        for (int e = tid; e < kDsStage * ROW; e += kDsThreads) {
          const int r = e / ROW, c = e % ROW;
          if (r < nb && c < dim) {
            f2::cp4(sq + r * ROW + c, qsrc + (b0 + r) * qk + c);
            f2::cp4(sk + r * ROW + c, ksrc + (b0 + r) * qk + c);
            if (CHAN) f2::cp4(sg + r * ROW + c, gsrc + (b0 + r) * a.g_row + (int64_t)c * a.g_chan);
          }
        }
      }
#pragma unroll
      for (int e0 = 0; e0 < kDsStage * kDsCols; e0 += kDsThreads) {
        const int e = e0 + tid, r = e / kDsCols, c = e % kDsCols;
        if (r < nb && jb + c < vd) f2::cp4(sv + e, vsrc + (b0 + r) * hv + c);
      }
      if (tid < nb) {
        f2::cp4(sb + tid, bsrc + (int64_t)(b0 + tid) * a.heads);
        if (!CHAN) f2::cp4(sb + kDsStage + tid, gsrc + (b0 + tid) * a.g_row);
      }
    };
    fetch(0, stage);
    for (int b0 = 0, it = 0; b0 < n_rows; b0 += kDsStage, ++it) {
      const int nb = min(kDsStage, n_rows - b0);
      const float* sq = stage + (it & 1) * BUF;
      const float* sk = sq + kDsStage * ROW;
      const float* sg = sk + kDsStage * ROW;
      const float* sv = sq + kDsStage * (CHAN ? 3 : 2) * ROW + warp * 4;
      const float* sb = sv - warp * 4 + kDsStage * kDsCols;
      f2::cp_wait_all();
      __syncthreads();   // the stage has landed for everybody, and the one before has been consumed
      if (b0 + kDsStage < n_rows) fetch(b0 + kDsStage, stage + ((it + 1) & 1) * BUF);
      if (DELTA) {
        for (int r = 2 * warp; r + 1 < nb; r += 2 * kDsWarps) {
          float xy[2] = {0.f, 0.f};
#pragma unroll
          for (int d = 0; d < ROW; d += 32) {
            const float k1 = sk[r * ROW + d + lane], k2 = sk[(r + 1) * ROW + d + lane];
            xy[0] = fmaf(CHAN ? k1 * sg[(r + 1) * ROW + d + lane] : k1, k2, xy[0]);
            xy[1] = fmaf(k1, sq[r * ROW + d + lane], xy[1]);
          }
          ds_reduce<2>(xy, lane);
          if (lane == 0) *reinterpret_cast<float2*>(kq + r) = make_float2(CHAN ? xy[0] : xy[0] * sb[kDsStage + r + 1], xy[1]);
        }
        __syncthreads();
      }
      auto decay_row = [&](const uint64_t (&gg)[NP]) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < NP; ++i) S[c][i] = f2::mul(S[c][i], gg[i]);
      };
      auto decays = [&](int r, uint64_t (&gg)[NP]) {
        if (CHAN) {
          ds_pairs<NP>(sg + r * ROW, lane, gg);
        } else {
          const uint64_t x = f2::both(sb[kDsStage + r]);
#pragma unroll
          for (int i = 0; i < NP; ++i) gg[i] = x;
        }
      };
      auto dots = [&](const uint64_t (&x)[NP], float* o) {   // the lane's part of S^T x for the four columns
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint64_t acc = f2::mul(S[c][0], x[0]);
#pragma unroll
          for (int i = 1; i < NP; ++i) acc = f2::fma(S[c][i], x[i], acc);
          o[c] = f2::sum(acc);
        }
      };
      int r = 0;
      for (int f0 = 0; f0 < nb; f0 += kDsFlush) {
      const int f1 = min(f0 + kDsFlush, nb);
      if (DELTA) {
        for (; r + 1 < f1; r += 2) {
          uint64_t g1[NP], g2[NP], k1[NP], k2[NP], q1[NP], q2[NP];
          decays(r, g1);
          ds_pairs<NP>(sk + r * ROW, lane, k1);
          decays(r + 1, g2);
          ds_pairs<NP>(sk + (r + 1) * ROW, lane, k2);
          ds_pairs<NP>(sq + r * ROW, lane, q1);
          ds_pairs<NP>(sq + (r + 1) * ROW, lane, q2);
          const float4 v1 = *reinterpret_cast<const float4*>(sv + r * kDsCols), v2 = *reinterpret_cast<const float4*>(sv + (r + 1) * kDsCols);
          const float2 bb = *reinterpret_cast<const float2*>(sb + r), kk = *reinterpret_cast<const float2*>(kq + r);
          float d[8], o1[4], o2[4];
          decay_row(g1);
          dots(k1, d);
          dots(q1, o1);
          decay_row(g2);
          dots(k2, d + 4);
          ds_reduce<8>(d, lane);
          const float va[4] = {v1.x, v1.y, v1.z, v1.w}, vb[4] = {v2.x, v2.y, v2.z, v2.w};
          uint64_t kg[NP];
#pragma unroll
          for (int i = 0; i < NP; ++i) kg[i] = f2::mul(k1[i], g2[i]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float u1 = bb.x * (va[c] - d[c]), u2 = bb.y * (vb[c] - fmaf(kk.x, u1, d[4 + c]));
            if (lane == 0) o1[c] = fmaf(kk.y, u1, o1[c]);
            const uint64_t w1 = f2::both(u1), w2 = f2::both(u2);
#pragma unroll
            for (int i = 0; i < NP; ++i) S[c][i] = f2::fma(k2[i], w2, f2::fma(kg[i], w1, S[c][i]));
          }
          dots(q2, o2);
          *reinterpret_cast<float4*>(part + (r - f0) * kDsPartRow + 4 * lane) = make_float4(o1[0], o1[1], o1[2], o1[3]);
          *reinterpret_cast<float4*>(part + (r + 1 - f0) * kDsPartRow + 4 * lane) = make_float4(o2[0], o2[1], o2[2], o2[3]);
        }
      }
#pragma unroll 2
      for (; r < f1; ++r) {
        uint64_t gg[NP], k[NP], q[NP];
        decays(r, gg);
        ds_pairs<NP>(sk + r * ROW, lane, k);
        ds_pairs<NP>(sq + r * ROW, lane, q);
        const float4 v4 = *reinterpret_cast<const float4*>(sv + r * kDsCols);
        const float va[4] = {v4.x, v4.y, v4.z, v4.w}, b = sb[r];
        float d[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
        decay_row(gg);
        if (DELTA) {
          dots(k, d);
          ds_reduce<4>(d, lane);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint64_t u = f2::both(b * (va[c] - d[c]));
#pragma unroll
          for (int i = 0; i < NP; ++i) S[c][i] = f2::fma(k[i], u, S[c][i]);
        }
        dots(q, o);
        *reinterpret_cast<float4*>(part + (r - f0) * kDsPartRow + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
      }
      __syncwarp();
      {   // four lanes a row, eight lanes' sums each
        const int rr = lane >> 2, quarter = lane & 3;
        const float* src = part + rr * kDsPartRow + quarter * 32;
        uint64_t x = 0, y = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + 4 * (i ^ quarter));   // (the four lanes' banks apart)
          x = f2::add(x, t.x);
          y = f2::add(y, t.y);
        }
        float o[4] = {f2::lo(x), f2::hi(x), f2::lo(y), f2::hi(y)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          o[c] += __shfl_xor_sync(0xffffffffu, o[c], 1);
          o[c] += __shfl_xor_sync(0xffffffffu, o[c], 2);
        }
        const float mine = quarter == 0 ? o[0] : quarter == 1 ? o[1] : quarter == 2 ? o[2] : o[3];
        if (f0 + rr < f1 && j0 + quarter < vd) a.out[(int64_t)(start + b0 + f0 + rr) * hv + (int64_t)h * vd + j0 + quarter] = mine;
      }
      __syncwarp();
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      float* p = S_st + (int64_t)c * dim + d;
      if (j0 + c >= vd || d >= dim) continue;
      if (a.vec) {
        *reinterpret_cast<uint64_t*>(p) = S[c][i];
      } else {
        p[0] = f2::lo(S[c][i]);
        if (d + 1 < dim) p[1] = f2::hi(S[c][i]);
      }
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
               int kv_heads, int dim, int vd, cudaStream_t s, bool single_rows) {
  return linear_scan(true, qn, kn, vn, beta, decay, (int64_t)heads * dim, dim, 1, positions, seq_start, seq_slots, state, slot_stride, out, S,
                     heads, kv_heads, dim, vd, s, single_rows);
}

int linear_scan(bool delta_rule, const float* qn, const float* kn, const float* vn, const float* beta, const float* decay, int64_t g_row,
                int g_head, int g_chan, const int32_t* positions, const int32_t* seq_start, const int32_t* seq_slots, float* state,
                int64_t slot_stride, float* out, int S, int heads, int kv_heads, int dim, int vd, cudaStream_t s, bool single_rows) {
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
#define SCAN3(D, R, CH)                                                                                       \
  do {                                                                                                        \
    static bool done[64] = {};                                                                                \
    const size_t smem = (size_t)ds_floats(D, CH) * 4;                                                         \
    if (single_rows) {                                                                                        \
      B200_CUDA(launch(delta_rows_kernel<D, R, CH>, grid, block, (size_t)0, s, a));                           \
      break;                                                                                                  \
    }                                                                                                         \
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
