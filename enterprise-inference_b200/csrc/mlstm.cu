// Matrix-memory recurrence (B200_MIXER_MLSTM).  Per head and sequence the state is S [dim][vdim], n [dim] and a running
// maximum m of the log gates, all fp32, kept in the sequence's state slot between steps:
//   i_t = cap tanh((w_i . h + b_i) / cap)              f_t = logsigmoid(cap tanh((w_f . h + b_f) / cap))
//   m_t = max(f_t + m_{t-1}, i_t)                      a = exp(f_t + m_{t-1} - m_t),  b = exp(i_t - m_t)
//   S_t = a S_{t-1} + b k_t v_t^T                      n_t = a n_{t-1} + b k_t
//   o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6),   q_t scaled by dim^-1/2
// then each head's o_t is brought to unit RMS, multiplied by a weight and by sigmoid(g_t).
//
//  * mlstm_gates: the two gate projections with fp32 accumulation and the gate transforms, [T][2 heads] fp32;
//  * mlstm_scan: the recurrence.  The columns of S do not interact, so a CTA takes (sequence, head, 32 value columns) and walks the
//    sequence's rows of the step in order (mlstm_walk.cuh; a decode row is a walk of one) with the state in registers; it is stored as
//    [head][vdim][dim].  n and m are kept once per 32 columns (every CTA of a head needs them from the step before, so they cannot
//    all share one copy that one of them overwrites).  A sequence whose first row is at position 0 starts from zeros.  Longer portions
//    go through the tensor cores in chunks (mlstm_chunk.cuh) and segments (mlstm_segment.cu).
//  * head_norm_gate: unit RMS per head, weight, sigmoid gate (or the gate's silu).
#include "mlstm_walk.cuh"

namespace b200 {
namespace {

template <typename AT> __device__ __forceinline__ void stx(AT* p, int64_t i, float v);
template <> __device__ __forceinline__ void stx<float>(float* p, int64_t i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stx<__nv_bfloat16>(__nv_bfloat16* p, int64_t i, float v) { p[i] = __float2bfloat16_rn(v); }

__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

template <typename AT>
__global__ void __launch_bounds__(128)
mlstm_gates_kernel(const AT* __restrict__ x, const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias, float* __restrict__ out,
                   int width, int heads, float cap) {
  extern __shared__ float xs[];
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = blockIdx.x;
  for (int c = threadIdx.x; c < width; c += 128) xs[c] = ldx<AT>(x, t * width + c);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int o = warp; o < 2 * heads; o += 4) {
    const __nv_bfloat16* wr = w + (int64_t)o * width;
    float a = 0.f;
    for (int c = lane; c < width; c += 32) a = fmaf(__bfloat162float(wr[c]), xs[c], a);
    a = warp_sum(a);
    if (lane == 0) {
      const float z = cap * tanhf((a + (bias ? bias[o] : 0.f)) / cap);
      out[t * 2 * heads + o] = o < heads ? z : log_sigmoid(z);
    }
  }
}

// the walk of mlstm_walk.cuh on its own
template <typename AT, int NP>
__global__ void __launch_bounds__(kScanThreads, NP <= 2 ? 2 : 1) mlstm_scan_kernel(const MlstmArgs a) {
  extern __shared__ __align__(16) float stage[];
  pdl_wait();
  pdl_launch_dependents();
  if (a.both && a.seq_start[blockIdx.x + 1] - a.seq_start[blockIdx.x] >= kChunkFrom) return;   // the chunk kernel's
  mlstm_walk<AT, NP>(a, stage, blockIdx.z, gridDim.z);
}

// Steps of decode rows only (one row per sequence): no staging, no shared memory, a warp's lanes side by side in the state's rows, so that
// many CTAs share an SM and the state's loads and stores, which are all of the work, overlap (128 rows of 8 heads, 128 x 256: 47.5 us; the
// walk above, without its staging: 66).  DPL: key dimensions per lane.
template <typename AT, int DPL>
__global__ void __launch_bounds__(kNWarp * 32) mlstm_rows_kernel(const MlstmArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, zb = blockIdx.z, nz = gridDim.z, heads = a.heads, dim = a.dim, vd = a.vd;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows <= 0) return;
  const bool fresh = a.positions[start] == 0;
  float* S_st = a.state + (int64_t)a.seq_slots[s] * a.slot_stride;                                     // [heads][vd][dim]
  float* n_st = S_st + (int64_t)heads * vd * dim + ((int64_t)h * nz + zb) * dim;                       // [heads][nz][dim]
  float* m_st = S_st + (int64_t)heads * vd * dim + (int64_t)heads * nz * dim + (int64_t)h * nz + zb;   // [heads][nz]
  const int j0 = zb * kScanCols + warp * 4;
  float Sr[4][DPL], nr[DPL];
#pragma unroll
  for (int i = 0; i < DPL; ++i) {
    const int d = lane + 32 * i;
    nr[i] = (!fresh && d < dim) ? n_st[d] : 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) Sr[c][i] = (!fresh && d < dim && j0 + c < vd) ? S_st[((int64_t)h * vd + j0 + c) * dim + d] : 0.f;
  }
  float m = fresh ? 0.f : *m_st;
  __syncthreads();   // every warp has read n and m before warp 0 may store them
  for (int t = start; t < start + n_rows; ++t) {
    const AT* row = static_cast<const AT*>(a.qkv) + (int64_t)t * a.ld;
    const float ig = a.gates[(int64_t)t * 2 * heads + h], fg = a.gates[(int64_t)t * 2 * heads + heads + h];
    const float m_new = fmaxf(fg + m, ig);
    const float da = expf(fg + m - m_new), b = expf(ig - m_new);
    m = m_new;
    float nq = 0.f, acc[4], v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[c] = 0.f;
      v[c] = j0 + c < vd ? ldx<AT>(row, a.v_off + h * vd + j0 + c) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int d = lane + 32 * i;
      const float qv = d < dim ? ldx<AT>(row, a.q_off + h * dim + d) * a.qscale : 0.f;
      const float bk = b * (d < dim ? ldx<AT>(row, a.k_off + h * dim + d) : 0.f);
      nr[i] = fmaf(da, nr[i], bk);
      nq = fmaf(nr[i], qv, nq);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        Sr[c][i] = fmaf(da, Sr[c][i], bk * v[c]);
        acc[c] = fmaf(Sr[c][i], qv, acc[c]);
      }
    }
    nq = warp_sum(nq);
    const float den = fmaxf(fabsf(nq), expf(-m)) + 1e-6f;
    float mine = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float o = warp_sum(acc[c]);
      if (lane == c) mine = o;
    }
    if (lane < 4 && j0 + lane < vd) a.out[((int64_t)t * heads + h) * vd + j0 + lane] = mine / den;
  }
#pragma unroll
  for (int i = 0; i < DPL; ++i) {
    const int d = lane + 32 * i;
    if (d >= dim) continue;
    if (warp == 0) n_st[d] = nr[i];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (j0 + c < vd) S_st[((int64_t)h * vd + j0 + c) * dim + d] = Sr[c][i];
  }
  if (warp == 0 && lane == 0) *m_st = m;
}

// one CTA per row, one warp per head (round robin)
template <typename AT>
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float* __restrict__ o, const float* __restrict__ w, const AT* __restrict__ gate, int64_t ldg,
                      AT* __restrict__ out, int heads, int vd, float eps, int gate_silu) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int h = warp; h < heads; h += 4) {
    const float* src = o + (t * heads + h) * vd;
    float ss = 0.f;
    for (int j = lane; j < vd; j += 32) ss = fmaf(src[j], src[j], ss);
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss / (float)vd + eps);
    for (int j = lane; j < vd; j += 32) {
      float v = src[j] * inv;
      if (w) v *= w[h * vd + j];
      if (gate) {
        const float gz = ldx<AT>(gate, t * ldg + h * vd + j);
        v *= (gate_silu ? gz : 1.0f) / (1.0f + expf(-gz));
      }
      stx<AT>(out, (t * heads + h) * vd + j, v);
    }
  }
}

}  // namespace

int mlstm_gates(bool f32, const void* x, const __nv_bfloat16* w, const float* bias, float* out, int T, int width, int heads, float cap,
                cudaStream_t s) {
  if (T == 0) return B200_OK;
  B200_REQUIRE(cap > 0.f, B200_ERR_INVALID, "mlstm_gates: cap %f", (double)cap);
  const size_t smem = (size_t)width * 4;
  B200_REQUIRE(smem <= 200 * 1024, B200_ERR_UNSUPPORTED, "mlstm_gates: width %d does not fit shared memory", width);
  static bool done[2][64] = {};
  if (f32) {
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(mlstm_gates_kernel<float>, 200 * 1024, done[0]));
    B200_CUDA(launch(mlstm_gates_kernel<float>, dim3(T), dim3(128), smem, s, (const float*)x, w, bias, out, width, heads, cap));
  } else {
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(mlstm_gates_kernel<__nv_bfloat16>, 200 * 1024, done[1]));
    B200_CUDA(launch(mlstm_gates_kernel<__nv_bfloat16>, dim3(T), dim3(128), smem, s, (const __nv_bfloat16*)x, w, bias, out, width, heads,
                     cap));
  }
  return B200_OK;
}

int mlstm_col_blocks(int vd) { return (vd + kScanCols - 1) / kScanCols; }

// floats of one layer's recurrent state in a slot: S [heads][vd][dim], n [heads][col blocks][dim], m [heads][col blocks]
int64_t mlstm_state_floats(int heads, int dim, int vd) {
  const int64_t nz = mlstm_col_blocks(vd);
  return (int64_t)heads * vd * dim + (int64_t)heads * nz * dim + (int64_t)heads * nz;
}

template <typename AT>
static int mlstm_scan_t(const MlstmArgs& a, int S, bool single_rows, cudaStream_t s) {
  const dim3 grid(S, a.heads, mlstm_col_blocks(a.vd));
#define SCAN(D)                                                                                                            \
  do {                                                                                                                     \
    static bool done[64] = {};                                                                                             \
    constexpr size_t smem = (size_t)ml_floats(D) * 4;                                                                      \
    if (single_rows) {                                                                                                     \
      B200_CUDA(launch(mlstm_rows_kernel<AT, 2 * D>, grid, dim3(kNWarp * 32), (size_t)0, s, a));                           \
    } else {                                                                                                               \
      B200_CUDA(ensure_dynamic_smem(mlstm_scan_kernel<AT, D>, (int)smem, done));                                           \
      B200_CUDA(launch(mlstm_scan_kernel<AT, D>, grid, dim3(kScanThreads), smem, s, a));                                   \
    }                                                                                                                      \
  } while (0)
  if (a.dim <= 64) SCAN(1);
  else if (a.dim <= 128) SCAN(2);
  else SCAN(4);
#undef SCAN
  return B200_OK;
}

// Steps of a few bf16 portions on the tensor cores where they are long.  While all clusters of a launch in segments run at a time, one launch takes all:
// segments from 193 rows on, chunks from 97, the walk below.  (36 clusters, 9 heads of 256 columns: 160 rows 33.7 us, in chunks 16.6; 300 rows 36.2 and 25.2; 2 048
// rows 109 and 142, but the length is known on the device only.)
// Where the rows of the step are known to be too few for a long portion, chunks and walk are launched by themselves: in the segments' launch (us, in a graph, 8 heads)
// 2 rows 5.3 instead of 5.0, 140 rows 17.8 and 16.5 (128 x 256); 2 rows 4.9 and 4.3, 69 rows 14.7 and 13.5, 215 rows 18.6 and 17.3 (64 x 128).  (A kernel in which tensor memory is allocated at all
// takes 0.3 us longer to start: the walk alone in that launch's shape 3.9 us for the 2 rows, with an allocation that it never comes to 4.2.)  Segments pay from
// 193 rows (215 rows 20.1, in chunks 20.8), with keys of 64 from 257 (300 rows 18.6 and 20.8); 2 048 rows of 128 x 256 58 and 142.
// Beyond that chunks for all long portions, one or two CTAs an SM, and while these fit at once the chunk kernel walks the short portions itself; else each kernel
// takes its portions (64 rows of four sequences: 15.0 us, in one kernel 23.1: the idle half of each cluster holds up the next).  Segments there too were a
// third launch, 5 us of host time for a call of 20 rows, and slower for portions of some hundred rows (three of 400 together, 4 heads, 29 -> 50 us); they won
// from about 200 rows a portion on (four of 1 000, 8 heads, 111 -> 97), which the host does not know.
// More sequences than four go to the walk alone (64 of one row 36 us; longer portions of many sequences on the tensor cores have not been measured).
enum class MlstmRoute { kWalk, kChunks, kSegments };
static MlstmRoute mlstm_route(const MlstmArgs& a, int S, bool f32, int rows) {   // rows 0: not known
  if (f32 || rows == S || S > 4 || !mlstm_chunk_supported(a)) return MlstmRoute::kWalk;
  const bool too_few = rows > 0 && rows - S + 1 < (a.dim <= 64 ? 257 : kSegmentFrom);
  return mlstm_segments_fit(a, S) && !too_few ? MlstmRoute::kSegments : MlstmRoute::kChunks;
}

int mlstm_scan(bool f32, const void* qkv, int64_t ld, int q_off, int k_off, int v_off, const float* gates, const int32_t* positions,
               const int32_t* seq_start, const int32_t* seq_slots, float* state, int64_t slot_stride, float* out, int S, int heads,
               int dim, int vd, cudaStream_t s, int rows) {
  if (S == 0) return B200_OK;
  B200_REQUIRE(dim > 0 && dim <= 256 && vd > 0, B200_ERR_UNSUPPORTED, "mlstm_scan: key size %d outside (0, 256]", dim);
  B200_REQUIRE(positions && seq_start && seq_slots && state, B200_ERR_INVALID, "mlstm_scan: null argument");
  MlstmArgs a = {qkv, gates, positions, seq_start, seq_slots, state, out, ld, slot_stride, q_off, k_off, v_off, heads, dim, vd, 1.0f / sqrtf((float)dim), -0.5 * log2((double)dim), 0, 0, 0, 0};
  mlstm_walk_widths(a, f32);
  const MlstmRoute route = mlstm_route(a, S, f32, rows);
  if (route == MlstmRoute::kSegments) return mlstm_segments(a, S, s);
  if (route == MlstmRoute::kChunks) {
    a.both = mlstm_chunk_ctas(a, S) > 2 * kNumSMs;
    if (const int e = mlstm_chunk(a, S, s)) return e;
    if (!a.both) return B200_OK;
    const PdlScope after_chunks;
    return mlstm_scan_t<__nv_bfloat16>(a, S, false, s);
  }
  return f32 ? mlstm_scan_t<float>(a, S, rows == S, s) : mlstm_scan_t<__nv_bfloat16>(a, S, rows == S, s);
}

int head_norm_gate(bool f32, const float* o, const float* w, const void* gate, int64_t ldg, void* out, int T, int heads, int vd, float eps,
                   cudaStream_t s, bool gate_silu) {
  if (T == 0) return B200_OK;
  if (f32)
    B200_CUDA(launch(head_norm_gate_kernel<float>, dim3(T), dim3(128), (size_t)0, s, o, w, (const float*)gate, ldg, (float*)out, heads, vd,
                     eps, gate_silu ? 1 : 0));
  else
    B200_CUDA(launch(head_norm_gate_kernel<__nv_bfloat16>, dim3(T), dim3(128), (size_t)0, s, o, w, (const __nv_bfloat16*)gate, ldg,
                     (__nv_bfloat16*)out, heads, vd, eps, gate_silu ? 1 : 0));
  return B200_OK;
}

}  // namespace b200

// debug helper (not in the public header): how a step of bf16 rows (0: not known how many) goes, with everything aligned (0 the walk alone, 1 chunks, 2 segments)
extern "C" __attribute__((visibility("default"))) int b200_debug_mlstm_route(int32_t n_seqs, int32_t heads, int32_t dim, int32_t vdim, int32_t rows) {
  using namespace b200;
  MlstmArgs a = {};
  a.qkv = reinterpret_cast<const void*>(64);
  a.heads = heads, a.dim = dim, a.vd = vdim;
  return (int)mlstm_route(a, n_seqs, false, rows);
}
