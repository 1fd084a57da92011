// Matrix-memory recurrence (B200_MIXER_MLSTM).  Per head and sequence the state is S [dim][vdim], n [dim] and a running
// maximum m of the log gates, all fp32, kept in the sequence's state slot between steps:
//   i_t = cap tanh((w_i . h + b_i) / cap)              f_t = logsigmoid(cap tanh((w_f . h + b_f) / cap))
//   m_t = max(f_t + m_{t-1}, i_t)                      a = exp(f_t + m_{t-1} - m_t),  b = exp(i_t - m_t)
//   S_t = a S_{t-1} + b k_t v_t^T                      n_t = a n_{t-1} + b k_t
//   o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6),   q_t scaled by dim^-1/2
// then each head's o_t is brought to unit RMS, multiplied by a weight and by sigmoid(g_t).
//
//  * mlstm_gates: the two gate projections with fp32 accumulation and the gate transforms, [T][2 heads] fp32;
//  * mlstm_scan: the recurrence.  The columns of S do not interact, so a CTA takes (sequence, head, 16 value columns) and walks the
//    sequence's rows of the step in order (a decode row is a walk of one) with the state in registers; it is stored as
//    [head][vdim][dim].  n and m are kept once per 32 columns (every CTA of a head needs them from the step before, so they cannot
//    all share one copy that one of them overwrites).  A sequence whose first row is at position 0 starts from zeros.
//  * head_norm_gate: unit RMS per head, weight, sigmoid gate (or the gate's silu).
#include "common.cuh"
#include "f32x2.cuh"

namespace b200 {
namespace {

template <typename AT> __device__ __forceinline__ float ldx(const AT* p, int64_t i);
template <> __device__ __forceinline__ float ldx<float>(const float* p, int64_t i) { return p[i]; }
template <> __device__ __forceinline__ float ldx<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }
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

// The walk.  A lane holds a few neighbouring key dimensions of four value columns (so one shared-memory read of k and of q per row
// serves all four, every lane another 16 bytes), a warp owns those four columns, a CTA's four column warps sixteen; the state lives
// in registers as pairs for the packed fp32 arithmetic.  A fifth warp walks n and works out the gate scalars two stages ahead.
// The step's rows are staged 16 at a time, values already times their input weight; nothing in a column's walk waits for another
// lane: the per-lane read-out sums of a stage are added and divided while the next one is walked.  Two CTAs (a cluster) share one
// stored copy of n and m: a cluster barrier keeps the even one from storing them before both have read.
// Bound by issue slots and latency at one to two warps per scheduler (24 packed operations and 6 shared-memory accesses a row and
// warp).  2 048 rows of 8 heads, 128 x 256: 332 us (unpacked, a gate chain of shuffles in every warp: 723 us; packed with
// eight lanes a column, whose 16-byte reads repeat across the warp: 419 us).
constexpr int kScanCols = 16, kScanBlock = 32;   // value columns per CTA; per stored copy of n and m
constexpr int kScanStage = 16;                   // rows staged in shared memory at a time
constexpr int kScanThreads = 160, kNWarp = 4;
constexpr int kPartRow = 136;                    // floats of a row of read-out sums: 32 lanes x 4 columns, rows 32 bytes apart in the banks

struct MlstmArgs {
  const void* qkv;
  const float* gates;
  const int32_t* positions;
  const int32_t* seq_start;
  const int32_t* seq_slots;
  float* state;
  float* out;
  int64_t ld, slot_stride;
  int q_off, k_off, v_off, heads, dim, vd;
  float qscale;
  int max_rows;   // sequences that bring more rows are left alone (0: none)
  int vec;        // rows of q and k can be read 16 bytes at a time
  int vec_state;  // state columns 8 bytes at a time
};

// NP: pairs of dimensions per lane (1, 2, 4: dim up to 64, 128, 256).  A staged row holds 64 NP floats, zero beyond dim; pair i of lane x
// starts at dimension 2 x (NP 1), 4 x + 2 i (NP 2), 4 x + 2 (i & 1) + 128 (i >> 1) (NP 4).
__host__ __device__ constexpr int ml_row(int np) { return 64 * np; }
__host__ __device__ constexpr int ml_buf(int np) { return kScanStage * (2 * ml_row(np) + 2 * kScanCols); }   // q rows | k rows | weighted values, twice each
// two stage buffers; of four stages a (twice), b, exp(-m) per row; n . q of two stages; the gate warp's scratch; read-out sums
__host__ __device__ constexpr int ml_floats(int np) {
  return 2 * ml_buf(np) + 4 * kScanStage * 4 + 2 * kScanStage + 2 * kScanStage + kNWarp * kScanStage * kPartRow + kScanStage * 36;
}

template <int NP>
__device__ __forceinline__ void ml_pairs(const float* row, int lane, uint64_t (&x)[NP]) {
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
__device__ __forceinline__ int ml_dim(int lane, int i) {   // first dimension of the lane's pair i
  return NP == 1 ? 2 * lane : 4 * lane + 2 * (i & 1) + 128 * (i >> 1);
}

// STAGED false: the step has decode rows only (one row per sequence), no shared memory.
template <typename AT, int NP, bool STAGED>
__global__ void __launch_bounds__(kScanThreads) mlstm_scan_kernel(const MlstmArgs a) {
  extern __shared__ __align__(16) float stage[];
  constexpr int ROW = ml_row(NP), BUF = ml_buf(NP);
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, zb = blockIdx.z >> 1, nz = gridDim.z >> 1, jb = blockIdx.z * kScanCols;
  const bool keeper = (blockIdx.z & 1) == 0;   // stores n and m
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows <= 0 || (a.max_rows > 0 && n_rows > a.max_rows)) return;   // the cluster's other CTA leaves too
  const int heads = a.heads, dim = a.dim, vd = a.vd;
  const bool fresh = a.positions[start] == 0;
  const AT* qkv = static_cast<const AT*>(a.qkv);
  float* slot = a.state + (int64_t)a.seq_slots[s] * a.slot_stride;                              // S [heads][vd][dim]
  float* n_st = slot + (int64_t)heads * vd * dim + ((int64_t)h * nz + zb) * dim;                // n [heads][nz][dim]
  float* m_st = slot + (int64_t)heads * vd * dim + (int64_t)heads * nz * dim + (int64_t)h * nz + zb;   // m [heads][nz]
  const int j0 = jb + warp * 4;   // a column warp's first column
  float* S_st = slot + ((int64_t)h * vd + j0) * dim;
  auto load_state = [&](const float* p, uint64_t (&x)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ml_dim<NP>(lane, i);
      if (a.vec_state) x[i] = d < dim ? *reinterpret_cast<const uint64_t*>(p + d) : 0;
      else x[i] = f2::pack(d < dim ? p[d] : 0.f, d + 1 < dim ? p[d + 1] : 0.f);
    }
  };
  auto store_state = [&](float* p, const uint64_t (&x)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ml_dim<NP>(lane, i);
      if (a.vec_state) {
        if (d < dim) *reinterpret_cast<uint64_t*>(p + d) = x[i];
      } else {
        if (d < dim) p[d] = f2::lo(x[i]);
        if (d + 1 < dim) p[d + 1] = f2::hi(x[i]);
      }
    }
  };
  uint64_t S[4][NP], n[NP];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int i = 0; i < NP; ++i) S[c][i] = 0;
    if (!fresh && warp < kNWarp && j0 + c < vd) load_state(S_st + (int64_t)c * dim, S[c]);
  }
#pragma unroll
  for (int i = 0; i < NP; ++i) n[i] = 0;
  float m = fresh ? 0.f : *m_st;
  if (n_rows == 1) {
    // a decode row: every column warp carries its own copy of n beside its columns
    if (!fresh && warp < kNWarp) load_state(n_st, n);
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    if (warp < kNWarp) {
      const AT* row = qkv + (int64_t)start * a.ld;
      const float ig = a.gates[(int64_t)start * 2 * heads + h], fg = a.gates[(int64_t)start * 2 * heads + heads + h];
      const float m_new = fmaxf(fg + m, ig);
      const float da = expf(fg + m - m_new), b = expf(ig - m_new);
      m = m_new;
      const uint64_t aa = f2::both(da), bb = f2::both(b);
      uint64_t nacc = 0, acc[4] = {0, 0, 0, 0}, vv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) vv[c] = f2::both(j0 + c < vd ? ldx<AT>(row, a.v_off + h * vd + j0 + c) : 0.f);
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const int d = ml_dim<NP>(lane, i);
        const uint64_t qq = f2::pack(d < dim ? ldx<AT>(row, a.q_off + h * dim + d) * a.qscale : 0.f, d + 1 < dim ? ldx<AT>(row, a.q_off + h * dim + d + 1) * a.qscale : 0.f);
        const uint64_t bk = f2::mul(bb, f2::pack(d < dim ? ldx<AT>(row, a.k_off + h * dim + d) : 0.f, d + 1 < dim ? ldx<AT>(row, a.k_off + h * dim + d + 1) : 0.f));
        n[i] = f2::fma(aa, n[i], bk);
        nacc = f2::fma(n[i], qq, nacc);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          S[c][i] = f2::fma(aa, S[c][i], f2::mul(bk, vv[c]));
          acc[c] = f2::fma(S[c][i], qq, acc[c]);
        }
      }
      float o[4], nq = f2::sum(nacc);
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] = f2::sum(acc[c]);
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) {
        nq += __shfl_xor_sync(0xffffffffu, nq, x);
#pragma unroll
        for (int c = 0; c < 4; ++c) o[c] += __shfl_xor_sync(0xffffffffu, o[c], x);
      }
      const float mine = lane == 0 ? o[0] : lane == 1 ? o[1] : lane == 2 ? o[2] : o[3];
      if (lane < 4 && j0 + lane < vd) a.out[((int64_t)start * heads + h) * vd + j0 + lane] = mine / (fmaxf(fabsf(nq), expf(-m)) + 1e-6f);
    }
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (warp < kNWarp) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (j0 + c < vd) store_state(S_st + (int64_t)c * dim, S[c]);
    }
    if (keeper && warp == 0) store_state(n_st, n);
    if (keeper && tid == 0) *m_st = m;
    return;
  }
  if (!fresh && warp == kNWarp) load_state(n_st, n);
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");   // n and m have been read
  if constexpr (STAGED) {
    float* sa = stage + 2 * BUF;                          // [4][kScanStage][2] decay of a row, twice
    float* sb = sa + 4 * kScanStage * 2;                  // [4][kScanStage] input weight
    float* em = sb + 4 * kScanStage;                      // [4][kScanStage] exp(-m)
    float* nqs = em + 4 * kScanStage;                     // [2][kScanStage] n . q
    float* gs = nqs + 2 * kScanStage;                     // [2][kScanStage] the gate warp's gates
    float* part = gs + 2 * kScanStage + warp * kScanStage * kPartRow;   // [kScanStage][kPartRow] (n warp: [kScanStage][36])
    const int n_stages = (n_rows + kScanStage - 1) / kScanStage;
    // zeros beyond dim, once: the copies leave them alone
    if (dim < ROW)
      for (int e = tid; e < 2 * BUF; e += kScanThreads) stage[e] = 0.f;
    // rows of a stage travel through registers (converted on the way into shared memory); rows past the portion's end are zeros
    constexpr int PER = 16 / (int)sizeof(AT), CPR = ROW / PER;   // elements of a 16-byte piece, pieces of a padded row
    constexpr int NF = (2 * kScanStage * CPR + kScanThreads - 1) / kScanThreads, NFV = (kScanStage * kScanCols + kScanThreads - 1) / kScanThreads;
    uint4 rq[NF];
    float rv[NFV];
    auto fetch = [&](int st) {
      const int b0 = st * kScanStage, nb = min(kScanStage, n_rows - b0);
      if (a.vec) {
#pragma unroll
        for (int i = 0; i < NF; ++i) {
          const int e = tid + kScanThreads * i, x = e / CPR, c = (e % CPR) * PER, r = x >> 1;
          rq[i] = make_uint4(0u, 0u, 0u, 0u);
          if (r < nb && c < dim)
            rq[i] = __ldg(reinterpret_cast<const uint4*>(qkv + (int64_t)(start + b0 + r) * a.ld + ((x & 1) ? a.k_off : a.q_off) + h * dim + c));
        }
      }
#pragma unroll
      for (int i = 0; i < NFV; ++i) {
        const int e = tid + kScanThreads * i, r = e / kScanCols, c = e % kScanCols;
        rv[i] = (r < nb && jb + c < vd) ? ldx<AT>(qkv + (int64_t)(start + b0 + r) * a.ld, a.v_off + h * vd + jb + c) : 0.f;
      }
    };
    auto put = [&](int st, float* buf) {
      float* sv = buf + 2 * kScanStage * ROW;
      if (a.vec) {
#pragma unroll
        for (int i = 0; i < NF; ++i) {
          const int e = tid + kScanThreads * i, x = e / CPR, c = (e % CPR) * PER, r = x >> 1;
          if (r >= kScanStage || c >= dim) continue;
          float* dst = buf + ((x & 1) * kScanStage + r) * ROW + c;
          const float f = (x & 1) ? 1.f : a.qscale;
          if constexpr (sizeof(AT) == 2) {
            *reinterpret_cast<float4*>(dst) = make_float4(bf16lo(rq[i].x) * f, bf16hi(rq[i].x) * f, bf16lo(rq[i].y) * f, bf16hi(rq[i].y) * f);
            *reinterpret_cast<float4*>(dst + 4) = make_float4(bf16lo(rq[i].z) * f, bf16hi(rq[i].z) * f, bf16lo(rq[i].w) * f, bf16hi(rq[i].w) * f);
          } else {
            *reinterpret_cast<float4*>(dst) =
                make_float4(__uint_as_float(rq[i].x) * f, __uint_as_float(rq[i].y) * f, __uint_as_float(rq[i].z) * f, __uint_as_float(rq[i].w) * f);
          }
        }
      } else {
        const int b0 = st * kScanStage, nb = min(kScanStage, n_rows - b0);
        for (int e = tid; e < 2 * kScanStage * ROW; e += kScanThreads) {
          const int x = e / ROW, c = e % ROW, r = x >> 1;
          if (c < dim)
            buf[((x & 1) * kScanStage + r) * ROW + c] =
                r < nb ? ldx<AT>(qkv + (int64_t)(start + b0 + r) * a.ld, ((x & 1) ? a.k_off : a.q_off) + h * dim + c) * ((x & 1) ? 1.f : a.qscale) : 0.f;
        }
      }
#pragma unroll
      for (int i = 0; i < NFV; ++i) {
        const int e = tid + kScanThreads * i, r = e / kScanCols;
        if (r < kScanStage) {
          const float u = sb[(st & 3) * kScanStage + r] * rv[i];
          *reinterpret_cast<float2*>(sv + 2 * e) = make_float2(u, u);
        }
      }
    };
    // n warp: decays, input weights and exp(-m) of a stage's rows; the running maximum is a chain of one add and one max a row.  Rows
    // past the end leave the state alone (decay 1, weight 0).
    float ig = 0.f, fg = 0.f;
    auto fetch_gates = [&](int st) {
      const int t = st * kScanStage + lane;
      const bool ok = lane < kScanStage && t < n_rows;
      ig = ok ? a.gates[(int64_t)(start + t) * 2 * heads + h] : 0.f;
      fg = ok ? a.gates[(int64_t)(start + t) * 2 * heads + heads + h] : 0.f;
    };
    auto gate_stage = [&](int st) {
      const int nb = min(kScanStage, n_rows - st * kScanStage);
      if (lane < kScanStage) {
        gs[lane] = ig;
        gs[kScanStage + lane] = fg;
      }
      __syncwarp();
      float mp = 0.f, mm = 0.f;
#pragma unroll
      for (int r = 0; r < kScanStage; ++r) {
        const float mn = fmaxf(gs[kScanStage + r] + m, gs[r]);
        if (lane == r) {
          mp = m;
          mm = mn;
        }
        if (r < nb) m = mn;
      }
      if (lane < kScanStage) {
        const int x = (st & 3) * kScanStage + lane;
        const bool ok = lane < nb;
        const float da = ok ? expf(fg + mp - mm) : 1.f;
        *reinterpret_cast<float2*>(sa + 2 * x) = make_float2(da, da);
        sb[x] = ok ? expf(ig - mm) : 0.f;
        em[x] = expf(-mm);
      }
      __syncwarp();
    };
    // sums, normaliser and division of stage st: two lanes a row, sixteen lanes' sums each
    auto finish = [&](int st) {
      const int b0 = st * kScanStage, nb = min(kScanStage, n_rows - b0), r = lane >> 1, half = lane & 1;
      const float* src = part + r * kPartRow + half * 64;
      uint64_t x = 0, y = 0;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + 4 * (i ^ half));   // (the two lanes' banks apart)
        x = f2::add(x, t.x);
        y = f2::add(y, t.y);
      }
      float o[4] = {f2::lo(x), f2::hi(x), f2::lo(y), f2::hi(y)};
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] += __shfl_xor_sync(0xffffffffu, o[c], 1);
      const float den = fmaxf(fabsf(nqs[(st & 1) * kScanStage + r]), em[(st & 3) * kScanStage + r]) + 1e-6f;
      if (r < nb) {
        float* dst = a.out + ((int64_t)(start + b0 + r) * heads + h) * vd + j0 + 2 * half;
        if (j0 + 2 * half < vd) dst[0] = (half ? o[2] : o[0]) / den;
        if (j0 + 2 * half + 1 < vd) dst[1] = (half ? o[3] : o[1]) / den;
      }
      __syncwarp();
    };
    fetch(0);
    if (warp == kNWarp) {
      fetch_gates(0);
      gate_stage(0);
      fetch_gates(1);
      gate_stage(1);
      fetch_gates(2);
    }
    __syncthreads();
    for (int st = 0; st < n_stages; ++st) {
      float* buf = stage + (st & 1) * BUF;
      put(st, buf);
      __syncthreads();   // the stage is there, and the one before has been walked by every warp
      if (st + 1 < n_stages) fetch(st + 1);
      const float* sq = buf;
      const float* sk = buf + kScanStage * ROW;
      const float* su = buf + 2 * kScanStage * ROW + 8 * warp;
      const float* sd = sa + (st & 3) * kScanStage * 2;
      if (warp < kNWarp) {
        if (st > 0) finish(st - 1);
        // row r + 1 is read before row r is worked on (its sums' store would hold the reads back)
        uint64_t k[2][NP], q[2][NP], aa[2];
        ulonglong2 u[2][2];
        auto read = [&](int r) {
          ml_pairs<NP>(sk + r * ROW, lane, k[r & 1]);
          ml_pairs<NP>(sq + r * ROW, lane, q[r & 1]);
          u[r & 1][0] = *reinterpret_cast<const ulonglong2*>(su + r * 2 * kScanCols);
          u[r & 1][1] = *reinterpret_cast<const ulonglong2*>(su + r * 2 * kScanCols + 4);
          aa[r & 1] = *reinterpret_cast<const uint64_t*>(sd + 2 * r);
        };
        read(0);
#pragma unroll
        for (int r = 0; r < kScanStage; ++r) {
          if (r + 1 < kScanStage) read(r + 1);
          const uint64_t uc[4] = {u[r & 1][0].x, u[r & 1][0].y, u[r & 1][1].x, u[r & 1][1].y};
          float o[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint64_t acc = 0;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
              S[c][i] = f2::fma(aa[r & 1], S[c][i], f2::mul(k[r & 1][i], uc[c]));
              acc = i ? f2::fma(S[c][i], q[r & 1][i], acc) : f2::mul(S[c][i], q[r & 1][i]);
            }
            o[c] = f2::sum(acc);
          }
          *reinterpret_cast<float4*>(part + r * kPartRow + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
        }
        __syncwarp();
      } else {
        const float* sbn = sb + (st & 3) * kScanStage;
#pragma unroll 4
        for (int r = 0; r < kScanStage; ++r) {
          uint64_t k[NP], q[NP], acc = 0;
          ml_pairs<NP>(sk + r * ROW, lane, k);
          ml_pairs<NP>(sq + r * ROW, lane, q);
          const uint64_t aa = *reinterpret_cast<const uint64_t*>(sd + 2 * r), bb = f2::both(sbn[r]);
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            n[i] = f2::fma(aa, n[i], f2::mul(bb, k[i]));
            acc = f2::fma(n[i], q[i], acc);
          }
          part[r * 36 + lane] = f2::sum(acc);
        }
        __syncwarp();
        float x = 0.f;   // two lanes a row
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 t = *reinterpret_cast<const float4*>(part + (lane >> 1) * 36 + (lane & 1) * 16 + 4 * i);
          x += (t.x + t.y) + (t.z + t.w);
        }
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        if ((lane & 1) == 0) nqs[(st & 1) * kScanStage + (lane >> 1)] = x;
        gate_stage(st + 2);   // (past the end: neutral rows that nobody reads)
        fetch_gates(st + 3);
      }
    }
    __syncthreads();
    if (warp < kNWarp) finish(n_stages - 1);
  }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (warp < kNWarp) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (j0 + c < vd) store_state(S_st + (int64_t)c * dim, S[c]);
  } else if (keeper) {
    store_state(n_st, n);
    if (lane == 0) *m_st = m;
  }
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

int mlstm_col_blocks(int vd) { return (vd + kScanBlock - 1) / kScanBlock; }

// floats of one layer's recurrent state in a slot: S [heads][vd][dim], n [heads][col blocks][dim], m [heads][col blocks]
int64_t mlstm_state_floats(int heads, int dim, int vd) {
  const int64_t nz = mlstm_col_blocks(vd);
  return (int64_t)heads * vd * dim + (int64_t)heads * nz * dim + (int64_t)heads * nz;
}

template <typename AT>
static int mlstm_scan_t(const MlstmArgs& a, int S, bool single_rows, cudaStream_t s) {
  const dim3 grid(S, a.heads, 2 * mlstm_col_blocks(a.vd)), block(kScanThreads), cluster(1, 1, 2);
#define SCAN1(D, ST)                                                                                                     \
  do {                                                                                                                   \
    static bool done[64] = {};                                                                                           \
    const size_t smem = ST ? (size_t)ml_floats(D) * 4 : 0;                                                               \
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(mlstm_scan_kernel<AT, D, ST>, (int)smem, done));                 \
    B200_CUDA(launch_cluster(mlstm_scan_kernel<AT, D, ST>, grid, block, smem, s, cluster, a));                           \
  } while (0)
#define SCAN(D)                       \
  do {                                \
    if (single_rows) SCAN1(D, false); \
    else SCAN1(D, true);              \
  } while (0)
  if (a.dim <= 64) SCAN(1);
  else if (a.dim <= 128) SCAN(2);
  else SCAN(4);
#undef SCAN1
#undef SCAN
  return B200_OK;
}

int mlstm_scan(bool f32, const void* qkv, int64_t ld, int q_off, int k_off, int v_off, const float* gates, const int32_t* positions,
               const int32_t* seq_start, const int32_t* seq_slots, float* state, int64_t slot_stride, float* out, int S, int heads,
               int dim, int vd, cudaStream_t s, bool single_rows) {
  if (S == 0) return B200_OK;
  B200_REQUIRE(dim > 0 && dim <= 256 && vd > 0, B200_ERR_UNSUPPORTED, "mlstm_scan: key size %d outside (0, 256]", dim);
  B200_REQUIRE(positions && seq_start && seq_slots && state, B200_ERR_INVALID, "mlstm_scan: null argument");
  // longer portions of bf16 rows in chunks on the tensor cores (2 048 rows of 8 heads, 128 x 256: 141 us against 332); decode steps, fp32
  // rows and odd shapes row by row.  How many rows a sequence brings is known on the device only: both kernels are launched, each
  // leaves the other's sequences alone.  Steps of many sequences are mostly decode rows, and the walk fills the SMs.  A chunk kernel's first chunk costs about what 96 rows of the walk do (64 rows of four
  // sequences: 16 us row by row, 22 in chunks)
  constexpr int kWalkRows = 96;
  const bool chunks = !f32 && !single_rows && S <= 16 && mlstm_chunk_supported(qkv, ld, q_off, k_off, v_off, dim, vd);
  if (chunks) {
    const int rc = mlstm_chunk((const __nv_bfloat16*)qkv, ld, q_off, k_off, v_off, gates, positions, seq_start, seq_slots, state, slot_stride, out, S,
                               heads, dim, vd, kWalkRows, s);
    if (rc) return rc;
  }
  MlstmArgs a = {qkv, gates, positions, seq_start, seq_slots, state, out, ld, slot_stride, q_off, k_off, v_off, heads, dim, vd, 1.0f / sqrtf((float)dim), chunks ? kWalkRows : 0, 0, 0};
  const auto at = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr); };
  const int per = f32 ? 4 : 8;   // elements of a 16-byte piece
  a.vec = dim % per == 0 && ld % per == 0 && q_off % per == 0 && k_off % per == 0 && at(qkv) % 16 == 0;
  a.vec_state = dim % 2 == 0 && slot_stride % 2 == 0 && at(state) % 8 == 0;
  if (chunks) {
    const PdlScope after_chunks;
    return mlstm_scan_t<__nv_bfloat16>(a, S, false, s);
  }
  return f32 ? mlstm_scan_t<float>(a, S, single_rows, s) : mlstm_scan_t<__nv_bfloat16>(a, S, single_rows, s);
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
