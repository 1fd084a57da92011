// The matrix-memory recurrence of mlstm.cu over portions of a few chunks of 64 rows on the tensor cores (bf16 rows), a CTA of a cluster sixteen value columns.
//
// With F_t the sum of the log forget gates of the chunk up to row t, m_t = F_t + max(m_0, max_{s<=t} (i_s - F_s)) is the running maximum
// of the row-by-row walk, and
//   S_t = exp(F_t + m_0 - m_t) S_0 + sum_{s<=t} exp(F_t - F_s + i_s - m_t) k_s v_s^T          (n_t likewise with v = 1)
// so a chunk is four products: P = Q K^T, weighted by the exponentials under the diagonal; P V; Q S_0; K^T (w V) for the next state.
// Everything that was fp32 in the walk stays so in effect: sums F are taken in 64 bits (differences of large sums), an fp32 operand (P, S_0,
// w V) enters the bf16 MMA as three bf16 terms (24 bits) against rows that are bf16 to begin with, accumulators are fp32.  n is carried
// as a 17th column with value 1.
//
// One CTA per (sequence, head, 16 value columns) walks the chunks; two neighbours share one stored copy of n and m, and a barrier of the cluster keeps either from storing before both have read.
// Warps w of 8: rows 16 (w % 4) of P and O, the key blocks (and for Q S_0 the dimensions) dealt to the two warps of a row group, whose
// sums meet in shared memory; dimensions 16 w of the state, kept in fp32 accumulator fragments.  A ninth warp works out the next
// chunk's gate scalars.  Rows arrive by cp.async a chunk ahead.
// Bound by latency (about 800 instructions a warp and chunk, two barriers, 4.5 us): 97 rows of 8 heads, 128 x 256: 12.9 us, 160: 17.8 (in segments 16.3 and
// 18.5, walked 23 and 37).
#pragma once
#include "mlstm_walk.cuh"

namespace b200 {
namespace {

constexpr int kMcRows = 64, kMcCols = 16, kMcW = 24;   // rows of a chunk; value columns; columns with n and its padding (bf16 rows of 48 bytes)
constexpr int kMcThreads = 288, kMcGate = 8;

__device__ __forceinline__ uint32_t sa(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sa(p)) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sa(p)) : "memory");
}
__device__ __forceinline__ void ldsm2t(uint32_t (&r)[2], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(sa(p)) : "memory");
}
__device__ __forceinline__ void mc_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16 bytes, or zeros (live false)
__device__ __forceinline__ void cp16z(void* dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
// two fp32 values as three packed bf16 terms each: x = t0 + t1 + t2 up to 2^-24 of x (each rest is exact)
__device__ __forceinline__ void split3(float x, float y, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  t0 = pack_bf16(x, y);
  const float x1 = x - bf16lo(t0), y1 = y - bf16hi(t0);
  t1 = pack_bf16(x1, y1);
  t2 = pack_bf16(x1 - bf16lo(t1), y1 - bf16hi(t1));
}

// either of two packed bf16 an infinity or NaN
__device__ __forceinline__ bool odd2(uint32_t x) { return (x & 0x7f800000u) == 0x7f800000u || (x & 0x7f80u) == 0x7f80u; }

struct GateRows {   // of one chunk
  double a[kMcRows];       // F_t - m_t
  double g[kMcRows];       // i_t - F_t
  float alpha[kMcRows];    // exp(F_t + m_0 - m_t)
  float em[kMcRows];       // exp(-m_t)
  float w[kMcRows];        // exp(F_L - F_t + i_t - m_L)
  float gamma, pad;     // exp(F_L + m_0 - m_L)
};

template <int KS>
struct McSmem {
  static constexpr int QS = KS * 16 + 8;   // bf16 per staged q / k row
  __nv_bfloat16 q[2][kMcRows][QS], k[2][kMcRows][QS], v[2][kMcRows][kMcW], w[3][kMcRows][kMcW], s[3][KS * 16][kMcW];
  float o[kMcRows][kMcW + 2];   // one warp's sums of a row group, for the other
  GateRows gate[2];
  int odd[2];   // a value of the chunk is not finite
};

// One warp's sums of a chunk (three column tiles of its 16 rows) when a value is not finite: every row adds its own keys one by one, so that nothing
// is multiplied with a later row's value; what comes from the state before is as in the kernel.
template <int KS>
__device__ __noinline__ void mc_careful(const McSmem<KS>& sm, int buf, int hf, int rg, int lane, float qscale, float* out) {
  const GateRows& gt = sm.gate[buf];
  const int g = lane >> 2, t4 = lane & 3;
  float O[3][4] = {}, J[3][4] = {};
#pragma unroll 1
  for (int sb = hf * 16; sb <= rg; sb += 32) {
    float p[2][4] = {};
#pragma unroll 1
    for (int k = 0; k < KS; ++k) {
      uint32_t qk[4], b[4];
      ldsm4(qk, &sm.q[buf][rg + (lane & 15)][k * 16 + (lane >> 4) * 8]);
      ldsm4(b, &sm.k[buf][sb + (lane & 7) + ((lane >> 4) << 3)][k * 16 + ((lane >> 3) & 1) * 8]);
      mc_mma(p[0], qk, b[0], b[1]);
      mc_mma(p[1], qk, b[2], b[3]);
    }
#pragma unroll 1
    for (int j = 0; j < 16; ++j) {
      const int from = (lane & ~3) | ((j & 7) >> 1);
      const __nv_bfloat16* v = &sm.v[buf][sb + j][2 * t4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int t = rg + g + 8 * x;
        const float w = __shfl_sync(0xffffffffu, j < 8 ? (j & 1 ? p[0][2 * x + 1] : p[0][2 * x]) : (j & 1 ? p[1][2 * x + 1] : p[1][2 * x]), from) * qscale *
                        expf((float)(gt.a[t] + gt.g[sb + j]));
        if (sb + j <= t) {
#pragma unroll
          for (int n = 0; n < 3; ++n) {
            O[n][2 * x] = fmaf(w, __bfloat162float(v[n * 8]), O[n][2 * x]);
            O[n][2 * x + 1] = fmaf(w, __bfloat162float(v[n * 8 + 1]), O[n][2 * x + 1]);
          }
        }
      }
    }
  }
#pragma unroll 1
  for (int k = hf * (KS / 2); k < (hf + 1) * (KS / 2); ++k) {
    uint32_t qk[4];
    ldsm4(qk, &sm.q[buf][rg + (lane & 15)][k * 16 + (lane >> 4) * 8]);
#pragma unroll
    for (int x = 2; x >= 0; --x) {
      uint32_t b4[4], b2[2];
      ldsm4t(b4, &sm.s[x][k * 16 + (lane & 15)][(lane >> 4) * 8]);
      ldsm2t(b2, &sm.s[x][k * 16 + (lane & 15)][kMcCols]);
      mc_mma(J[0], qk, b4[0], b4[1]);
      mc_mma(J[1], qk, b4[2], b4[3]);
      mc_mma(J[2], qk, b2[0], b2[1]);
    }
  }
#pragma unroll
  for (int n = 0; n < 3; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[n * 4 + i] = fmaf(gt.alpha[rg + g + 8 * (i >> 1)] * qscale, J[n][i], O[n][i]);
}

// Columns 16 block .. of (sequence, head) = blockIdx (x, y), by the first kMcThreads threads of a CTA (the others have left); every CTA of the cluster comes here.
// KS: 16-wide steps over the (zero padded) key dimensions
// ROLE: all warps (0), or those with rows (1) and the gate warp (2) in code of their own, for a register count of their own.
template <int KS, int ROLE>
__device__ __forceinline__ void mlstm_chunks(const MlstmArgs& a, unsigned char* raw, int block) {
  McSmem<KS>& sm = *reinterpret_cast<McSmem<KS>*>(raw);
  const int s = blockIdx.x, h = blockIdx.y, nz = (a.vd + kScanCols - 1) / kScanCols, zb = block >> 1, jb = block * kMcCols;
  const bool keeper = (block & 1) == 0 && zb < nz;   // stores n and m
  const int tid = threadIdx.x, warp = ROLE == 2 ? kMcGate : tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const bool gates = ROLE == 2 || (ROLE == 0 && warp == kMcGate);
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  const int heads = a.heads, dim = a.dim, vd = a.vd;
  const bool fresh = a.positions[start] == 0;
  float* slot = a.state + (int64_t)a.seq_slots[s] * a.slot_stride;                                     // S [heads][vd][dim]
  const int zr = min(zb, nz - 1);   // (CTAs beyond the columns only meet the others)
  float* n_st = slot + (int64_t)heads * vd * dim + ((int64_t)h * nz + zr) * dim;                       // n [heads][nz][dim]
  float* m_st = slot + (int64_t)heads * vd * dim + (int64_t)heads * nz * dim + (int64_t)h * nz + zr;   // m [heads][nz]
  float* S_st = slot + ((int64_t)h * vd + jb) * dim;
  const int n_chunks = (n_rows + kMcRows - 1) / kMcRows;
  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.qkv) + (int64_t)start * a.ld;

  auto fetch = [&](int c) {   // warps 0..7
    const int b0 = c * kMcRows, buf = c & 1;
    for (int e = tid; e < kMcRows * KS * 2; e += 256) {
      const int r = e / (KS * 2), d = (e % (KS * 2)) * 8;
      const bool live = b0 + r < n_rows && d < dim;
      const __nv_bfloat16* row = src + (live ? (int64_t)(b0 + r) * a.ld + h * dim + d : 0);
      cp16z(&sm.q[buf][r][d], row + (live ? a.q_off : 0), live);
      cp16z(&sm.k[buf][r][d], row + (live ? a.k_off : 0), live);
    }
    if (tid < kMcRows * 2) {
      const int r = tid >> 1, c8 = (tid & 1) * 8;
      const bool live = b0 + r < n_rows && jb + c8 < vd;
      cp16z(&sm.v[buf][r][c8], src + (live ? (int64_t)(b0 + r) * a.ld + a.v_off + h * vd + jb + c8 : 0), live);
    }
  };
  // state of this warp's 16 dimensions: accumulator fragments of two column tiles and of n (column 16)
  float S[3][4];
#pragma unroll
  for (int n = 0; n < 3; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = warp * 16 + g + (i >> 1) * 8, col = n * 8 + 2 * t4 + (i & 1);
      S[n][i] = 0.f;
      if (!fresh && (!gates && warp < KS) && d < dim) {
        if (n < 2 && jb + col < vd) S[n][i] = S_st[(int64_t)col * dim + d];
        if (n == 2 && col == kMcCols) S[n][i] = n_st[d];
      }
    }
  auto publish = [&]() {   // the state as three bf16 terms, for everybody's Q S (nobody reads it between a chunk's second barrier and the next one's first)
    if ((!gates && warp < KS)) {
#pragma unroll
      for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t t[3];
          split3(S[n][2 * hf], S[n][2 * hf + 1], t[0], t[1], t[2]);
#pragma unroll
          for (int x = 0; x < 3; ++x) *reinterpret_cast<uint32_t*>(&sm.s[x][warp * 16 + g + hf * 8][n * 8 + 2 * t4]) = t[x];
        }
    }
  };
  double m0 = fresh ? 0.0 : (double)*m_st;   // (the gate warp's)
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");   // n and m have been read
  float ig[2], fg[2];
  auto fetch_gates = [&](int c) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int t = c * kMcRows + lane + 32 * x;
      const bool ok = t < n_rows;
      const float* p = a.gates + (int64_t)(start + (ok ? t : 0)) * 2 * heads + h;
      ig[x] = ok ? p[0] : -INFINITY;   // rows past the end: no weight, no decay
      fg[x] = ok ? p[heads] : 0.f;
    }
  };
  auto gate_chunk = [&](GateRows& o) {
    double F[2], G[2], M[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {   // inclusive sums (a gate below -1e5 leaves nothing in fp32 either way)
      F[x] = fg[x] < -1e5f ? -1e5f : fg[x];   // (NaN stays)
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, F[x], d);
        if (lane >= d) F[x] += v;
      }
    }
    F[1] += __shfl_sync(0xffffffffu, F[0], 31);
#pragma unroll
    for (int x = 0; x < 2; ++x) {   // inclusive maxima of i - F
      G[x] = (double)ig[x] - F[x];
      M[x] = G[x];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, M[x], d);
        if (lane >= d) M[x] = fmax(M[x], v);
      }
    }
    M[1] = fmax(M[1], __shfl_sync(0xffffffffu, M[0], 31));
    float m[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) m[x] = (float)(F[x] + fmax(m0, M[x]));
    const double FL = __shfl_sync(0xffffffffu, F[1], 31);
    const double mL = (double)__shfl_sync(0xffffffffu, m[1], 31);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int t = lane + 32 * x;
      o.a[t] = F[x] - (double)m[x];
      o.g[t] = G[x];
      o.alpha[t] = expf((float)(F[x] + m0 - (double)m[x]));
      o.em[t] = expf(-m[x]);
      o.w[t] = expf((float)(G[x] + (FL - mL)));
    }
    if (lane == 0) o.gamma = expf((float)(FL + m0 - mL));
    m0 = mL;
  };
  // the ones column of v (and zeros beside it), once: the copies leave it alone
  for (int e = tid; e < 2 * kMcRows * 8; e += kMcThreads) sm.v[e / (kMcRows * 8)][(e / 8) % kMcRows][kMcCols + e % 8] = __float2bfloat16_rn(e % 8 == 0 ? 1.f : 0.f);
  if (!gates) {
    fetch(0);
    publish();
  } else {
    fetch_gates(0);
    gate_chunk(sm.gate[0]);
    fetch_gates(1);
  }
  // the row groups of a scheduler's two warps add up to about the same number of key blocks
  const int hf = warp >> 2, rg = (hf ? 3 - (warp & 3) : warp & 3) * 16;
  for (int c = 0; c < n_chunks; ++c) {
    const int buf = c & 1;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();   // rows, gates and state of the chunk are there; the chunk before has been finished with
    const GateRows& gt = sm.gate[buf];
    if (gates) {
      // (beside the other warps' products: inside them the same question cost 4 % of the whole)
      bool odd = false;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const uint4 v = *reinterpret_cast<const uint4*>(&sm.v[buf][lane + 32 * (x >> 1)][(x & 1) * 8]);
        odd |= odd2(v.x) || odd2(v.y) || odd2(v.z) || odd2(v.w);
      }
      odd = __any_sync(0xffffffffu, odd);
      if (lane == 0) sm.odd[buf] = odd;
      __syncwarp();
      asm volatile("bar.arrive 1, 288;" ::: "memory");
      gate_chunk(sm.gate[buf ^ 1]);
      fetch_gates(c + 2);
      continue;
    }
    if (c + 1 < n_chunks) fetch(c + 1);
    for (int e = tid; e < kMcRows * kMcW / 2; e += 256) {   // w v as three terms
      const int r = e / (kMcW / 2), col = (e % (kMcW / 2)) * 2;
      const uint32_t v2 = *reinterpret_cast<const uint32_t*>(&sm.v[buf][r][col]);
      const float w = gt.w[r];
      uint32_t x[3];
      split3(w * bf16lo(v2), w * bf16hi(v2), x[0], x[1], x[2]);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&sm.w[i][r][col]) = x[i];
    }
    uint32_t qf[KS][4];
#pragma unroll
    for (int k = 0; k < KS; ++k) ldsm4(qf[k], &sm.q[buf][rg + (lane & 15)][k * 16 + (lane >> 4) * 8]);
    float O[3][4] = {}, I[3][3][4] = {};   // within the chunk; from the state before it, one sum per term (short chains)
    const double a_lo = gt.a[rg + g], a_hi = gt.a[rg + g + 8];
    for (int sb = hf * 16; sb <= rg; sb += 32) {   // key blocks up to the diagonal
      float p[2][4] = {};
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        uint32_t b[4];
        ldsm4(b, &sm.k[buf][sb + (lane & 7) + ((lane >> 4) << 3)][k * 16 + ((lane >> 3) & 1) * 8]);
        mc_mma(p[0], qf[k], b[0], b[1]);
        mc_mma(p[1], qf[k], b[2], b[3]);
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = rg + g + (i >> 1) * 8, j = sb + n * 8 + 2 * t4 + (i & 1);
          // (selected, not weighted with 0: a later row's key may be anything)
          p[n][i] = j <= t ? p[n][i] * a.qscale * expf((float)(((i >> 1) ? a_hi : a_lo) + gt.g[j])) : 0.f;
        }
      uint32_t pa[3][4];
      split3(p[0][0], p[0][1], pa[0][0], pa[1][0], pa[2][0]);
      split3(p[0][2], p[0][3], pa[0][1], pa[1][1], pa[2][1]);
      split3(p[1][0], p[1][1], pa[0][2], pa[1][2], pa[2][2]);
      split3(p[1][2], p[1][3], pa[0][3], pa[1][3], pa[2][3]);
      uint32_t v4[4], v2[2];
      ldsm4t(v4, &sm.v[buf][sb + (lane & 15)][(lane >> 4) * 8]);
      ldsm2t(v2, &sm.v[buf][sb + (lane & 15)][kMcCols]);
#pragma unroll
      for (int x = 2; x >= 0; --x) {
        mc_mma(O[0], pa[x], v4[0], v4[1]);
        mc_mma(O[1], pa[x], v4[2], v4[3]);
        mc_mma(O[2], pa[x], v2[0], v2[1]);
      }
    }
    if (c > 0 || !fresh) {   // (else the state is zeros)
#pragma unroll
    for (int kk = 0; kk < KS / 2; ++kk) {
      uint32_t qk[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qk[i] = hf ? qf[KS / 2 + kk][i] : qf[kk][i];
      const int k = hf * (KS / 2) + kk;
#pragma unroll
      for (int x = 2; x >= 0; --x) {
        uint32_t b4[4], b2[2];
        ldsm4t(b4, &sm.s[x][k * 16 + (lane & 15)][(lane >> 4) * 8]);
        ldsm2t(b2, &sm.s[x][k * 16 + (lane & 15)][kMcCols]);
        mc_mma(I[x][0], qk, b4[0], b4[1]);
        mc_mma(I[x][1], qk, b4[2], b4[3]);
        mc_mma(I[x][2], qk, b2[0], b2[1]);
      }
    }
    }
    const float al[2] = {gt.alpha[rg + g] * a.qscale, gt.alpha[rg + g + 8] * a.qscale};
#pragma unroll
    for (int n = 0; n < 3; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) O[n][i] = fmaf(al[i >> 1], (I[2][n][i] + I[1][n][i]) + I[0][n][i], O[n][i]);
    if (hf) {
#pragma unroll
      for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int x = 0; x < 2; ++x) *reinterpret_cast<float2*>(&sm.o[rg + g + 8 * x][n * 8 + 2 * t4]) = make_float2(O[n][2 * x], O[n][2 * x + 1]);
    }
    asm volatile("bar.sync 1, 288;" ::: "memory");   // w v is complete, the other warps' sums and the gate warp's look at the values are there
    const int odd = sm.odd[buf];
    if ((!gates && warp < KS)) {
      float U[3][3][4] = {};
#pragma unroll
      for (int k = 0; k < kMcRows / 16; ++k) {
        uint32_t ka[4];
        ldsm4t(ka, &sm.k[buf][k * 16 + (lane & 7) + ((lane >> 4) << 3)][warp * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
        for (int x = 2; x >= 0; --x) {
          uint32_t b4[4], b2[2];
          ldsm4t(b4, &sm.w[x][k * 16 + (lane & 15)][(lane >> 4) * 8]);
          ldsm2t(b2, &sm.w[x][k * 16 + (lane & 15)][kMcCols]);
          mc_mma(U[x][0], ka, b4[0], b4[1]);
          mc_mma(U[x][1], ka, b4[2], b4[3]);
          mc_mma(U[x][2], ka, b2[0], b2[1]);
        }
      }
      const float gamma = gt.gamma;
#pragma unroll
      for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[n][i] = fmaf(gamma, S[n][i], (U[2][n][i] + U[1][n][i]) + U[0][n][i]);
    }
    if (odd) {
      // in the blocks on the diagonal the products of such a value with the zeros above it reached earlier rows: the sums once more, with care
      float o[12];
      mc_careful(sm, buf, hf, rg, lane, a.qscale, o);
#pragma unroll
      for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) O[n][i] = o[n * 4 + i];
      if (hf) {
#pragma unroll
        for (int n = 0; n < 3; ++n)
#pragma unroll
          for (int x = 0; x < 2; ++x) *reinterpret_cast<float2*>(&sm.o[rg + g + 8 * x][n * 8 + 2 * t4]) = make_float2(O[n][2 * x], O[n][2 * x + 1]);
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
    }
    publish();
    if (!hf) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int t = rg + g + 8 * x, row = c * kMcRows + t;
        float o[3][2];
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          const float2 y = *reinterpret_cast<const float2*>(&sm.o[t][n * 8 + 2 * t4]);
          o[n][0] = O[n][2 * x] + y.x;
          o[n][1] = O[n][2 * x + 1] + y.y;
        }
        const float nq = __shfl_sync(0xffffffffu, o[2][0], lane & ~3);   // column 16 sits with the first lane of four
        const float den = fmaxf(fabsf(nq), gt.em[t]) + 1e-6f;
        if (row < n_rows) {
          float* dst = a.out + ((int64_t)(start + row) * heads + h) * vd + jb;
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int col = n * 8 + 2 * t4 + i;
              if (jb + col < vd) dst[col] = o[n][i] / den;
            }
        }
      }
    }
  }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if ((!gates && warp < KS)) {
#pragma unroll
    for (int n = 0; n < 3; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = warp * 16 + g + (i >> 1) * 8, col = n * 8 + 2 * t4 + (i & 1);
        if (d >= dim) continue;
        if (n < 2 && jb + col < vd) S_st[(int64_t)col * dim + d] = S[n][i];
        if (n == 2 && col == kMcCols && keeper) n_st[d] = S[n][i];
      }
  } else if (gates && keeper && lane == 0) {
    *m_st = (float)m0;   // (chunks past the last row leave it alone)
  }
}

}  // namespace
}  // namespace b200
