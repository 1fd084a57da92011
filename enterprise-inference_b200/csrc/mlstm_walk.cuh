// The row-by-row walk of the matrix-memory recurrence (mlstm.cu), which the segments' and the chunks' kernels (mlstm_segment.cu, mlstm_chunk.cu) can take for short portions too.
#pragma once
#include "common.cuh"
#include "f32x2.cuh"

namespace b200 {

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
  double log2_qscale;
  int vec;        // rows of q and k can be read 16 bytes at a time
  int vec_state;  // state columns 8 bytes at a time
  int vec_out;    // outputs 16 bytes at a time
  int both;       // the walk's and the chunks' kernel are both launched, each for its portions
};

// bf16 rows on the tensor cores (mlstm_segment.cu, mlstm_chunk.cu)
bool mlstm_chunk_supported(const MlstmArgs& a);
bool mlstm_segments_fit(const MlstmArgs& a, int S);
int64_t mlstm_chunk_ctas(const MlstmArgs& a, int S);
int mlstm_segments(MlstmArgs a, int S, cudaStream_t s);
int mlstm_chunk(const MlstmArgs& a, int S, cudaStream_t s);

namespace {

template <typename AT> __device__ __forceinline__ float ldx(const AT* p, int64_t i);
template <> __device__ __forceinline__ float ldx<float>(const float* p, int64_t i) { return p[i]; }
template <> __device__ __forceinline__ float ldx<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }

// The walk.  A lane holds a few neighbouring key dimensions of four value columns (so one shared-memory read of k and of q per row
// serves all four, every lane another 16 bytes), a warp owns those four columns, a CTA's eight column warps the 32 that share a stored
// copy of n and m; the state lives in registers as pairs for the packed fp32 arithmetic.  A ninth warp walks n and works out the gate
// scalars two stages ahead.  The step's rows are staged 16 at a time, values already times their input weight; nothing in a column's
// walk waits for another lane: the per-lane read-out sums of a stage are added and divided while the next one is walked.
// Bound by issue slots and latency.  The recurrence of 8 heads of 128 x 256, against the scalar walk before it (gates by a chain of shuffles
// in every warp): 64 rows of one sequence 23.3 -> 17.2 us, 2 048 rows of 16 sequences 316 -> 201 us, 64 decode rows beside others 50 -> 37 us.
// Sixteen columns a CTA in clusters of two are quicker for one sequence (64 rows 14.9 us) and slower for many (64 decode rows 70 us: a
// cluster waits for two free places at a time).
constexpr int kScanCols = 32;                    // value columns of a CTA, which keeps one stored copy of n and m
constexpr int kScanStage = 16;                   // rows staged in shared memory at a time
constexpr int kScanThreads = 288, kNWarp = 8;
constexpr int kChunkFrom = 97;                   // rows of a portion from which chunks pay (97 rows of one sequence: 15 us, walked 23)
constexpr int kSegmentFrom = 193;                // rows of a portion from which segments pay (256 rows of one sequence 20.0 us, in chunks 22.3; 192 in chunks 17.9)
constexpr int kPartRow = 132;                    // floats of a row of read-out sums: 32 lanes x 4 columns, rows 16 bytes apart in the banks

// which of its accesses the walk can make wide
inline void mlstm_walk_widths(MlstmArgs& a, bool f32) {
  const auto at = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr); };
  const int per = f32 ? 4 : 8;   // elements of a 16-byte piece
  a.vec = a.dim % per == 0 && a.ld % per == 0 && a.q_off % per == 0 && a.k_off % per == 0 && at(a.qkv) % 16 == 0;
  a.vec_state = a.dim % 2 == 0 && a.slot_stride % 2 == 0 && at(a.state) % 8 == 0;
}

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

// Columns 32 zb .. of (sequence, head) = blockIdx (x, y), by a whole CTA of kScanThreads. 
template <typename AT, int NP>
__device__ __forceinline__ void mlstm_walk(const MlstmArgs& a, float* stage, int zb, int nz) {
  constexpr int ROW = ml_row(NP), BUF = ml_buf(NP);
  const int s = blockIdx.x, h = blockIdx.y, jb = zb * kScanCols;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows <= 0) return;
  const int heads = a.heads, dim = a.dim, vd = a.vd;
  const bool fresh = a.positions[start] == 0;
  const AT* qkv = static_cast<const AT*>(a.qkv);
  float* slot = a.state + (int64_t)a.seq_slots[s] * a.slot_stride;                              // S [heads][vd][dim]
  float* n_st = slot + (int64_t)heads * vd * dim + ((int64_t)h * nz + zb) * dim;                // n [heads][nz][dim]
  float* m_st = slot + (int64_t)heads * vd * dim + (int64_t)heads * nz * dim + (int64_t)h * nz + zb;   // m [heads][nz]
  const int j0 = jb + warp * 4;   // a column warp's first column
  float* S_st = slot + ((int64_t)h * vd + j0) * dim;
  // (read whether or not the sequence starts here, so that the state does not wait for the position)
  auto load_state = [&](const float* p, bool live, uint64_t (&x)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ml_dim<NP>(lane, i);
      if (a.vec_state) x[i] = live && d < dim ? *reinterpret_cast<const uint64_t*>(p + d) : 0;
      else x[i] = live ? f2::pack(d < dim ? p[d] : 0.f, d + 1 < dim ? p[d + 1] : 0.f) : 0;
    }
  };
  auto or_zero = [&](uint64_t (&x)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; ++i) x[i] = fresh ? 0 : x[i];
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
  for (int c = 0; c < 4; ++c) load_state(S_st + (int64_t)c * dim, warp < kNWarp && j0 + c < vd, S[c]);
  float m = *m_st;
  if (n_rows == 1) {
    // a decode row: every column warp carries its own copy of n beside its columns.  The row and the state are on their way together.
    load_state(n_st, warp < kNWarp, n);
    uint64_t qq[NP], kk[NP], vv[4];
    const AT* row = qkv + (int64_t)start * a.ld;
    const float ig = a.gates[(int64_t)start * 2 * heads + h];
    const float fg = a.gates[(int64_t)start * 2 * heads + heads + h];
#pragma unroll
    for (int c = 0; c < 4; ++c) vv[c] = f2::both(warp < kNWarp && j0 + c < vd ? ldx<AT>(row, a.v_off + h * vd + j0 + c) : 0.f);
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ml_dim<NP>(lane, i);
      const AT *q = row + a.q_off + h * dim, *k = row + a.k_off + h * dim;
      qq[i] = f2::pack(d < dim ? ldx<AT>(q, d) * a.qscale : 0.f, d + 1 < dim ? ldx<AT>(q, d + 1) * a.qscale : 0.f);
      kk[i] = f2::pack(d < dim ? ldx<AT>(k, d) : 0.f, d + 1 < dim ? ldx<AT>(k, d + 1) : 0.f);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) or_zero(S[c]);
    or_zero(n);
    if (fresh) m = 0.f;
    __syncthreads();   // every warp has read n and m
    if (warp < kNWarp) {
      const float m_new = fmaxf(fg + m, ig);
      const float da = expf(fg + m - m_new), b = expf(ig - m_new);
      m = m_new;
      const uint64_t aa = f2::both(da), bb = f2::both(b);
      uint64_t nacc = 0, acc[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const uint64_t bk = f2::mul(bb, kk[i]);
        n[i] = f2::fma(aa, n[i], bk);
        nacc = f2::fma(n[i], qq[i], nacc);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          S[c][i] = f2::fma(aa, S[c][i], f2::mul(bk, vv[c]));
          acc[c] = f2::fma(S[c][i], qq[i], acc[c]);
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
    if (warp < kNWarp) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (j0 + c < vd) store_state(S_st + (int64_t)c * dim, S[c]);
    }
    if (warp == 0) store_state(n_st, n);
    if (tid == 0) *m_st = m;
    return;
  }
  load_state(n_st, warp == kNWarp, n);
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
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + 4 * (i ^ (4 * half)));   // (all eight lanes of a phase on banks of their own)
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
  if (warp == kNWarp) fetch_gates(0);
#pragma unroll
  for (int c = 0; c < 4; ++c) or_zero(S[c]);
  or_zero(n);
  if (fresh) m = 0.f;
  if (warp == kNWarp) {
    gate_stage(0);
    if (n_stages > 1) {
      fetch_gates(1);
      gate_stage(1);
      fetch_gates(2);
    }
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
        if (st * kScanStage + r >= n_rows) break;
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
      if (st + 2 < n_stages) {
        gate_stage(st + 2);
        fetch_gates(st + 3);   // (past the end: nothing to read)
      }
    }
  }
  __syncthreads();
  if (warp < kNWarp) finish(n_stages - 1);
  if (warp < kNWarp) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (j0 + c < vd) store_state(S_st + (int64_t)c * dim, S[c]);
  } else {
    store_state(n_st, n);
    if (lane == 0) *m_st = m;
  }
}

}  // namespace
}  // namespace b200
