// Paged causal attention over latent cache rows on the tensor cores (bf16 serving mode of B200_MIXER_LATENT), over the whole
// context or over a sliding window of its last `window` keys.
//
// One kv head serves every query head, and a key row's leading `rank` entries are its value, so all heads of a token share
// every byte of the cache: a CTA takes 16 (row, head) pairs of one run of consecutive rows of a sequence and walks the
// context in tiles of 64 keys.  Per tile the key rows are gathered once into shared memory (cp.async, 16-byte chunks through
// the block table), S = Q K^T and O += P V run as bf16 mma.sync m16n8k16 with fp32 accumulators, and the softmax between
// them is fp32: scores scaled and masked per pair (a pair sees keys below its own context length), running maximum and sum
// per pair, weights rounded to bf16 only as the second product's operand.  An optional per-head sink joins the denominator
// at the end.  Warp w (of 8) owns keys 8w..8w+7 of a tile for the scores and value columns 16(w + 8g) .. for the output.
//
// Steps with few (row, head) pairs and long contexts split the context over several CTAs per pair group (n_splits): each
// leaves unnormalised sums with its maximum and denominator, a merge kernel combines them.
//
// The same kernel serves grouped-query attention with a value cache of its own (paged_attn_mma): the pairs of a CTA are then
// (row, head) pairs of ONE kv head's group, the key tile [64][dim] and the value tile [64][vdim] are gathered side by side.
//
// Queries come as fp32 rows [T][heads][krow] (rounded to bf16 when staged); output rows are bf16 [T][heads][rank].
// Shapes: krow and rank multiples of 16, rank <= 512.  Everything else (and the 32-bit mode) takes attn_anydim.cu; both walk
// the same cache and the same run list, and agree within bf16 rounding of the operands.
#include <algorithm>
#include <climits>

#include "runs.cuh"

namespace b200 {
namespace {

constexpr int kLaKeys = 64, kLaPairs = 16, kLaWarps = 8, kLaThreads = kLaWarps * 32;
constexpr int kSsStride = kLaKeys + 4;    // fp32 score rows
constexpr int kPsStride = kLaKeys + 8;    // bf16 weight rows (144 bytes: 16-byte aligned, conflict-free for ldmatrix)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm_x2(uint32_t (&r)[2], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void mma_bf16(float& c0, float& c1, float& c2, float& c3, const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c0), "+f"(c1), "+f"(c2), "+f"(c3)
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// NG: 16-column output groups per warp (rank <= 128 NG).  EX: score cap, distance bias, per-head gate and kept first keys of AttnExtra.
// MANY: launched beside a tcgen05 kernel for its share of the runs, as many CTAs as fit the device, each of which walks over items; otherwise one
// item a CTA (with the loops in every launch 128 decode rows took 65.2 us, without 64.3).
// LO: weights of 16 bits, in two bf16 terms, for long steps whose heads attn_rows_tc.cu had taken with such weights.
template <int NG, bool EX, bool MANY, bool LO>
__global__ void __launch_bounds__(kLaThreads, NG == 1 ? 4 : NG == 2 ? 3 : 2)
latent_attn_mma_kernel(const float* __restrict__ q, const __nv_bfloat16* __restrict__ kc, const __nv_bfloat16* __restrict__ vc,
                       int kv_heads, const int32_t* __restrict__ block_table,
                       int bt_stride, const int32_t* __restrict__ row_to_seq, const int32_t* __restrict__ ctx_lens,
                       __nv_bfloat16* __restrict__ out, const int32_t* __restrict__ runs, const int32_t* __restrict__ n_runs, int heads,
                       int krow, int rank, int block_size, float scale, const float* __restrict__ sink, int n_splits,
                       float* __restrict__ part, int window, AttnExtra ex, RunShare share) {
  extern __shared__ __align__(16) unsigned char smraw[];
  pdl_wait();
  pdl_launch_dependents();
  // G query heads share kv head g; a pair i of the group is (row t0 + i / G, head g G + i % G).  Latent rows: one kv head, G = heads.
  const int G = heads / kv_heads;
  const int n_items = *n_runs, short_pairs = MANY ? run_share(share, G) : 0;
  if (MANY && short_pairs == 0) return;
  // the CTAs that share a run's chunks of pairs: as many as the device has places for (all G of them where it does not matter)
  const int lanes = n_items * kv_heads * n_splits, chunks = MANY ? min(G, max(1, 8 * kNumSMs / max(lanes, 1))) : G;
  const int total = MANY ? lanes * chunks : 1;
  for (int v = MANY ? blockIdx.x : 0; v < total;) {
  int ticket = 0;   // the next item is asked for before this one is worked on
  if (MANY && threadIdx.x == 0) ticket = gridDim.x + atomicAdd(share.ticket, 1);
  // a run's first chunks of pairs lead, so that chunks that do not exist come last
  const int item = MANY ? v % n_items : blockIdx.x, c0 = MANY ? v / lanes : blockIdx.y % G;
  const int g = MANY ? v / n_items % kv_heads : blockIdx.y / G, split = MANY ? v % lanes / (n_items * kv_heads) : blockIdx.z;
  if (!MANY && item >= n_items) return;
  const int t0 = runs[2 * item], run = runs[2 * item + 1], nr = run & kRunLength;
  const int nq = !MANY || run_is_short(short_pairs, run, G) ? nr * G : 0;
  for (int i0 = c0 * kLaPairs; i0 < nq; i0 += chunks * kLaPairs) {
  const int ks = krow + 8;   // bf16 elements per staged row: 16-byte aligned, 4 words off a bank multiple
  // a value cache of its own (vc) is staged beside the keys in rows of rank + 8; else a key row's leading entries are its value
  const int vs = vc ? rank + 8 : ks;
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smraw);      // [64][ks]
  __nv_bfloat16* Vs = vc ? Ks + kLaKeys * ks : Ks;                  // [64][vs]
  __nv_bfloat16* Qs = Vs + (vc ? kLaKeys * vs : kLaKeys * ks);      // [16][ks]
  float* Ss = reinterpret_cast<float*>(Qs + kLaPairs * ks);         // [16][68]
  __nv_bfloat16* Ps = reinterpret_cast<__nv_bfloat16*>(Ss + kLaPairs * kSsStride);   // [16][72]
  float* corr = reinterpret_cast<float*>(Ps + kLaPairs * kPsStride);                 // [16]
  float* mrow = corr + kLaPairs;
  float* lrow = mrow + kLaPairs;
  int* ctxp = reinterpret_cast<int*>(lrow + kLaPairs);
  int* lop = ctxp + kLaPairs;   // the first key a pair sees (0 without a window)
  __nv_bfloat16* Pl = reinterpret_cast<__nv_bfloat16*>(lop + kLaPairs);   // LO: [16][72], what rounding took from the weights
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < kLaPairs) {
    const int i = i0 + tid;
    ctxp[tid] = i < nq ? ctx_lens[t0 + i / G] : 0;
    lop[tid] = window > 0 ? max(ctxp[tid] - window, 0) : 0;
    mrow[tid] = -INFINITY;
    lrow[tid] = 0.f;
  }
  for (int e = tid; e < kLaPairs * krow; e += kLaThreads) {
    const int p = e / krow, d = e % krow, i = i0 + p;
    Qs[p * ks + d] = __float2bfloat16_rn(i < nq ? q[((int64_t)(t0 + i / G) * heads + g * G + i % G) * krow + d] : 0.f);
  }
  const int last_row = min(nr - 1, (i0 + kLaPairs - 1) / G);
  const int ctx_max = ctx_lens[t0 + last_row];
  const int32_t* bt = block_table + (int64_t)(row_to_seq ? row_to_seq[t0] : t0) * bt_stride;
  const int cpr = krow >> 3, cpv = rank >> 3;   // 16-byte chunks per key / value row
  float o[NG][8];
#pragma unroll
  for (int cg = 0; cg < NG; ++cg)
#pragma unroll
    for (int j = 0; j < 8; ++j) o[cg][j] = 0.f;
  __syncthreads();

  // with n_splits > 1 this CTA walks only its share of the tiles and leaves unnormalised sums for the merge kernel
  // (with a window the walk starts at the tile that holds the oldest key the group's first row sees)
  const int tile0 = window > 0 ? max(ctx_lens[t0 + i0 / G] - window, 0) / kLaKeys : 0;
  // first keys that the window keeps: their tiles lead the walk, those between them and the window are skipped
  const int keep = EX ? ex.keep_first : 0, lead = EX ? min((keep + kLaKeys - 1) / kLaKeys, tile0) : 0;
  const int tiles = (ctx_max + kLaKeys - 1) / kLaKeys - tile0 + lead, per = (tiles + n_splits - 1) / n_splits;
  const int walk_lo = split * per, walk_hi = min(tiles, (split + 1) * per);
  for (int w = walk_lo; w < walk_hi; ++w) {
    const int base = (w < lead ? w : w - lead + tile0) * kLaKeys;
    const int n = min(kLaKeys, ctx_max - base);
    {
      // four threads per key row, alternate 16-byte chunks: one block-table lookup per thread and tile
      const int r = tid >> 2;
      __nv_bfloat16* dst = Ks + r * ks;
      __nv_bfloat16* dstv = Vs + r * vs;
      if (r < n) {
        const int j = base + r;
        const int64_t crow = ((int64_t)bt[j / block_size] * kv_heads + g) * block_size + j % block_size;
        const __nv_bfloat16* src = kc + crow * krow;
        for (int c = tid & 3; c < cpr; c += 4) cp_async16(dst + c * 8, src + c * 8);
        if (vc) {
          const __nv_bfloat16* srcv = vc + crow * rank;
          for (int c = tid & 3; c < cpv; c += 4) cp_async16(dstv + c * 8, srcv + c * 8);
        }
      } else {
        // rows past the context: finite values under zero weights
        for (int c = tid & 3; c < cpr; c += 4) *reinterpret_cast<uint4*>(dst + c * 8) = make_uint4(0u, 0u, 0u, 0u);
        if (vc)
          for (int c = tid & 3; c < cpv; c += 4) *reinterpret_cast<uint4*>(dstv + c * 8) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    cp_async_wait_all();
    __syncthreads();
    // scores of this warp's 8 keys for all 16 pairs
    {
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
      const __nv_bfloat16* ap = Qs + (lane & 15) * ks + (lane >> 4) * 8;
      const __nv_bfloat16* bp = Ks + (warp * 8 + (lane & 7)) * ks + ((lane >> 3) & 1) * 8;
#pragma unroll 4
      for (int k0 = 0; k0 < krow; k0 += 16) {
        uint32_t a[4], b[2];
        ldsm_x4(a, ap + k0);
        ldsm_x2(b, bp + k0);
        mma_bf16(s0, s1, s2, s3, a, b[0], b[1]);
      }
      const int row = lane >> 2, col = warp * 8 + (lane & 3) * 2;
      Ss[row * kSsStride + col] = s0;
      Ss[row * kSsStride + col + 1] = s1;
      Ss[(row + 8) * kSsStride + col] = s2;
      Ss[(row + 8) * kSsStride + col + 1] = s3;
    }
    __syncthreads();
    // softmax bookkeeping: this warp's 2 pairs, two keys per lane
#pragma unroll
    for (int rr = 0; rr < kLaPairs / kLaWarps; ++rr) {
      const int row = warp * (kLaPairs / kLaWarps) + rr, c = ctxp[row], lo = lop[row];
      const int j0 = base + lane, j1 = j0 + 32;
      const bool see0 = j0 < c && (j0 >= lo || (EX && j0 < keep)), see1 = j1 < c && (j1 >= lo || (EX && j1 < keep));
      float s0 = see0 ? Ss[row * kSsStride + lane] * scale : -INFINITY;
      float s1 = see1 ? Ss[row * kSsStride + lane + 32] * scale : -INFINITY;
      if constexpr (EX) {
        const float* brow = ex.dist_bias ? ex.dist_bias + (int64_t)(g * G + (i0 + row) % G) * ex.bias_dist : nullptr;
        const float inv_cap2 = ex.softcap > 0.f ? 2.0f / ex.softcap : 0.f;
        if (see0) s0 = score_shape_fast(s0, ex.softcap, inv_cap2, brow, c - 1 - j0, ex.bias_dist);
        if (see1) s1 = score_shape_fast(s1, ex.softcap, inv_cap2, brow, c - 1 - j1, ex.bias_dist);
      }
      const float m_old = mrow[row];
      const float m_new = fmaxf(m_old, warp_max(fmaxf(s0, s1)));
      float p0 = 0.f, p1 = 0.f, cr = 1.f;
      if (m_new != -INFINITY) {
        p0 = see0 ? expf(s0 - m_new) : 0.f;
        p1 = see1 ? expf(s1 - m_new) : 0.f;
        cr = expf(m_old - m_new);
      }
      const float sum = warp_sum(p0 + p1);
      Ps[row * kPsStride + lane] = __float2bfloat16_rn(p0);
      Ps[row * kPsStride + lane + 32] = __float2bfloat16_rn(p1);
      if constexpr (LO) {
        Pl[row * kPsStride + lane] = __float2bfloat16_rn(p0 - round_bf16(p0));
        Pl[row * kPsStride + lane + 32] = __float2bfloat16_rn(p1 - round_bf16(p1));
      }
      __syncwarp();
      if (lane == 0) {
        mrow[row] = m_new;
        lrow[row] = lrow[row] * cr + sum;
        corr[row] = cr;
      }
    }
    __syncthreads();
    // O = O * corr + P V over this warp's column groups
    {
      const float c_lo = corr[lane >> 2], c_hi = corr[(lane >> 2) + 8];
#pragma unroll
      for (int cg = 0; cg < NG; ++cg) {
        o[cg][0] *= c_lo; o[cg][1] *= c_lo; o[cg][4] *= c_lo; o[cg][5] *= c_lo;
        o[cg][2] *= c_hi; o[cg][3] *= c_hi; o[cg][6] *= c_hi; o[cg][7] *= c_hi;
      }
      const __nv_bfloat16* ap = Ps + (lane & 15) * kPsStride + (lane >> 4) * 8;
      const __nv_bfloat16* vp = Vs + ((lane & 7) + ((lane >> 3) & 1) * 8) * vs + (lane >> 4) * 8;
#pragma unroll
      for (int kk = 0; kk < kLaKeys / 16; ++kk) {
        uint32_t a[4], al[4];
        ldsm_x4(a, ap + kk * 16);
        if constexpr (LO) ldsm_x4(al, ap + (Pl - Ps) + kk * 16);
#pragma unroll
        for (int cg = 0; cg < NG; ++cg) {
          const int col0 = (warp + kLaWarps * cg) * 16;
          if (col0 < rank) {
            uint32_t b[4];
            ldsm_x4_t(b, vp + kk * 16 * vs + col0);
            mma_bf16(o[cg][0], o[cg][1], o[cg][2], o[cg][3], a, b[0], b[1]);
            mma_bf16(o[cg][4], o[cg][5], o[cg][6], o[cg][7], a, b[2], b[3]);
            if constexpr (LO) {
              mma_bf16(o[cg][0], o[cg][1], o[cg][2], o[cg][3], al, b[0], b[1]);
              mma_bf16(o[cg][4], o[cg][5], o[cg][6], o[cg][7], al, b[2], b[3]);
            }
          }
        }
      }
    }
    __syncthreads();
  }
  if (n_splits > 1) {
    // partial rows [pair][split][rank | m | l] fp32
    const int prow = rank + 2;
    if (tid < kLaPairs && i0 + tid < nq) {
      const int i = i0 + tid;
      float* dst = part + (((int64_t)(t0 + i / G) * heads + g * G + i % G) * n_splits + split) * prow;
      dst[rank] = mrow[tid];
      dst[rank + 1] = lrow[tid];
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int p = (lane >> 2) + half * 8, i = i0 + p;
      if (i >= nq) continue;
      float* dst = part + (((int64_t)(t0 + i / G) * heads + g * G + i % G) * n_splits + split) * prow;
#pragma unroll
      for (int cg = 0; cg < NG; ++cg) {
        const int col0 = (warp + kLaWarps * cg) * 16;
        if (col0 < rank) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const int col = col0 + nt * 8 + (lane & 3) * 2;
            dst[col] = o[cg][nt * 4 + half * 2];
            dst[col + 1] = o[cg][nt * 4 + half * 2 + 1];
          }
        }
      }
    }
    if constexpr (!MANY) return;
    __syncthreads();   // shared memory is the next chunk's
    continue;
  }
  // finish: sink, normalise, store
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int p = (lane >> 2) + half * 8, i = i0 + p;
    if (i >= nq) continue;
    const int t = t0 + i / G, h = g * G + i % G;
    float l = lrow[p], osc = 1.f;
    if (sink != nullptr) {
      const float m = mrow[p], sk = sink[h], mn = fmaxf(m, sk);
      osc = expf(m - mn);
      l = l * osc + expf(sk - mn);
    }
    float inv = l > 0.f ? osc / l : 0.f;
    if constexpr (EX)
      if (ex.gate) inv /= 1.0f + expf(-__bfloat162float(static_cast<const __nv_bfloat16*>(ex.gate)[t * ex.ldg + h]));
    __nv_bfloat16* dst = out + ((int64_t)t * heads + h) * rank;
#pragma unroll
    for (int cg = 0; cg < NG; ++cg) {
      const int col0 = (warp + kLaWarps * cg) * 16;
      if (col0 < rank) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const int col = col0 + nt * 8 + (lane & 3) * 2;
          *reinterpret_cast<__nv_bfloat162*>(dst + col) =
              __floats2bfloat162_rn(o[cg][nt * 4 + half * 2] * inv, o[cg][nt * 4 + half * 2 + 1] * inv);
        }
      }
    }
  }
  if constexpr (!MANY) return;
  __syncthreads();   // shared memory is the next chunk's
  }
  if constexpr (!MANY) return;
  __shared__ int next;
  if (threadIdx.x == 0) next = ticket;
  __syncthreads();
  v = next;
  __syncthreads();
  }
}

// One warp per (row, head): the splits' sums are brought to one maximum (the sink's included), added and normalised.
// Lane z holds split z's maximum and denominator; the per-split factors are then shared by shuffles and every lane's loads
// of a column are independent of one another.
constexpr int kLaMaxSplits = 16;
__global__ void __launch_bounds__(128)
latent_attn_merge_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ out, int n_pairs, int heads, int rank, int n_splits,
                         const float* __restrict__ sink, const __nv_bfloat16* __restrict__ gate, int64_t ldg, const LatentShare share) {
  pdl_wait();
  pdl_launch_dependents();
  if (share.plan && latent_by_rows(share)) return;   // there is nothing to merge
  const int pair = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (pair >= n_pairs) return;
  const int prow = rank + 2;
  const float* src = part + (int64_t)pair * n_splits * prow;
  const float mz = lane < n_splits ? src[lane * prow + rank] : -INFINITY;
  const float lz = lane < n_splits ? src[lane * prow + rank + 1] : 0.f;
  const float sk = sink ? sink[pair % heads] : -INFINITY;
  const float m = fmaxf(warp_max(mz), sk);
  const float ez = mz != -INFINITY ? expf(mz - m) : 0.f;
  const float l = warp_sum(lz * ez) + (sink ? expf(sk - m) : 0.f);
  float fz = l > 0.f ? ez / l : 0.f;
  if (gate) fz /= 1.0f + expf(-__bfloat162float(gate[(int64_t)(pair / heads) * ldg + pair % heads]));
  float f[kLaMaxSplits];
#pragma unroll
  for (int z = 0; z < kLaMaxSplits; ++z) f[z] = __shfl_sync(0xffffffffu, fz, z);
  for (int c = lane; c < rank; c += 32) {
    float v[kLaMaxSplits];
#pragma unroll
    for (int z = 0; z < kLaMaxSplits; ++z) v[z] = z < n_splits ? src[z * prow + c] : 0.f;
    float a = 0.f;
#pragma unroll
    for (int z = 0; z < kLaMaxSplits; ++z) a = fmaf(v[z], f[z], a);
    out[(int64_t)pair * rank + c] = __float2bfloat16_rn(a);
  }
}

}  // namespace

// Splits of the context for a step of T rows whose longest context is max_ctx: 1 when the (row, head) pairs fill the SMs
// anyway or the context is short; else enough CTAs for two per SM, at least two tiles each, within a workspace of ws_bytes.
int latent_attn_splits(int T, int heads, int rank, int max_ctx, int64_t ws_bytes) {
  const int ctas = (T * heads + kLaPairs - 1) / kLaPairs;
  // measured at 513 tokens: with 64 pair groups the merge launch costs what the split saves, with one it pays
  if (ctas >= kNumSMs || max_ctx <= (ctas < 16 ? 4 : 16) * kLaKeys) return 1;
  const int tiles = (max_ctx + kLaKeys - 1) / kLaKeys;
  int n = std::min(std::min((tiles + 1) / 2, (2 * kNumSMs + ctas - 1) / ctas), kLaMaxSplits);
  const int64_t per_split = (int64_t)T * heads * (rank + 2) * 4;
  while (n > 1 && n * per_split > ws_bytes) --n;
  return std::max(n, 1);
}

static size_t la_smem(int krow, int rank, bool own_values) {
  return (size_t)(kLaKeys + kLaPairs) * (krow + 8) * 2 + (own_values ? (size_t)kLaKeys * (rank + 8) * 2 : 0) +
         kLaPairs * (kSsStride * 4 + kPsStride * 2 + 20);
}

bool latent_attn_mma_supported(int heads, int krow, int rank) {
  static const int env = getenv("B200_LATENT_MMA") ? atoi(getenv("B200_LATENT_MMA")) : 1;
  return env && heads > 0 && krow % 16 == 0 && rank % 16 == 0 && rank > 0 && rank <= 512 && rank <= krow && la_smem(krow, rank, false) <= 200 * 1024;
}

// grouped-query attention with a value cache of its own on the same kernel: key rows of `dim`, value rows of `vdim` entries
bool paged_attn_mma_supported(int heads, int kv_heads, int dim, int vdim) {
  static const int env = getenv("B200_ATTN_MMA") ? atoi(getenv("B200_ATTN_MMA")) : 1;
  return env && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim % 16 == 0 && vdim % 16 == 0 && vdim > 0 && vdim <= 512 &&
         la_smem(dim, vdim, true) <= 200 * 1024;
}

static int attn_mma_launch(const float* q, const __nv_bfloat16* kc, const __nv_bfloat16* vc, int kv_heads, const int32_t* block_table,
                           int bt_stride, const int32_t* row_to_seq, const int32_t* ctx_lens, __nv_bfloat16* out, const int32_t* runs,
                           const int32_t* n_runs, int T, int heads, int krow, int rank, int block_size, float scale, const float* sink,
                           cudaStream_t s, int n_splits, float* part, int window, const AttnExtra& ex, const RunShare* share = nullptr, bool lo = false) {
  if (n_splits < 1 || part == nullptr) n_splits = 1;
  B200_REQUIRE(n_splits <= kLaMaxSplits, B200_ERR_INVALID, "attention: %d splits (at most %d)", n_splits, kLaMaxSplits);
  B200_REQUIRE(reinterpret_cast<uintptr_t>(kc) % 16 == 0 && reinterpret_cast<uintptr_t>(vc) % 16 == 0, B200_ERR_INVALID,
               "attention: cache not 16-byte aligned");
  const size_t smem = la_smem(krow, rank, vc != nullptr) + (lo ? kLaPairs * kPsStride * 2 : 0);
  // a run has at most 16 rows, so a kv head's group has at most 16 G pairs: G chunks of 16
  // (for a share of the runs: one wave of CTAs)
  const int64_t wave = (int64_t)kNumSMs * std::max(1, std::min(4, (int)(224 * 1024 / (smem + 1024))));
  const dim3 grid = share ? dim3((unsigned)std::min<int64_t>((int64_t)T * heads * n_splits, wave)) : dim3(T, heads, n_splits), block(kLaThreads);
#define LA2(NGV, EXV, MV, LOV)                                                                                                             \
  do {                                                                                                                              \
    static bool done[64] = {};                                                                                                      \
    if (smem > 48 * 1024) B200_CUDA(ensure_dynamic_smem(latent_attn_mma_kernel<NGV, EXV, MV, LOV>, 200 * 1024, done));                       \
    B200_CUDA(launch(latent_attn_mma_kernel<NGV, EXV, MV, LOV>, grid, block, smem, s, q, kc, vc, kv_heads, block_table, bt_stride, row_to_seq, \
                     ctx_lens, out, runs, n_runs, heads, krow, rank, block_size, scale, sink, n_splits, part, window, ex, share ? *share : RunShare())); \
  } while (0)
#define LA(NGV, MV, LOV)                     \
  do {                                       \
    if (ex.any()) LA2(NGV, true, MV, LOV);   \
    else LA2(NGV, false, MV, LOV);           \
  } while (0)
  if (share) LA(1, true, false);   // (rank <= 128: attn_rows_tc.cu's shapes)
  else if (lo) LA(1, false, true);
  else if (rank <= 128) LA(1, false, false);
  else if (rank <= 256) LA(2, false, false);
  else LA(4, false, false);
#undef LA
#undef LA2
  if (n_splits > 1)
    B200_CUDA(launch(latent_attn_merge_kernel, dim3((T * heads + 3) / 4), dim3(128), (size_t)0, s, (const float*)part, out, T * heads, heads,
                     rank, n_splits, sink, static_cast<const __nv_bfloat16*>(ex.gate), ex.ldg, LatentShare()));
  return B200_OK;
}

static LatentShare latent_share(const int32_t* plan, int T, int heads, int krow, int rank, int n_splits, int window) {
  LatentShare s = {};
  s.plan = plan;
  s.rows = T;
  s.splits = n_splits;
  s.halves = latent_attn_tc_halves(rank);
  s.rows_per_item = latent_attn_tc_rows(heads);
  s.seen = window > 0 ? window : INT_MAX;
  const int groups = latent_attn_rows_items(1, heads);
  const float by_row = 4.2f + 0.035f * krow, by_run = 1.15f * std::max(16.5f, 0.043f * krow);
  s.row_key = by_row / latent_attn_rows_cluster(T * groups);
  s.row_tile = by_row * 64 * groups / kNumSMs;
  s.run_fixed = 10000.f + 54.f * krow;
  s.run_key = by_run / n_splits;
  s.run_item = by_run * 64 / n_splits;
  return s;
}

// Rows by themselves (attn_latent_rows.cu) wherever they fit, but
//  * more items of 16 heads than SMs: only rows that are known to be sequences of their own (a prefill chunk's runs share their keys), and up to 32 heads (one of
//    128 fills the other kernel's MMAs: 512 rows at 2 000 tokens 1 543 us here, 931 there; of 32 heads 404 and 432, of 16 256 and 433);
//  * contexts that may be so long that the caller's splits would pay for a chunk or a long row among short ones (runs.cuh): the device decides.  Up to seven items have
//    splits of their own.  Without splits neither is much slower than the other anywhere (100 rows of one sequence of 3 100 tokens 86 and 93).
// One or two rows with less than 4 KB of queries (T * heads * krow) keep the plan and the attention as two launches, the second overlapping the first, which is
// what a captured call of two rows of 4 heads over 64 + 16 holds (tests/test_launch_gpu.py): 13.5 us, by themselves 10.  (Rows of more queries: 64 of these heads
// at 900 tokens 28 us over runs, 13 by themselves.)
LatentRoute latent_attn_route(const float* q, const __nv_bfloat16* kc, const int32_t* row_to_seq, const __nv_bfloat16* out, const int32_t* runs, int T, int heads,
                              int krow, int rank, int block_size, float scale, int n_splits, const float* part, int64_t longest, bool one_row_each) {
  const auto at = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr); };
  if (T <= 0 || !(scale > 0.f) || !latent_attn_mma_supported(heads, krow, rank) || !latent_attn_rows_supported(heads, krow, rank, block_size) ||
      (T <= 2 && (int64_t)T * heads * krow < 1024) || (at(q) | at(kc) | at(out)) % 16 != 0)
    return LatentRoute::kRuns;
  const bool own = one_row_each || !row_to_seq, tc = latent_attn_tc_supported(heads, krow, rank, block_size) && at(out) % 32 == 0 && ((at(runs) | at(part)) & 7) == 0;
  const int items = latent_attn_rows_items(T, heads);
  if (items > kNumSMs && (!own || (heads > 32 && tc))) return LatentRoute::kRuns;
  if (n_splits <= 1 || !part || !tc || (items <= 7 && longest > 32768)) return LatentRoute::kRows;
  // the longest row alone: what its CTAs take, and what they would take over runs in splits, with the launches that tell
  const LatentShare s = latent_share(nullptr, T, heads, krow, rank, n_splits, 0);
  const float gain = (s.row_key - s.run_key / 1.15f) * (float)longest;
  return gain > s.run_fixed + 12000.f ? LatentRoute::kEither : LatentRoute::kRows;
}

// runs / n_runs: the run list of the step (attn_anydim.cu builds it: runs of at most 16 consecutive rows of one sequence)
int latent_attn_mma(const float* q, const __nv_bfloat16* kc, const int32_t* block_table, int bt_stride, const int32_t* row_to_seq,
                    const int32_t* ctx_lens, __nv_bfloat16* out, const int32_t* runs, const int32_t* n_runs, int T, int heads, int krow,
                    int rank, int block_size, float scale, const float* sink, cudaStream_t s, int n_splits, float* part, int window,
                    bool one_row_each, int64_t longest) {
  if (T == 0) return B200_OK;
  B200_REQUIRE(latent_attn_mma_supported(heads, krow, rank), B200_ERR_UNSUPPORTED, "latent_attn_mma: shape %d / %d / %d", heads, krow, rank);
  if (n_splits < 1 || part == nullptr) n_splits = 1;
  B200_REQUIRE(n_splits <= kLaMaxSplits, B200_ERR_INVALID, "attention: %d splits (at most %d)", n_splits, kLaMaxSplits);
  const auto at = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr); };
  B200_REQUIRE(at(kc) % 16 == 0, B200_ERR_INVALID, "attention: cache not 16-byte aligned");
  const auto merge = [&](int splits, const LatentShare& share) -> int {
    B200_CUDA(launch(latent_attn_merge_kernel, dim3((T * heads + 3) / 4), dim3(128), (size_t)0, s, (const float*)part, out, T * heads, heads, rank, splits,
                     sink, (const __nv_bfloat16*)nullptr, (int64_t)0, share));
    return B200_OK;
  };
  const LatentRoute route = latent_attn_route(q, kc, row_to_seq, out, runs, T, heads, krow, rank, block_size, scale, n_splits, part, longest, one_row_each);
  const LatentShare share = route == LatentRoute::kEither ? latent_share(n_runs, T, heads, krow, rank, n_splits, window) : LatentShare();
  if (route != LatentRoute::kRuns) {
    int splits = n_splits;
    const int rc = latent_attn_rows(q, kc, block_table, bt_stride, row_to_seq, ctx_lens, out, T, heads, krow, rank, block_size, scale, sink, s, window,
                                    at(part) % 8 == 0 ? part : nullptr, longest, share, &splits);
    if (rc || (route == LatentRoute::kRows && splits == 1)) return rc;
    const PdlScope after_rows;
    if (route == LatentRoute::kRows) return merge(splits, share);
    if (const int e = latent_attn_tc(q, kc, block_table, bt_stride, row_to_seq, ctx_lens, out, runs, n_runs, T, heads, krow, rank, block_size, scale, sink, s, n_splits,
                                     part, window, share))
      return e;
    return merge(n_splits, share);
  }
  // tcgen05 wherever the shape fits and the rows can be read and written in its wide pieces (what it measured stands there); other shapes, blocks
  // that a key tile would straddle and odd addresses stay here, and so do scales that are not positive (masks and maxima there are taken of
  // the unscaled scores) and steps whose rows are known to be sequences of their own (or have one head: 16 pairs a run at most) where
  // they would make more than three rounds of items there: 256 decode rows of 16 heads 102 us there, 88 here, 64 of one head in 5 splits 74 and 45
  const bool few_pairs = (one_row_each || !row_to_seq || heads == 1) && heads <= 16 && (int64_t)T * latent_attn_tc_halves(rank) * n_splits > 3 * kNumSMs;
  if (scale > 0.f && !few_pairs && latent_attn_tc_supported(heads, krow, rank, block_size) && at(q) % 16 == 0 && at(out) % 32 == 0 &&
      ((at(runs) | at(part)) & 7) == 0) {
    const int rc = latent_attn_tc(q, kc, block_table, bt_stride, row_to_seq, ctx_lens, out, runs, n_runs, T, heads, krow, rank, block_size, scale,
                                  sink, s, n_splits, part, window, share);
    return rc || n_splits == 1 ? rc : merge(n_splits, share);
  }
  return attn_mma_launch(q, kc, nullptr, 1, block_table, bt_stride, row_to_seq, ctx_lens, out, runs, n_runs, T, heads, krow, rank, block_size,
                         scale, sink, s, n_splits, part, window, AttnExtra());
}

// caches [block][kv_heads][block_size][dim | vdim] bf16, fp32 queries [T][heads][dim], bf16 output [T][heads][vdim]
int paged_attn_mma(const float* q, const __nv_bfloat16* kc, const __nv_bfloat16* vc, const int32_t* block_table, int bt_stride,
                   const int32_t* row_to_seq, const int32_t* ctx_lens, __nv_bfloat16* out, const int32_t* runs, const int32_t* n_runs, int T,
                   int heads, int kv_heads, int dim, int vdim, int block_size, float scale, const float* sink, cudaStream_t s, int n_splits,
                   float* part, int window, const AttnExtra& ex, bool one_row_each) {
  if (T == 0) return B200_OK;
  B200_REQUIRE(vc && paged_attn_mma_supported(heads, kv_heads, dim, vdim), B200_ERR_UNSUPPORTED, "paged_attn_mma: shape %d / %d / %d / %d", heads,
               kv_heads, dim, vdim);
  if (n_splits < 1 || part == nullptr) n_splits = 1;
  B200_REQUIRE(n_splits <= kLaMaxSplits, B200_ERR_INVALID, "attention: %d splits (at most %d)", n_splits, kLaMaxSplits);
  const auto at = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr); };
  B200_REQUIRE(at(kc) % 16 == 0 && at(vc) % 16 == 0, B200_ERR_INVALID, "attention: cache not 16-byte aligned");
  // tcgen05 for longer runs of rows (1 900 rows of three sequences 74 us against 278); wider heads, smaller blocks and odd addresses stay here,
  // and so do scales that are not positive (masks and maxima of the other kernel are those of the unscaled scores) and decode rows, which fill
  // G of an item's 256 pairs there (256 rows at contexts 300..600, 16 heads over 4: 184 us against 80).  Short steps stay here
  // altogether; others launch both kernels, which share the step's runs (runs.cuh), unless every row is known to be a sequence of its own
  const bool runs_of_rows = T > 128 && row_to_seq && !one_row_each && scale > 0.f && at(q) % 16 == 0 && at(out) % 16 == 0 && at(part) % 8 == 0;
  if (runs_of_rows && attn_rows_tc_supported(heads, kv_heads, dim, vdim, block_size)) {
    RunShare share;
    const int rc = attn_rows_tc_runs(q, kc, vc, block_table, bt_stride, row_to_seq, ctx_lens, out, runs, n_runs, T, heads, kv_heads, dim, vdim,
                                     block_size, scale, sink, s, n_splits, part, window, ex, &share);
    if (rc) return rc;
    const PdlScope after_rows;
    return attn_mma_launch(q, kc, vc, kv_heads, block_table, bt_stride, row_to_seq, ctx_lens, out, runs, n_runs, T, heads, dim, vdim, block_size,
                           scale, sink, s, n_splits, part, window, ex, &share);
  }
  return attn_mma_launch(q, kc, vc, kv_heads, block_table, bt_stride, row_to_seq, ctx_lens, out, runs, n_runs, T, heads, dim, vdim, block_size,
                         scale, sink, s, n_splits, part, window, ex, nullptr, runs_of_rows && attn_rows_tc_declined(heads, kv_heads, dim, vdim, block_size));
}

}  // namespace b200

// debug helpers (not in the public header): which kernel a call of these forms takes, with everything aligned (0 rows by themselves, 1 the device decides, 2 over
// runs), and what the device decides of a step whose plan has so many runs, that longest context and so many tiles (1 rows by themselves)
extern "C" __attribute__((visibility("default"))) int b200_debug_latent_route(int32_t T, int32_t heads, int32_t krow, int32_t rank, int32_t block_size,
                                                                              int32_t n_splits, int64_t longest, int32_t own) {
  using namespace b200;
  const auto p = [](uintptr_t a) { return reinterpret_cast<void*>(a); };
  return (int)latent_attn_route(static_cast<const float*>(p(64)), static_cast<const __nv_bfloat16*>(p(64)), static_cast<const int32_t*>(p(64)),
                                static_cast<const __nv_bfloat16*>(p(64)), static_cast<const int32_t*>(p(64)), T, heads, krow, rank, block_size, 1.f, n_splits,
                                n_splits > 1 ? static_cast<const float*>(p(64)) : nullptr, longest, own != 0);
}
extern "C" __attribute__((visibility("default"))) int b200_debug_latent_by_rows(int32_t T, int32_t heads, int32_t krow, int32_t rank, int32_t n_splits, int32_t window,
                                                                                int32_t n_runs, int32_t longest, int32_t tiles) {
  using namespace b200;
  return latent_by_rows(latent_share(nullptr, T, heads, krow, rank, n_splits, window), n_runs, longest, tiles) ? 1 : 0;
}
