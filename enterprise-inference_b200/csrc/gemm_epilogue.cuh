// What the tcgen05 linears (gemm_tc.cu, gemm_pair.cu) share: a launch's parameters and the epilogue's last step, in which one thread turns
// four neighbouring output features of a token into what the launch writes.
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int kBlockM = 128;   // weight rows per CTA = UMMA M
constexpr int kBlockK = 64;    // bf16 elements per stage row = 128 bytes = one swizzle span

struct TcParams {
  const __nv_bfloat16* bias;
  __nv_bfloat16* y;
  int64_t ldy;
  int T, n_out, n_kblocks, splits;
  float* partials;      // [splits][tok_tiles*N][n_out_pad] fp32
  unsigned int* tickets;  // [m_tiles * tok_tiles], zero on entry, zero on exit
  int n_out_pad;
  int cluster;  // 1: the `splits` CTAs of a slab form a thread-block cluster and reduce through DSMEM
  // MODE_ROPE_KV (slab == one 128-wide head of the fused qkv projection)
  const int32_t* positions;
  const int32_t* slots;
  const __nv_bfloat16* cos_sin;
  __nv_bfloat16* kc;
  __nv_bfloat16* vc;
  int hq, hkv, block_size;
  unsigned long long* trace;  // debug (B200_TC_TRACE=1): %globaltimer stamps of CTA 0, else null
  // Residual stream in fp32 (RMSNorm folded into the linears, T <= 64):
  //   producer (MODE kResidual, O / down projection): s = bf16(acc) + bf16(sres) in fp32 -> sres, and the sum of
  //     squares of the slab's 128 values of s -> ssq[tok][m_tile]              (n_out = hidden)
  //   consumer (NI, QKV / gate_up / lm_head): the B operand is bf16(bf16(s * rinv) * norm_w) built in shared memory
  //     from sres, rinv = 1/sqrt(sum_slabs ssq / hidden + eps)                  (k = hidden)
  float* sres;
  float* ssq;
  const __nv_bfloat16* norm_w;
  const int32_t* rows;   // consumer: token t of the launch reads stream row rows[t] (lm_head's logit rows), or null
  int nslab;             // hidden / 128
  float eps;
  // Grouped form (routed experts): w holds [experts][n_out][k]; token tile j multiplies the rows of expert grp_tile[j]
  // (-1: the tile is not in use and its CTAs leave at once).  The token rows are the experts' tokens, gathered so that
  // no tile holds rows of two experts.
  const int32_t* grp_tile;
  // grouped gate|up with the SiLU*mul epilogue: an expert's rows are [gate (gu_ff) | up (gu_ff)]; slab m of the launch is
  // gate rows m*64.. and the matching up rows, fetched as two 64-row boxes (the layout kSiluMul expects, made by TMA)
  int gu_ff;
  int act;   // kSiluMul: b200_act_kind of the gate (0: silu, rounded to bf16 before the product as the fixed stack does)
  float act_limit;   // B200_ACT_SWIGLU_CLAMP: the clamp of gate and up value
  // kScatter: row t of the launch goes to grp_out[grp_pair[t]][n_out] (fp32, unrounded) times grp_wt[grp_pair[t]];
  // grp_pair[t] < 0 marks a padding row
  // (both null: the identity and weight 1, i.e. a plain fp32 output)
  const int32_t* grp_pair;
  const float* grp_wt;
  float* grp_out;
  int post_act;          // kPlain: 1 + b200_act_kind applied to the fp32 sum before the rounding (0: none)
  int tile_n;            // N of the instantiation (kScatter: index of a token inside its tile)
  // pairs of CTAs (gemm_pair.cu): tiles of 256 weight rows and up to 256 tokens
  const int4* pair_tile; // grouped form: pair_tile[0].x token tiles follow, each (expert, first row, rows, -); null: pair_tok tiles of pair_n tokens
  int pair_n, pair_tok, pair_m, pair_group;   // pair_m: 256-row tiles of W; pair_group: token tiles that share a pass over W
};

// Epilogue modes (template parameter):
//  kPlain    y[t][row] = bf16(acc + bias), or bf16(act(acc + bias)) (TcParams::post_act)
//  kSiluMul  the slab holds 64 gate rows then the 64 matching up rows (B200_W_GATE_UP_INTERLEAVED):
//            y[t][m_tile*64 + i] = bf16(bf16(silu(bf16(g_i))) * bf16(u_i))          (R5)
//            (TcParams::act != 0: bf16(act(bf16(g_i)) * bf16(u_i)) for the other gate activations)
//  kRopeKv   the slab is one head of the fused qkv projection: NeoX RoPE in bf16 arithmetic (R3) on q
//            and k heads, q rows to y, k/v rows straight into the paged cache at slots[t]
//  kResidual the linear's output is added to the fp32 residual stream (see TcParams::sres): no y is written
//  kScatter  (grouped form) the fp32 row times a per-row weight goes to the row the indirection names; no y
enum { kPlain = 0, kSiluMul = 1, kRopeKv = 2, kResidual = 3, kScatter = 4 };


// One thread finalises 4 consecutive slab rows (r4..r4+3, lane = r4/4) of one token.  kScatter: `pair` and `wt` are the row's destination and weight.
template <int MODE>
__device__ __forceinline__ void finalize4(const TcParams& p, int m_tile, int lane, int tok, float4 a, const float (&bb)[4], int pair = -1, float wt = 1.0f) {
  const int r4 = lane * 4;
  float v[4] = {round_bf16(a.x + bb[0]), round_bf16(a.y + bb[1]), round_bf16(a.z + bb[2]), round_bf16(a.w + bb[3])};
  if constexpr (MODE == kPlain) {
    if (p.post_act == 1 + B200_ACT_RELU2) {
      const float r[4] = {fmaxf(a.x + bb[0], 0.f), fmaxf(a.y + bb[1], 0.f), fmaxf(a.z + bb[2], 0.f), fmaxf(a.w + bb[3], 0.f)};
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = r[e] * r[e];
    } else if (p.post_act == 1 + B200_ACT_GELU_ERF) {
      v[0] = gelu_erf_fast(a.x + bb[0]), v[1] = gelu_erf_fast(a.y + bb[1]);
      v[2] = gelu_erf_fast(a.z + bb[2]), v[3] = gelu_erf_fast(a.w + bb[3]);
    } else if (p.post_act) {
      v[0] = act_apply(a.x + bb[0], p.post_act - 1), v[1] = act_apply(a.y + bb[1], p.post_act - 1);
      v[2] = act_apply(a.z + bb[2], p.post_act - 1), v[3] = act_apply(a.w + bb[3], p.post_act - 1);
    }
    const int row = m_tile * kBlockM + r4;
    __nv_bfloat16* dst = p.y + (int64_t)tok * p.ldy + row;
    if (row + 3 < p.n_out && (p.ldy % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.y) & 7) == 0)) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (row + e < p.n_out) dst[e] = __float2bfloat16_rn(v[e]);
    }
  } else if constexpr (MODE == kSiluMul) {
    // lanes 0..15 hold 4 gate rows, lanes 16..31 the 4 matching up rows: after the exchange every lane has
    // both, and each half-warp finalises two of the four features (all 32 lanes busy: the accurate
    // expf + division of R5 is what this epilogue costs at large T)
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = __shfl_xor_sync(0xffffffffu, v[e], 16);
    const bool lo = lane < 16;
    const float g0 = lo ? v[0] : x[2], g1 = lo ? v[1] : x[3];
    const float u0 = lo ? x[0] : v[2], u1 = lo ? x[1] : v[3];
    const int f = m_tile * 64 + (lane & 15) * 4 + (lo ? 0 : 2);                  // output feature
    const float o0 = p.act == 0 ? silu_to_bf16(g0) * u0 : gate_combine(g0, u0, p.act, p.act_limit);
    const float o1 = p.act == 0 ? silu_to_bf16(g1) * u1 : gate_combine(g1, u1, p.act, p.act_limit);
    __nv_bfloat16* dst = p.y + (int64_t)tok * p.ldy + f;
    if ((p.ldy % 2 == 0) && ((reinterpret_cast<uintptr_t>(p.y) & 3) == 0)) {
      *reinterpret_cast<uint32_t*>(dst) = pack_bf16(o0, o1);
    } else {
      dst[0] = __float2bfloat16_rn(o0);
      dst[1] = __float2bfloat16_rn(o1);
    }
  } else if constexpr (MODE == kResidual) {
    // x = bf16(acc + bias); s = x + bf16(s_old) in fp32 (R1: the residual is kept in bf16, the sum is not rounded
    // before the variance and the normalisation); sum of squares in a fixed order: lane's 4 rows, then the warp tree
    const int row = m_tile * kBlockM + r4;
    float4* sp = reinterpret_cast<float4*>(p.sres + (int64_t)tok * p.n_out + row);
    const float4 so = *sp;
    const float4 sn = make_float4(v[0] + round_bf16(so.x), v[1] + round_bf16(so.y), v[2] + round_bf16(so.z),
                                  v[3] + round_bf16(so.w));
    *sp = sn;
    float ss = fmaf(sn.x, sn.x, 0.f);
    ss = fmaf(sn.y, sn.y, ss);
    ss = fmaf(sn.z, sn.z, ss);
    ss = fmaf(sn.w, sn.w, ss);
    ss = warp_sum(ss);
    if (lane == 0) p.ssq[(int64_t)tok * p.nslab + m_tile] = ss;
  } else if constexpr (MODE == kScatter) {
    if (pair < 0) return;   // warp-uniform
    const int row = m_tile * kBlockM + r4;
    float* dst = p.grp_out + (int64_t)pair * p.n_out + row;
    if (row + 3 < p.n_out && (p.n_out % 4 == 0)) {
      *reinterpret_cast<float4*>(dst) = make_float4(a.x * wt, a.y * wt, a.z * wt, a.w * wt);
    } else {
      const float o[4] = {a.x * wt, a.y * wt, a.z * wt, a.w * wt};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (row + e < p.n_out) dst[e] = o[e];
    }
  } else {  // kRopeKv
    const int head = m_tile;
    float o[4];
    if (head < p.hq + p.hkv) {
      float other[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) other[e] = __shfl_xor_sync(0xffffffffu, v[e], 16);
      const int i0 = r4 & 63;
      const __nv_bfloat16* cs = p.cos_sin + (int64_t)p.positions[tok] * kHeadDim;
      const uint2 cq = *reinterpret_cast<const uint2*>(cs + i0);
      const uint2 sq = *reinterpret_cast<const uint2*>(cs + 64 + i0);
      const float c[4] = {bf16lo(cq.x), bf16hi(cq.x), bf16lo(cq.y), bf16hi(cq.y)};
      const float sn[4] = {bf16lo(sq.x), bf16hi(sq.x), bf16lo(sq.y), bf16hi(sq.y)};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // lanes 0..15 hold x1 (o1 = x1*c - x2*s), lanes 16..31 hold x2 (o2 = x2*c + x1*s); every op rounds
        const float a0 = round_bf16(v[e] * c[e]), b0 = round_bf16(other[e] * sn[e]);
        o[e] = lane < 16 ? round_bf16(a0 - b0) : round_bf16(a0 + b0);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = v[e];
    }
    __nv_bfloat16* dst;
    if (head < p.hq) {
      dst = p.y + (int64_t)tok * p.ldy + head * kHeadDim + r4;
    } else {
      const int slot = p.slots[tok];
      if (slot < 0) return;
      const bool is_k = head < p.hq + p.hkv;
      const int kvh = is_k ? head - p.hq : head - p.hq - p.hkv;
      const int64_t blk = slot / p.block_size, off = slot % p.block_size;
      dst = (is_k ? p.kc : p.vc) + ((blk * p.hkv + kvh) * p.block_size + off) * kHeadDim + r4;
    }
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
  }
}

// pairs of SMs (gemm_pair.cu)
struct PairPlan {
  int n, splits;   // tokens a tile; CTA pairs that share a tile's k
};
PairPlan linear_pair_plan(int T, int n_out, int k);
int linear_pair(int mode, TcParams p, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int k, PairPlan pl, cudaStream_t s);
// The same over the gathered rows of every expert: w [experts][n_out][k], an expert's rows a run of x, cut into token tiles by a table on the device
// (TcParams::pair_tile).  y[row] = act(x . w_e^T) (post_act: 1 + b200_act_kind, 0 none); gate_up: w [experts][2 ff][k], gate rows then up rows, y[row][ff]
// the activated product; scatter: out[row_pair[row]] = wts[row_pair[row]] * (x . w_e^T) in fp32 (row_pair < 0: a padding row).
struct GroupedPairs {
  const int4* tiles;
  int max_tiles;    // of the table
  int64_t rows;     // of x, at most
  int experts;
};
int linear_pair_grouped(const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int n_out, int k, __nv_bfloat16* y, int64_t ldy,
                        cudaStream_t s, int post_act = 0);
int linear_pair_gate_up(const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int ff, int k, __nv_bfloat16* y, cudaStream_t s,
                        int act, float act_limit);
int linear_pair_scatter(const GroupedPairs& g, const __nv_bfloat16* x, int64_t ldx, const __nv_bfloat16* w, int n_out, int k, const int32_t* row_pair,
                        const float* wts, float* out, cudaStream_t s);

}  // namespace b200
