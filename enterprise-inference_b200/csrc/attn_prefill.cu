// (a6, prefill rows) Causal paged attention for the rows of prefill chunks: the step's row plan and its entry points.
//
// attn_tc.cu puts the 128 cached tokens of a tile on the UMMA M dimension and at most 16 query heads on N: right for decode (every
// cached byte is used once per step), but a 2048-row chunk then streams the sequence's K/V once per four rows and pays about 100
// softmax instructions per (tile, column).  Rows of a chunk go to attn_rows_tc.cu instead, whose MMA rows are (row, head) pairs of one
// kv head; weights reach the second product as hi + lo bf16 (the CPU oracle keeps them in fp32).
//
// Rows come in any mix (chunked prefill + decode rows in one step): a plan kernel of one CTA cuts the step's rows into items (maximal
// runs of one sequence, at most as many rows as fill two tiles of 128 pairs); a decode row becomes an item with one live row.
//
// Replaces: the prefill half of the vLLM-CPU attention backend ([V22] vllm/v1/attention/backends/
// cpu_attn.py:377-396); chunked prefill is selected by the chart (xeon-values.yaml:80-83).
#include "common.cuh"

namespace b200 {

namespace {

constexpr int kTileTok = 128;

struct PlanItem {
  int row0, nrows, seq, ctx_max;
};

// ---- plan: rows -> items (one CTA: 1024 rows at a time, then a warp per item) -------------------------
// plan[0] = {n_items, 0, 0, 0}; plan[1 + i] = item i: rows [row0, row0 + nrows) of sequence seq, all of
// one sequence, nrows <= rb, ctx_max = their longest context.
__global__ void __launch_bounds__(1024) attn_prefill_plan_kernel(const int32_t* __restrict__ row_to_seq,
                                                                  const int32_t* __restrict__ ctx_lens, int n_rows, int rb,
                                                                  PlanItem* __restrict__ plan) {
  __shared__ int wseg[32], wcnt[32], carry_seg, carry_cnt;
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) carry_seg = carry_cnt = 0;
  __syncthreads();
  for (int c0 = 0; c0 < n_rows; c0 += 1024) {
    const int r = c0 + tid;
    const bool valid = r < n_rows;
    const int seq = valid ? (row_to_seq ? row_to_seq[r] : r) : -1;
    const int prev = (valid && r > 0) ? (row_to_seq ? row_to_seq[r - 1] : r - 1) : -2;
    // start row of the segment (run of one sequence) that row r belongs to: inclusive max-scan
    int seg = (valid && (r == 0 || seq != prev)) ? r : -1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, seg, o);
      if (lane >= o) seg = max(seg, v);
    }
    if (lane == 31) wseg[warp] = seg;
    __syncthreads();
    int before = carry_seg;
    for (int w = 0; w < warp; ++w) before = max(before, wseg[w]);
    seg = max(seg, before);
    const bool start = valid && ((r - seg) % rb == 0);
    const unsigned m = __ballot_sync(0xffffffffu, start);
    if (lane == 0) wcnt[warp] = __popc(m);
    __syncthreads();
    int idx = carry_cnt + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) idx += wcnt[w];
    if (start) {
      plan[1 + idx].row0 = r;
      plan[1 + idx].seq = seq;
    }
    __syncthreads();
    if (tid == 1023) {
      carry_seg = seg;
      carry_cnt = idx + (start ? 1 : 0);
    }
    __syncthreads();
  }
  const int n_items = carry_cnt;
  if (tid == 0) plan[0].row0 = n_items;
  for (int i = warp; i < n_items; i += 32) {
    const int row0 = plan[1 + i].row0;
    const int next = (i + 1 < n_items) ? plan[2 + i].row0 : n_rows;
    int cmax = 0;
    for (int r = row0 + lane; r < next; r += 32) cmax = max(cmax, ctx_lens[r]);
    cmax = __reduce_max_sync(0xffffffffu, cmax);
    if (lane == 0) {
      plan[1 + i].nrows = next - row0;
      plan[1 + i].ctx_max = cmax;
    }
  }
}

}  // namespace

int64_t paged_attn_prefill_plan_bytes(int T) { return (int64_t)(T + 1) * (int64_t)sizeof(PlanItem); }

bool paged_attn_prefill_fa_supported(int hq, int hkv, int block_size) {
  if (hkv <= 0 || hq % hkv != 0 || block_size != kTileTok) return false;
  const int G = hq / hkv;
  return G == 1 || G == 2 || G == 4 || G == 5 || G == 8;
}

// Same contract as paged_attn (attn.cu); `ws` holds the plan (paged_attn_prefill_plan_bytes(T)).
// The plan depends on the step's rows only, not on the layer: a caller that runs many layers over the same
// rows builds it once (this function) and passes plan_ready = true to paged_attn_prefill_fa.
int paged_attn_prefill_plan(const int32_t* row_to_seq, const int32_t* ctx_lens, int T, int hq, int hkv, void* ws,
                            int64_t ws_bytes, cudaStream_t s) {
  B200_REQUIRE(hkv > 0 && hq % hkv == 0, B200_ERR_INVALID, "attn_prefill: hq=%d not a multiple of hkv=%d", hq, hkv);
  if (T == 0) return B200_OK;
  B200_REQUIRE(ws && ws_bytes >= paged_attn_prefill_plan_bytes(T), B200_ERR_INVALID,
               "attn_prefill: workspace too small (%lld < %lld)", (long long)ws_bytes,
               (long long)paged_attn_prefill_plan_bytes(T));
  B200_CUDA(launch(attn_prefill_plan_kernel, dim3(1), dim3(1024), (size_t)0, s, row_to_seq, ctx_lens, T, attn_rows_tc_rows(T, hq, hkv),
                   static_cast<PlanItem*>(ws)));
  return B200_OK;
}

int paged_attn_prefill_fa(const __nv_bfloat16* q, int64_t ldq, const __nv_bfloat16* kc, const __nv_bfloat16* vc,
                          const int32_t* block_table, int bt_stride, const int32_t* row_to_seq, const int32_t* ctx_lens,
                          __nv_bfloat16* out, int64_t ldo, int T, int hq, int hkv, int block_size, float scale, void* ws,
                          int64_t ws_bytes, bool plan_ready, cudaStream_t s) {
  B200_REQUIRE(paged_attn_prefill_fa_supported(hq, hkv, block_size), B200_ERR_UNSUPPORTED, "attn_prefill: unsupported shape");
  B200_REQUIRE(ldq % 8 == 0 && ldo % 8 == 0, B200_ERR_INVALID, "attn_prefill: ldq/ldo must be multiples of 8");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0, B200_ERR_INVALID,
               "attn_prefill: q and out must be 16-byte aligned");
  B200_REQUIRE(scale > 0.f, B200_ERR_INVALID, "attn_prefill: scale must be positive");
  if (T == 0) return B200_OK;
  B200_REQUIRE(ws && ws_bytes >= paged_attn_prefill_plan_bytes(T), B200_ERR_INVALID,
               "attn_prefill: workspace too small (%lld < %lld)", (long long)ws_bytes,
               (long long)paged_attn_prefill_plan_bytes(T));
  if (!plan_ready) {
    const int rc0 = paged_attn_prefill_plan(row_to_seq, ctx_lens, T, hq, hkv, ws, ws_bytes, s);
    if (rc0) return rc0;
    const PdlScope after_plan;
    return attn_rows_tc_plan(q, ldq, kc, vc, block_table, bt_stride, ctx_lens, out, ldo, T, hq, hkv, kHeadDim, block_size, scale, ws, s);
  }
  return attn_rows_tc_plan(q, ldq, kc, vc, block_table, bt_stride, ctx_lens, out, ldo, T, hq, hkv, kHeadDim, block_size, scale, ws, s);
}

}  // namespace b200
