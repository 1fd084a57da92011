// Launches of the matrix-memory recurrence in chunks (mlstm_chunk.cuh), for steps that do not go in segments (mlstm_segment.cu).
#include <algorithm>

#include "mlstm_chunk.cuh"

namespace b200 {

namespace {

// Chunks on their own; short portions are the pair's first CTA's, with both halves' columns, or the walk's kernel's.
// CTAS: that share an SM, one where all have an SM of their own (the registers of two cost one portion of 300 rows, 9 heads of 256 columns, 25.2 -> 29.4 us).
template <int KS, int CTAS>
__global__ void __launch_bounds__(kMcThreads, CTAS) mlstm_chunk_kernel(const MlstmArgs a) {
  extern __shared__ __align__(16) unsigned char raw[];
  pdl_wait();
  pdl_launch_dependents();
  const int n_rows = a.seq_start[blockIdx.x + 1] - a.seq_start[blockIdx.x];
  if (n_rows >= kChunkFrom) mlstm_chunks<KS, 0>(a, raw, blockIdx.z);
  else if ((blockIdx.z & 1) == 0 && !a.both) mlstm_walk<__nv_bfloat16, KS / 4>(a, reinterpret_cast<float*>(raw), blockIdx.z >> 1, gridDim.z >> 1);
}

}  // namespace

// rows of q, k and v in 16-byte pieces, key dimensions within eight 16-wide steps
bool mlstm_chunk_supported(const MlstmArgs& a) {
  return a.dim > 0 && a.dim <= 128 && a.dim % 8 == 0 && a.vd % 8 == 0 && a.ld % 8 == 0 && (a.q_off | a.k_off | a.v_off) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a.qkv) % 16 == 0;
}
// A launch's CTAs
int64_t mlstm_chunk_ctas(const MlstmArgs& a, int S) { return (int64_t)S * a.heads * 2 * mlstm_col_blocks(a.vd); }

int mlstm_chunk(const MlstmArgs& a, int S, cudaStream_t s) {
  const dim3 grid(S, a.heads, 2 * mlstm_col_blocks(a.vd)), block(kMcThreads), cluster(1, 1, 2);
#define CHUNK(K, C)                                                                                            \
  do {                                                                                                         \
    static bool done[64] = {};                                                                                 \
    constexpr size_t smem = std::max(sizeof(McSmem<K>), (size_t)ml_floats(K / 4) * 4);   /* chunks; walk */         \
    B200_CUDA(ensure_dynamic_smem(mlstm_chunk_kernel<K, C>, (int)smem, done));                                 \
    B200_CUDA(launch_cluster(mlstm_chunk_kernel<K, C>, grid, block, smem, s, cluster, a));                     \
  } while (0)
  const bool own = mlstm_chunk_ctas(a, S) <= kNumSMs;   // an SM each
  if (a.dim <= 64) {
    if (own) CHUNK(4, 1);
    else CHUNK(4, 2);
  } else {
    if (own) CHUNK(8, 1);
    else CHUNK(8, 2);
  }
#undef CHUNK
  return B200_OK;
}

}  // namespace b200
