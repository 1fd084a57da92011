// How a step's runs of rows are shared between the tcgen05 attention kernel (attn_rows_tc.cu) and the mma.sync one (attn_latent.cu).  How the rows
// fall into runs is known on the device only, so both are launched, one after the other, and each finds its share by the same rule over the
// same run lists.
#pragma once
#include "common.cuh"

namespace b200 {

struct RunShare {
  const int32_t* n_runs;   // runs of the list that the tcgen05 kernel walks; null: it is launched alone
  int32_t* ticket;         // the mma.sync kernel's next item, which the tcgen05 kernel before it sets to 0
  int rows;                // of the step
  int lanes, parts;        // kv heads x splits; items that the tcgen05 kernel cuts a run into
};

constexpr int kRunsAll = 1 << 30;

// Whole runs (runs that are all of their rows' segment) of at most so many (row, head) pairs are the mma.sync kernel's: 0 none, kRunsAll
// every run, whole or not.  A tcgen05 CTA takes an item of few pairs in the time that it takes 128 in, an mma.sync one 16 pairs in about half
// of that with four to an SM; the kernels run one after the other.  So
//  * one kernel takes the step while the tcgen05 kernel needs no more than two rounds of CTAs: the mma.sync one where an item has 16 pairs or
//    fewer on average;
//  * larger steps are shared: runs of up to two chunks go to the mma.sync kernel.
// Measured with 16 heads at contexts 300 to 600, us, the step on the mma.sync kernel alone, on one of the two by its runs' mean length, by this
// rule: 300 decode rows and 700 of one sequence 230, 417, 193 (over 4 kv heads) and 159, 1 100, 129 (over one); 64 and 1 000 213, 131, 119; 40 and
// 260 71, 70, 69; 50 runs of 4 rows 56, 72, 66, of 6 rows 58, 41, 41; 100 runs of 2 rows over one kv head 47, 116, 48.  What the second launch
// costs a step that does not need it: 200 decode rows 94 -> 100, 1 000 308 -> 327 (decode steps that say so are launched without it).
__device__ __forceinline__ int run_share(const RunShare& s, int G) {
  const int n = *s.n_runs;
  if (n * s.lanes * s.parts > 2 * kNumSMs) return 32;
  return s.rows * G > 16 * n ? 0 : kRunsAll;
}

// Latent attention of a step that either of two kernels may take.  Rows by themselves (attn_latent_rows.cu) put `cluster` CTAs on a row's 16 heads, which
// walk its context together; over runs (attn_latent_tc.cu) up to 128 (row, head) pairs share a walk, cut into `splits` by CTAs and merged.  Which is faster
// hangs on how the rows fall into runs and on how uneven their contexts are: known on the device only, so both are launched where it matters
// (latent_attn_route), and each estimates both from the run plan.  The estimates, in ns, from 1..148 rows of 4..128 heads over 512 + 64, 512, 256 + 32, 128 + 64
// and 64 + 16 at contexts 300..64 000, of one sequence, of as many as rows, and one long among short ones:
//   rows: 4.2 + 0.035 krow a key and CTA       runs: 10 us + 54 krow for splits and merge, 1.15 max(16.5, 0.043 krow) a key and CTA, whole rounds of items
// e.g. 100 rows of 16 heads over 512 + 64, us, rows and runs: one sequence of 16 100 tokens 385, 183; as many of 16 000 403, 732; one of 32 000 among 600s
// 756, 368.  The launches that a step does not need cost it 8 us.
struct LatentShare {
  const int32_t* plan;   // its words; null: the kernel has the step to itself
  int rows, splits, halves, rows_per_item, seen;   // seen: a window's tokens (or INT_MAX)
  // ns of a key of the longest row and of a 64-token tile of all runs, by rows; the fixed part, a key of the longest row and a key of an item over runs
  float row_key, row_tile, run_fixed, run_key, run_item;
};
// Every kernel of the step has to come to the same answer: products and sums are rounded one by one, not as a compiler joins them.
__host__ __device__ __forceinline__ float ls_mul(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
__host__ __device__ __forceinline__ bool latent_by_rows(const LatentShare& s, int n_runs, int longest, int tiles) {
  const float most = (float)(longest < s.seen ? longest : s.seen), each = ls_mul((float)((s.seen >> 6) + 2), (float)n_runs);
  const float walked = fminf((float)tiles, each);                                            // tiles of all runs
  const int parts = (s.rows + n_runs * s.rows_per_item - 1) / (n_runs * s.rows_per_item);    // items of a run in the mean
  const int rounds = (n_runs * parts * s.halves * s.splits + kNumSMs - 1) / kNumSMs;
  const float by_rows = fmaxf(ls_mul(s.row_key, most), ls_mul(s.row_tile, walked));
  const float per_item = ls_mul(walked, (float)rounds), run = fmaxf(ls_mul(ls_mul(s.run_key, most), (float)n_runs), ls_mul(s.run_item, per_item));
  // (both sides times n_runs: no division)
#ifdef __CUDA_ARCH__
  return ls_mul(by_rows, (float)n_runs) <= __fadd_rn(ls_mul(s.run_fixed, (float)n_runs), run);
#else
  return ls_mul(by_rows, (float)n_runs) <= s.run_fixed * (float)n_runs + run;
#endif
}
__device__ __forceinline__ bool latent_by_rows(const LatentShare& s) {
  return latent_by_rows(s, max(__ldcg(s.plan), 1), __ldcg(s.plan + kRunLongest), __ldcg(s.plan + kRunTiles));
}

// Is a run (its second word) the mma.sync kernel's?  A segment of at most kRunRows rows is one run in every list.
__device__ __forceinline__ bool run_is_short(int pairs, int run, int G) {
  return pairs == kRunsAll || ((run & kRunWhole) && (run & kRunLength) <= kRunRows && (run & kRunLength) * G <= pairs);
}

}  // namespace b200
