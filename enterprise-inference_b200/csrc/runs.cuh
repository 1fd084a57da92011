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

// Is a run (its second word) the mma.sync kernel's?  A segment of at most kRunRows rows is one run in every list.
__device__ __forceinline__ bool run_is_short(int pairs, int run, int G) {
  return pairs == kRunsAll || ((run & kRunWhole) && (run & kRunLength) <= kRunRows && (run & kRunLength) * G <= pairs);
}

}  // namespace b200
