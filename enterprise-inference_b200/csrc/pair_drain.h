// The end of a pair of CTAs (gemm_pair.cu) in which a wait ran out: what the leader's barriers still wait for.  Plain C++, checked on the CPU.
//
// Both CTAs' loads of a fill complete on the leader's barrier of its stage; the leader announces both CTAs' bytes when it issues its own.  A fill is issued
// once the MMAs of the fill before it in the same stage have been committed, which they are not for a fill whose barrier did not complete.  So the two CTAs'
// counts differ by at most one fill a stage when they stop, and at most one phase of a barrier is open:
//   * both issued it:       it completes by itself
//   * only the leader:      the peer's bytes never come; they are taken off the barrier's count
//   * only the peer:        nobody announced its bytes; they are announced now
// after which the phase completes exactly when everything that was issued has landed.
#pragma once

#if defined(__CUDACC__)
#define PAIR_DRAIN_HD __host__ __device__
#else
#define PAIR_DRAIN_HD
#endif

namespace b200 {

struct PairOwed {
  int parity;     // of the phase to wait for; -1: the stage was never filled
  int fill;       // the fill that one CTA alone issued (both: any)
  int announce;   // +1: its half is announced (one arrival); -1: its half is taken off; 0: nothing
};

// lead, peer: fills that either CTA issued in all, fill i into stage i % stages
PAIR_DRAIN_HD inline PairOwed pair_owed(int stage, int stages, int lead, int peer) {
  const int nl = (lead - stage + stages - 1) / stages, np = (peer - stage + stages - 1) / stages;   // fills of this stage (counts from 0 on)
  PairOwed r;
  r.fill = stage + ((nl > np ? nl : np) - 1) * stages;
  r.announce = np > nl ? 1 : np < nl ? -1 : 0;
  const int phases = nl > np ? nl : np;
  r.parity = phases > 0 ? (phases - 1) & 1 : -1;
  return r;
}

}  // namespace b200
