// Barriers between the softmax warps, the MMA issuer and the tensor core of sparse_mla_decode.cu, and the phase of them that says
// that a step of chunk c is over. A wait names only the parity of a phase: it may stand only where the phase BEFORE the one that
// it means is known to be over (else it returns at once) and the one AFTER it cannot be (else it never returns). The kernel takes
// its barriers and parities from here; tests/test_mla_waits.py walks through all orders in which the roles can run.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define MLA_HD __host__ __device__ __forceinline__
#else
#define MLA_HD inline
#endif

namespace umdk {

enum MlaStep : int {
  kMlaS,     // S(c) = Q * K(c) is in TMEM: one commit
  kMlaP,     // P(c) has taken its place: an arrival of every softmax warp
  kMlaO,     // P(c) * V(c) has been added to O: one commit, for all chunks but the last
  kMlaEnd,   // every MMA of the split is through: one commit, c is ignored
};
constexpr int kMlaBars = 6;
MLA_HD constexpr bool mla_of_softmax(int bar) { return bar == 2 || bar == 3; }   // which of them the softmax warps arrive at

struct MlaWait {
  int bar;   // of kMlaBars
  uint32_t parity;
};

MLA_HD constexpr MlaWait mla_wait(MlaStep step, int c) {
  switch (step) {
    // Two barriers in turn: S(c) is made only when P(c-2) * V is through, so everybody has seen S(c-2) and P(c-2) by then.
    case kMlaS: return {c & 1, (uint32_t)(c >> 1) & 1u};
    // With a single one the softmax warps, who need only S(c+1) for it, could all arrive for P(c+1) before the issuer has looked
    // for P(c): a phase that is gone by, and both would wait for each other.
    case kMlaP: return {2 + (c & 1), (uint32_t)(c >> 1) & 1u};
    // The issuer waits for c - 2 before it makes S(c), the softmax warps for c - 1 where they rescale O behind S(c): in both places
    // the phase before is over, and the next one needs the S or P that the waiting role still has to make.
    case kMlaO: return {4, (uint32_t)c & 1u};
    // A barrier with a single phase: behind the last chunk only P(n-3) * V is known to be through, and kMlaO's barrier in that
    // phase would let a wait for P(n-1) * V pass before the last two products.
    default: return {5, 0u};
  }
}

}  // namespace umdk
