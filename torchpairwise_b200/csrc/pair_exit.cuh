// How a pair of CTAs that share a ring of operand slots may end (gemm_tcgen05.cu, bool_tcgen05.cu).  Plain C++ that the host can
// run as well: the tests play every order of arrivals through these rules.
//
// Use u of the ring is slot u % slots, filled for the (u / slots)-th time.  Both CTAs copy their share of a use into their own slot,
// and both copies complete on rank 0's full[slot], which rank 0 arms for the bytes of both when it issues its own.  Rank 0's issuer
// reads the use and commits: an arrival at empty[slot] in either CTA.  Neither kind of arrival comes from a thread, so no barrier
// between threads waits for it, and the order in which two commits arrive is not defined.  A CTA whose shared memory is the target
// of one that is still under way must not end: the arrival would land in whatever runs there next.
//
// A run without errors: every use has been read, hence all copies have landed; what may be under way are the commits of each slot's
// last use, for which both CTAs' producers wait.
// After a wait that gave up, each role has stopped where it happened to be: the producers have issued `issued0` and `issued1` uses and
// `used` of them have been read (used <= both; neither is more than `slots` past it).  Besides the commits of the last uses that were
// read, the copies of the uses from `used` on are under way, and a full barrier whose use only one CTA issued never completes by
// itself: rank 0 accounts for the other CTA's part, then waits for it like for the rest.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TPW_BOTH_SIDES __host__ __device__ __forceinline__
#else
#define TPW_BOTH_SIDES inline
#endif

namespace tpw {

// The first of the uses that a slot each has seen last.
TPW_BOTH_SIDES uint32_t first_of_last_uses(uint32_t uses, uint32_t slots) { return uses > slots ? uses - slots : 0; }
TPW_BOTH_SIDES uint32_t parity_of_use(uint32_t use, uint32_t slots) { return (use / slots) & 1; }

// What rank 0 does to full[use % slots] before it waits for it after a wait that gave up.
enum class PairDebt {
    none,      // both CTAs have issued the use, and the barrier is armed for both
    arm_other, // only rank 1 has: arm the barrier for its bytes
    forgive    // only rank 0 has, and armed the barrier for both: count rank 1's bytes as here
};
TPW_BOTH_SIDES PairDebt debt_of_use(uint32_t use, uint32_t issued0, uint32_t issued1) {
    return use >= issued0 ? PairDebt::arm_other : use >= issued1 ? PairDebt::forgive : PairDebt::none;
}

} // namespace tpw
