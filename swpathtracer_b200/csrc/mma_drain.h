// mma_drain.h -- the end of a CTA whose wait for its MMAs ran out (plain C++: the host tests run it too).
#pragma once

#ifdef __CUDACC__
#define SPT_HOST_DEVICE __host__ __device__
#else
#define SPT_HOST_DEVICE
#endif

namespace spt {
namespace tc {

// No MMA may be in flight when its operands and its columns go.  By the thread that issued them all: the
// phase that was waited for (`waited`, a parity), then, behind a commit of their own, the MMAs that have
// been issued since that phase's commit.  Each wait is bounded; a commit whose phase has not completed is
// not followed by another.  True when nothing is in flight any more.
template <typename Wait, typename Commit>
SPT_HOST_DEVICE inline bool drain(unsigned waited, Wait&& wait, Commit&& commit) {
    if (!wait(waited)) return false;
    commit();
    return wait(waited ^ 1u);
}

}  // namespace tc
}  // namespace spt
