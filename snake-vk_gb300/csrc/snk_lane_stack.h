// snk_lane_stack.h -- the pop of a stack that several lanes of a warp keep in common.
//
// The lanes make the same calls and every lane stores every entry, so that a push needs
// no wait: a lane reads back what it (or a lane ahead of it) has stored, the same value.
// A pop does: the entry it frees is overwritten by the next push, and nothing else holds
// a lane that is ahead back from it.  wait() is a barrier of the stack's lanes that
// orders their memory accesses (__syncwarp of their mask).
#pragma once

#ifdef __CUDACC__
#define SNK_LANE_FN __device__ __forceinline__
#else
#define SNK_LANE_FN inline
#endif

namespace snk {

// the top entry (at(k): entry k) of a stack of sp entries
template <class T, class At, class Wait>
SNK_LANE_FN T lanes_pop(At&& at, int& sp, Wait&& wait) {
    const T v = at(--sp);
    wait();
    return v;
}

}  // namespace snk
