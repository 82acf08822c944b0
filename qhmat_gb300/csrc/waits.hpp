// The bounded wait of the tensor-memory kernels, without the device's
// instructions (checked on the CPU as well).
#pragma once

#ifdef __CUDACC__
#define QH_WAIT __host__ __device__ __forceinline__
#else
#define QH_WAIT inline
#endif

namespace qhg {

enum class Waited { kDone, kTold, kRanOut };

// Tests `done` until it is true; gives up when the block has been `told` to, or
// after `limit` tests (one that fails takes about 4 us).  A kernel that starts
// before its predecessor has finished would count the predecessor's time as its
// own, so every 256 tests it first waits for the predecessor (at once where that
// has finished): here, because a wait at the start of a role, or a test of its own
// in this loop, cost 3 - 7 % of an apply.
template <class Done, class Told, class Predecessor>
QH_WAIT Waited bounded_wait(Done&& done, Told&& told, Predecessor&& predecessor, int limit) {
    for (int i = 0; i < limit; ++i) {
        if (done()) return Waited::kDone;
        if ((i & 255) == 255) {
            if (told()) return Waited::kTold;
            predecessor();
        }
    }
    return Waited::kRanOut;
}

}  // namespace qhg

#undef QH_WAIT
