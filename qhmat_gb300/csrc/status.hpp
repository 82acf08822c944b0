// Pinned status words of the calls that wait for their result and report what
// the kernels flagged.  The kernels OR into the word itself (the host's int
// is device-accessible at the same address), so there is nothing to clear or to
// copy on the stream.
#pragma once

#include <cuda_runtime.h>

#include <mutex>

#include "../../include/qhmat_gb300.h"

namespace qhg {

// A handle's words: one per call in flight, up to kKept of them kept for the
// next calls, freed with the handle.
class StatusWords {
public:
    ~StatusWords() {
        for (int i = 0; i < n_; ++i) cudaFreeHost(idle_[i]);
    }
    // The first word, ahead of the first call (calls at the same time make more).
    // Without memory for it now, that call asks again.
    void prepare() {
        int* word = nullptr;
        if (take(&word) == cudaSuccess) give(word);
        else cudaGetLastError();
    }
    cudaError_t take(int** out) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (n_) {
                *out = idle_[--n_];
                return cudaSuccess;
            }
        }
        return cudaMallocHost(out, sizeof(int));
    }
    void give(int* word) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (n_ < kKept) {
                idle_[n_++] = word;
                return;
            }
        }
        cudaFreeHost(word);
    }

private:
    static constexpr int kKept = 8;
    std::mutex mu_;
    int n_ = 0;
    int* idle_[kKept];
};

// Run `launch(word)` (returns a QH_* status), wait for the stream and read
// what the kernels flagged (`fail(error, status bits, what failed)`).  A call
// refused for its arguments has launched nothing and returns at once.
template <class Launch, class Fail>
int checked_call(StatusWords& words, cudaStream_t s, Launch&& launch, Fail&& fail) {
    int* word = nullptr;
    cudaError_t e = words.take(&word);
    if (e != cudaSuccess) return fail(e, 0, "cudaMallocHost");
    *static_cast<volatile int*>(word) = 0;
    const int rc = launch(word);
    if (rc == QH_EINVAL || rc == QH_EOVERFLOW) {
        words.give(word);
        return rc;
    }
    // (also after a failed launch: kernels before it may still write the word)
    e = cudaStreamSynchronize(s);
    const int st = *static_cast<volatile int*>(word);
    words.give(word);
    if (rc) return rc;
    if (e != cudaSuccess || st) return fail(e, st, "CUDA kernel execution");
    return 0;
}

}  // namespace qhg
