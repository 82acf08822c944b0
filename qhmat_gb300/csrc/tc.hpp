// Host interface of the tensor-memory kernels of the plain form (tc.cu).
#pragma once

#include "plain.hpp"

namespace qhg {

struct TcArgs {
    Arena A;
    Work W;
    int n_items, n_row_items, n_dense, n_parts, n_tiles;
    int rhs, pv, n, n_pad, n_split, n_dslices, sms;
    double* y;
    long long ld;
    int* status;
};

// Once per device: the kernels' shared memory.
cudaError_t tc_setup();
// Column, row and combine kernels in stream order; mark(ctx, 2), if given, is
// called after the column kernel.
cudaError_t tc_launch(const TcArgs& a, cudaStream_t s, void (*mark)(void*, int), void* ctx);

// Test aid (qh_debug_wait_timeout): two warps whose waits nothing ends; status: two
// words, out: 64.
cudaError_t tc_debug_give_up(int polls, int* status, int* out);

}  // namespace qhg
