// CPU check of the tensor-memory kernels' bounded wait (test infrastructure,
// built by tests/test_waits.py): a phase that completes a few tests after the
// preceding kernel ends, on a clock that a test moves by one and the wait for the
// predecessor to its end.
#include <cstdio>

#include "waits.hpp"

using namespace qhg;

namespace {

struct Run {
    Waited w;
    long tests;
};

Run run(long predecessor_end, long phase_after, int limit, int flag = 0, long flag_at = -1) {
    long clock = 0, tests = 0;
    int abort_flag = flag;
    const Waited w = bounded_wait(
        [&] {
            ++tests;
            if (++clock == flag_at) abort_flag = 1;
            return clock >= predecessor_end + phase_after;
        },
        [&] { return abort_flag != 0; }, [&] { clock = clock > predecessor_end ? clock : predecessor_end; }, limit);
    return {w, tests};
}

}  // namespace

int main() {
    int bad = 0;
    auto check = [&](const char* what, bool ok) {
        if (!ok) std::printf("FAIL: %s\n", what);
        bad += !ok;
    };
    // the predecessor takes far longer than the limit: not this wait's time
    Run r = run(1000000, 10, 2000);
    check("a slow predecessor does not run the wait out", r.w == Waited::kDone && r.tests <= 2000);
    r = run(0, 10, 2000);
    check("a short wait ends by its own tests", r.w == Waited::kDone && r.tests == 10);
    r = run(0, 5000, 2000);
    check("a phase that does not complete runs the wait out", r.w == Waited::kRanOut && r.tests == 2000);
    r = run(0, 1000000, 100000, 0, 700);
    check("a wait ends when the block is told", r.w == Waited::kTold && r.tests > 700 && r.tests <= 700 + 256);
    r = run(0, 1, 2000, 1);
    check("a complete phase is seen in a block that has been told", r.w == Waited::kDone);
    std::printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
