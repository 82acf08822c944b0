// CPU check of the page populator (test infrastructure, built by
// tests/test_pages.py): threads that cannot be made leave their part to the
// copy and end nothing; every page of the rest is written, no byte outside.
// Argument: which allocation while the threads are made fails (0: none).
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "pages.hpp"

namespace {
int countdown = 0;  // the allocation that fails, counted from now (0: none)
}
void* operator new(std::size_t n) {
    if (countdown > 0 && --countdown == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main(int argc, char** argv) {
    const int fails = argc > 1 ? std::atoi(argv[1]) : 0;
    const std::size_t page = std::size_t(sysconf(_SC_PAGESIZE));
    int bad = 0;
    for (std::size_t bytes : {std::size_t(5) << 20, (std::size_t(33) << 20) + 8, (std::size_t(16) << 20) - 24}) {
        std::vector<unsigned char> v(bytes + 64, 0xFF);
        unsigned char* b = v.data() + 24;
        countdown = fails;
        { qhg::PagePopulator p(b, bytes); }
        countdown = 0;
        for (std::size_t i = 0; i < 24; ++i) bad += v[i] != 0xFF;
        for (std::size_t i = bytes + 24; i < v.size(); ++i) bad += v[i] != 0xFF;
        bad += b[bytes - 1] != 0;  // the caller's own part ends the buffer
        if (fails) continue;
        for (std::size_t i = 0; i < bytes; i += page) {  // a zero in every page
            std::size_t k = i;
            while (k < i + page && k < bytes && b[k]) ++k;
            bad += k == i + page || k == bytes;
        }
    }
    std::printf(bad ? "FAIL %d\n" : "OK\n", bad);
    return bad != 0;
}
