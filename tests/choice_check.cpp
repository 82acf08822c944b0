// CPU check of the kernel choice (test infrastructure, built by
// tests/test_choice.py with the library's layout.cpp): reads "order sms", a
// list of column counts ended by 0 and the blocks "row0 row1 col0 col1 rank"
// (rank 0: dense) from standard input, builds a matrix of that structure with
// made-up codes, and prints for each column count whether an apply takes the
// tensor-memory kernels.
#include <algorithm>
#include <cstdio>
#include <iostream>
#include <numeric>

#include "layout.hpp"

using namespace qhg;

int main() {
    HostMatrix m;
    int sms = 0;
    if (!(std::cin >> m.order >> sms)) return 2;
    std::vector<size_t> columns;
    for (size_t p; std::cin >> p && p;) columns.push_back(p);
    m.permutation.resize(m.order);
    std::iota(m.permutation.begin(), m.permutation.end(), uint64_t(0));
    // shares of the code widths, widest first
    const int widths[] = {32, 24, 16, 12, 8, 4};
    const double share[] = {0.20, 0.45, 0.56, 0.67, 0.80, 1.0};
    uint32_t seed = 1;
    auto words = [&](std::vector<uint32_t>& w, uint64_t codes, int width) {
        for (uint64_t k = words_for_bits(codes, width); k; --k) w.push_back(seed = seed * 1664525u + 1013904223u);
    };
    for (HostMatrix::Block b{}; std::cin >> b.row0 >> b.row1 >> b.col0 >> b.col1 >> b.rank;) {
        b.dense = b.rank == 0;
        if (b.dense) {
            b.dense_off = m.dense.size();
            m.dense.resize(m.dense.size() + (b.row1 - b.row0) * (b.col1 - b.col0), 1.0);
        }
        b.comp0 = m.width.size();
        for (uint64_t j = 0; j < b.rank; ++j) {
            const int w = widths[std::lower_bound(share, share + 5, (double(j) + 0.5) / double(b.rank)) - share];
            m.width.push_back(uint8_t(w));
            m.left_scale.push_back(1.0 / double(1ull << w));
            m.right_scale.push_back(1.0 / double(1ull << w));
            m.left_off.push_back(m.left_words.size());
            m.right_off.push_back(m.right_words.size());
            words(m.left_words, b.row1 - b.row0, w);
            words(m.right_words, b.col1 - b.col0, w);
        }
        m.blocks.push_back(b);
    }
    validate(m);
    const Layout L = build_layout(m);
    // (the warps of the column-by-column kernels' grids, as at upload)
    auto warps = [&](int units) { return 8 * std::max(1, std::min((units + 7) / 8, 2 * sms)); };
    const KernelChoice c = kernel_choice(L, schedule_units(column_costs(L), warps(L.n_tasks)),
                                         schedule_units(row_costs(L), warps(L.n_units)), sms);
    for (size_t p : columns) std::printf("%d ", int(c.tensor(p)));
    std::printf("\n");
}
