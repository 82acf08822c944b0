// CPU check of the tensor-memory kernels' work lists (test infrastructure, built
// by tests/test_worklists.py with the library's layout.cpp): for a QHMAT001 file,
// they cover every column task, dense unit, row unit and k-pair of the layout
// exactly once, within the sizes that the kernels' stages and accumulators have.
#include <algorithm>
#include <cstdio>
#include <fstream>
#include <iterator>
#include <map>
#include <tuple>
#include <vector>

#include "layout.hpp"

using namespace qhg;

namespace {

int fails = 0;
void check(bool ok, const char* what, long a = 0, long b = 0) {
    if (!ok && fails++ < 20) std::printf("FAIL: %s (%ld, %ld)\n", what, a, b);
}
template <class T>
const T* sec(const Layout& L, size_t off) {
    return reinterpret_cast<const T*>(L.arena.data() + off);
}

void columns(const Layout& L) {
    const auto* tasks = sec<ColTask>(L, L.sec.tasks);
    const auto* items = sec<TcItem>(L, L.sec.tc_items);
    const auto* parts = sec<TcTask>(L, L.sec.tc_tasks);
    const auto* dense = sec<DenseUnit>(L, L.sec.dense_units);
    std::map<std::pair<int32_t, int32_t>, const ColTask*> left;  // (first component, first chunk)
    std::vector<std::tuple<int, int, int, int, int>> units, listed;
    for (int i = 0; i < L.n_tasks; ++i) {
        const ColTask& T = tasks[i];
        if (T.width) left[{T.comp_idx, T.chunk0}] = &T;
        else units.emplace_back(T.col0, T.stride, T.comp_idx, T.chunk0, T.n);
    }
    for (int i = 0; i < L.n_tc_items; ++i) {
        const TcItem& I = items[i];
        const int planes = I.info & 255, count = I.info >> 8;
        check(count >= 1 && count <= 4 && planes >= 1 && planes <= 4, "item", i, I.info);
        for (int s = 0; s < 4; ++s) {
            const TcTask& t = parts[4 * i + s];
            if (s >= count) {
                check(t.info == 0 && t.stride == 0 && t.nparts == 1, "empty part", i, s);
                continue;
            }
            const auto at = left.find({t.comp_idx, I.chunk0});
            if (at == left.end()) {
                check(false, "no such task, or twice", t.comp_idx, I.chunk0);
                continue;
            }
            const ColTask& T = *at->second;
            check(T.col0 == I.col0 && T.nchunks == I.nchunks && code_planes(T.width) == planes, "item of a task", i, s);
            check(t.off == T.off + int64_t(T.chunk0) * T.stride && t.stride == T.stride, "codes", i, s);
            check(t.info == (T.count | T.width << 8) && t.split == T.split_id && t.nparts == T.nparts, "task", i, s);
            check((planes <= 2 ? 2 : 1) * t.stride <= 4096, "stage", i, t.stride);
            left.erase(at);
        }
    }
    check(left.empty(), "tasks left", long(left.size()));
    for (int i = 0; i < L.n_dense_units; ++i)
        listed.emplace_back(dense[i].tdense, dense[i].tile, dense[i].slice, dense[i].k0, dense[i].cols);
    std::sort(units.begin(), units.end());
    std::sort(listed.begin(), listed.end());
    check(units == listed, "dense units");
}

void rows(const Layout& L) {
    const auto* tiles = sec<RowTile>(L, L.sec.tiles);
    const auto* units = sec<RowUnit>(L, L.sec.units);
    const auto* items = sec<TcRowItem>(L, L.sec.tc_row_items);
    const auto* steps = sec<TcStep>(L, L.sec.tc_steps);
    const uint8_t* info = sec<uint8_t>(L, L.sec.kp_info);
    std::map<std::tuple<int, int, int>, const RowUnit*> unit;  // (tile, M-tile, split)
    for (int i = 0; i < L.n_units; ++i) unit[{units[i].tile, units[i].q, units[i].h}] = &units[i];
    std::map<int32_t, const TcRowItem*> item;  // by partial sum
    for (int i = 0; i < L.n_tc_row_items; ++i)
        check(item.insert({items[i].part, &items[i]}).second, "partial sum twice", items[i].part);
    check(int(item.size()) == L.n_parts, "partial sums", long(item.size()), L.n_parts);
    for (int t = 0; t < L.n_tiles; ++t) {
        const RowTile& T = tiles[t];
        const int rs = T.parts >> 16, parts = T.parts & 0xFFFF;
        check(rs == (T.rows <= 32 ? 32 : 64), "row shape", t, rs);
        int h = 0;  // the tile's splits, in the order of its items
        for (int p = T.part0; p < T.part0 + parts; ++p) {
            if (!item.count(p)) {
                check(false, "no item", t, p);
                continue;
            }
            const TcRowItem& I = *item[p];
            item.erase(p);
            check(I.shape == (rs | T.qrows << 8) && I.nsteps > 0, "shape", t, I.shape);
            for (int s = 0; s < I.nsteps; ++h) {
                if (h >= T.nh) {
                    check(false, "too many steps", t, s);
                    break;
                }
                const RowUnit& U0 = *unit[{t, 0, h}];
                int64_t done = 0;
                int segment = 0, planes = 0;
                for (int k = 0; k < U0.nkps && s < I.nsteps; k += 2, ++s) {
                    const TcStep& S = steps[I.step0 + s];
                    const int kps = std::min(2, U0.nkps - k);
                    check(S.slot == U0.slot0 + 32 * k && S.nslots == 32 * kps, "slots", t, s);
                    for (int q = 0; q < T.qrows; ++q)
                        check(int64_t(S.code[q]) * 256 == unit[{t, q, h}]->code_off + done, "codes", t, s);
                    int64_t bytes = 0;
                    for (int j = 0; j < 2; ++j) {
                        const int b = int(S.info >> (8 * j)) & 255;
                        const int expect = j < kps ? info[U0.kp_off + h + int64_t(k + j) * T.hsplit] : 0;
                        check(b == expect, "k-pair", t, s);
                        bytes += 512 * (b & 7) - ((b & 8) ? 256 : 0);
                        if (segment == 0 && j == 0) planes = b & 7;
                        check((b & 7) <= planes, "planes grow in a segment", t, s);
                    }
                    check(bytes <= 4096, "stage", t, bytes);
                    done += bytes;
                    const bool last = k + 2 >= U0.nkps;
                    const bool end = (S.info & kSegmentEnd) != 0;
                    check(end || (!last && segment == 0), "segment of more than two steps or one split", t, s);
                    check(((S.info & kItemEnd) != 0) == (s == I.nsteps - 1), "item end", t, s);
                    segment = end ? 0 : 1;
                }
            }
        }
        check(h == T.nh, "splits", t, h);
    }
    check(item.empty(), "items of no tile", long(item.size()));
}

}  // namespace

int main(int argc, char** argv) {
    if (argc < 2) return 2;
    std::ifstream f(argv[1], std::ios::binary);
    std::vector<uint8_t> bytes((std::istreambuf_iterator<char>(f)), {});
    const Layout L = build_layout(parse_qhmat(bytes.data(), bytes.size()));
    columns(L);
    rows(L);
    std::printf(fails ? "FAILED %d\n" : "OK\n", fails);
    return fails != 0;
}
