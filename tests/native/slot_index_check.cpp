// CPU check of the serial slice kernels' index arithmetic
// (peridyn_b200/csrc/pd_slots.h): two adjacent multi-type lattice blocks,
// particle counts on and off the multiples of 32, stencil slices built as
// the library builds them (the union of the lanes' offsets).  Every slot of
// every lane, used or not, must read a particle's record of its own block
// and index inside the block's pair table, and a used slot must find its own
// neighbour and pair.  Prints "ok <slots>" or the first
// failure; exit status 0 on success.
#include <algorithm>
#include <cstdio>
#include <functional>
#include <set>
#include <vector>

#include "../../peridyn_b200/csrc/pd_slots.h"

using namespace pd;

namespace {

struct Block {
    int dims[3], nt;
    int first, n, padded, pair_base;
};

int failures = 0;
long checked = 0;

int type_of(const Block &b, int i) { return (i * 7 + i / 5) % b.nt; }

// Family members (descending) of particle i of a lattice within r spacings.
std::vector<int> family(const Block &b, int i, double r) {
    std::vector<int> out;
    const int cx = i % b.dims[0], cy = i / b.dims[0] % b.dims[1], cz = i / (b.dims[0] * b.dims[1]);
    for (int j = b.n - 1; j >= 0; --j) {
        const int dx = j % b.dims[0] - cx, dy = j / b.dims[0] % b.dims[1] - cy, dz = j / (b.dims[0] * b.dims[1]) - cz;
        if (j != i && dx * dx + dy * dy + dz * dz < r * r) out.push_back(j);
    }
    return out;
}

void check(std::vector<Block> blocks, double r) {
    int N = 0, pairs = 0;
    for (auto &b : blocks) {
        b.n = b.dims[0] * b.dims[1] * b.dims[2];
        b.first = N;
        b.padded = (b.n + 31) / 32 * 32;
        b.pair_base = pairs;
        N += b.padded;
        pairs += b.nt * b.nt;
    }
    std::vector<int> tinfo(N, -1);
    for (size_t k = 0; k < blocks.size(); ++k)
        for (int i = 0; i < blocks[k].n; ++i) tinfo[blocks[k].first + i] = (int)k << 8 | type_of(blocks[k], i);
    for (const Block &b : blocks)
        for (int s = b.first; s < b.first + b.padded; s += 32) {
            std::vector<std::vector<int>> fam(32);
            std::set<int, std::greater<int>> offs;
            for (int l = 0; l < 32; ++l)
                if (s + l < b.first + b.n) {
                    fam[l] = family(b, s + l - b.first, r);
                    for (int &j : fam[l]) offs.insert((j += b.first) - (s + l));
                }
            if (offs.empty()) continue;
            // the layout's stencil condition: every lane with bonds names records of the environment
            bool ok = true;
            for (int l = 0; l < 32; ++l)
                if (!fam[l].empty()) ok = ok && s + l + *offs.begin() < N && s + l + *offs.rbegin() >= 0;
            if (!ok) continue;
            for (int l = 0; l < 32; ++l)
                for (const int o : offs) {
                    const int p = s + l;
                    const bool live = std::binary_search(fam[l].begin(), fam[l].end(), p + o, std::greater<int>());
                    const int q = slot_record(true, lane_record(p, tinfo[p]), o, live);
                    const int qe = slot_record(false, lane_record(p, tinfo[p]), live ? p + o : 0, live);
                    if (q < b.first || q >= b.first + b.n || q != qe || (live && q != p + o)) {
                        if (!failures++)
                            std::printf("lane %d of slice %d, offset %d: record %d (explicit %d) outside [%d, %d)\n", l,
                                        s / 32, o, q, qe, b.first, b.first + b.n);
                        continue;
                    }
                    const int tp = tinfo[p] >= 0 ? tinfo[p] & 255 : 0;
                    const int k = slot_pair(b.pair_base, b.nt, tp, tinfo[q], live);
                    ++checked;
                    if (k < b.pair_base || k >= b.pair_base + b.nt * b.nt ||
                        (live && k != b.pair_base + tp + type_of(b, q - b.first) * b.nt)) {
                        if (!failures++)
                            std::printf("lane %d of slice %d, offset %d: pair %d outside [%d, %d)\n", l, s / 32, o, k,
                                        b.pair_base, b.pair_base + b.nt * b.nt);
                    }
                }
        }
}

}  // namespace

int main() {
    for (const int e : {2, 3, 4, 5, 7, 8})
        for (const int nt : {2, 3, 128})
            check({{{7, e, 3}, nt, 0, 0, 0, 0}, {{e, 5, 4}, nt + 1, 0, 0, 0, 0}, {{8, 4, e}, 2, 0, 0, 0, 0}}, 2.3);
    if (failures) return 1;
    std::printf("ok %ld\n", checked);
    return 0;
}
