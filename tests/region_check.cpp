// The byte layout of the trailing updates' prepared operands, replayed on the
// host without a GPU: for every operand launch of an analysis's plans, each
// 16-byte piece that k_i8_split writes (the index arithmetic of i8_update.cuh
// restated here), and each that k_update_i8's tiles then copy. Checked:
//   - every piece lies inside its launch's regions (Launch::units, the stride
//     between the entries of a batch) and those inside the workspace of an entry;
//   - no piece is written twice, by one front or by two;
//   - a tile copies, of A and of B, and reads, of both rows' scales, only what
//     the operand launch just before it wrote for that front and panel group.
// tests/plan_check.cpp replays the arithmetic; its own check of the regions takes
// them for the 16 bytes a number of scaled rows, a third of what the digits take.
//
// Test infrastructure: built by oracle/Makefile, run by
// tests/test_operand_regions.py.
//
//   region_check cylinder <cells> [mistake] | fronts <seed> <count> <max_rows> [mistake]
//
// With [mistake] (short, units, workspace, brows, group: see plant_mistake) the
// plans are corrupted first, and the checks must fail.
// Prints one line per plan; exit status 0 when every check holds.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include "analysis.hpp"
#include "ordering.hpp"
#include "tc_config.hpp"
#include "workload.hpp"

using namespace aphi_b200;

namespace {

// A digit form: S digits, Nc complex columns a tile, bytes of a scale.
struct Form {
    const char* name;
    int S, Nc, real, kind_op, kind_up;
};
const Form kForms[2] = {{"fp64", kI8Digits64, kI8Nc64, 8, K_DMMA_SCALE, K_UPDATE_WIDE},
                        {"fp32", kI8Digits32, kI8Nc32, 4, K_TC_SPLIT, K_UPDATE_TC}};

constexpr long long kStage = kI8K;  // columns of K per stage, one byte each and digit

struct Layout {
    const Form& f;
    long long R;  // padded rows
    long long nst;
    long long block_a() const { return f.S * 2 * kTcM * kStage; }
    long long image_b() const { return f.S * 2 * f.Nc * kStage; }
    long long block_b() const { return 2 * image_b(); }
    long long a(long long r, long long c) const { return (r / kTcM * nst + c) * block_a(); }
    long long b(long long r, long long c) const { return R / kTcM * nst * block_a() + (r / f.Nc * nst + c) * block_b(); }
    long long scales() const { return R / kTcM * nst * block_a() + R / f.Nc * nst * block_b(); }
    static long long core(long long r, long long h) { return (r >> 3) * 256 + h * 128 + (r & 7) * 16; }
};

struct Counts {
    long long outside = 0, twice = 0, unwritten = 0, pieces = 0, tiles = 0, launches = 0;
    bool ok() const { return !outside && !twice && !unwritten; }
};

Counts check_plan(const aphi_analysis& A, const std::vector<Launch>& plan, const Form& f, long long ws_units) {
    const Symbolic& S = A.S;
    Counts n;
    std::vector<int> owner;                    // front that wrote each 16-byte piece of the launch's regions, or -1
    std::map<int, std::pair<int, int>> group;  // front -> (p0, K) of the operand launch
    const Launch* op = nullptr;
    for (const Launch& l : plan) {
        if (l.kind == f.kind_op) {
            op = &l;
            ++n.launches;
            if (l.units > ws_units) ++n.outside;
            owner.assign(static_cast<size_t>(std::max(l.units, 0)) * 16, -1);
            group.clear();
            for (int q = 0; q < l.count; ++q) {
                const Item& it = A.h_items[l.first + q];
                const int s = it.s, w = S.sn_first[s + 1] - S.sn_first[s], m = S.sn_rows[s];
                const int K = std::min(l.kcap, w - it.a), pe = it.a + K;
                const Layout y{f, (m - pe + kTcM - 1) / kTcM * kTcM, (K + kI8K - 1) / kI8K};
                group[s] = {it.a, K};
                auto put = [&](long long at, long long bytes) {
                    at += static_cast<long long>(it.d) * 256;
                    for (long long x = at / 16; x < (at + bytes + 15) / 16; ++x) {
                        ++n.pieces;
                        if (x < 0 || x >= static_cast<long long>(owner.size())) {
                            ++n.outside;
                            continue;
                        }
                        if (owner[x] >= 0) ++n.twice;
                        owner[x] = s;
                    }
                };
                for (int r = it.b; r < it.b + kTcM; ++r)
                    for (int c = 0; c < 2 * y.nst; ++c)
                        for (int p = 0; p < f.S; ++p)
                            for (int half = 0; half < 2; ++half) {  // re, im of A; the two halves of B's images
                                put(y.a(r, c >> 1) + Layout::core(r % kTcM, c & 1) + (2 * p + half) * kTcM * kStage, 16);
                                for (int image = 0; image < 2; ++image)
                                    put(y.b(r, c >> 1) + Layout::core(r % f.Nc, c & 1) + p * 2 * f.Nc * kStage +
                                            half * f.Nc * kStage + image * y.image_b(), 16);
                            }
                // Both scales of 128 rows: whole 16-byte pieces.
                put(y.scales() + static_cast<long long>(it.b) * f.real, static_cast<long long>(kTcM) * f.real);
                put(y.scales() + (y.R + it.b) * f.real, static_cast<long long>(kTcM) * f.real);
            }
        } else if (l.kind == f.kind_up) {
            for (int q = 0; q < l.count; ++q) {
                const Item& it = A.h_items[l.first + q];
                const int s = it.s, w = S.sn_first[s + 1] - S.sn_first[s], m = S.sn_rows[s];
                const int K = std::min(l.kcap, w - it.a), pe = it.a + K;
                const Layout y{f, (m - pe + kTcM - 1) / kTcM * kTcM, (K + kI8K - 1) / kI8K};
                const auto g = group.find(s);
                const bool fresh = op == &l - 1 && g != group.end() && g->second.first == it.a && g->second.second == K;
                if (!fresh || it.b < pe || it.c < pe || (it.b - pe) % kTcM || (it.c - pe) % kTcN) {
                    ++n.unwritten;
                    continue;
                }
                auto get = [&](long long at, long long bytes) {
                    at += static_cast<long long>(it.d) * 256;
                    for (long long x = at / 16; x < (at + bytes + 15) / 16; ++x)
                        if (x < 0 || x >= static_cast<long long>(owner.size()) || owner[x] != s) ++n.unwritten;
                };
                for (int j0 = it.c; j0 < it.c + kTcN; j0 += f.Nc) {
                    if (j0 >= m || it.b + kTcM <= j0) continue;  // the tile is skipped
                    ++n.tiles;
                    for (long long k = 0; k < y.nst; ++k) {
                        get(y.a(it.b - pe, k), y.block_a());
                        get(y.b(j0 - pe, k), y.block_b());
                    }
                    get(y.scales() + static_cast<long long>(it.b - pe) * f.real, static_cast<long long>(kTcM) * f.real);
                    get(y.scales() + (y.R + j0 - pe) * f.real, static_cast<long long>(f.Nc) * f.real);
                }
            }
        }
    }
    return n;
}

// The first operand launch of the FP64 plan, with its update just behind it,
// of at least `fronts` fronts.
Launch* operand_launch(aphi_analysis& A, int fronts) {
    for (size_t k = 0; k + 1 < A.plan_factor.size(); ++k) {
        Launch& l = A.plan_factor[k];
        if (l.kind != K_DMMA_SCALE) continue;
        int seen = 0, last = -1;
        for (int q = 0; q < l.count; ++q)
            if (A.h_items[l.first + q].s != last) last = A.h_items[l.first + q].s, ++seen;
        if (seen >= fronts) return &l;
    }
    return nullptr;
}

// A mistake in this process's copy of the FP64 plan: a region 20 % short, so
// that the next front's begins inside it ("short"); an entry's stride 20 % short
// ("units"); the workspace so ("workspace"); a block of B rows that no operand
// item wrote ("brows"); a tile of another panel group ("group").
bool plant_mistake(aphi_analysis& A, const std::string& what) {
    Launch* l = operand_launch(A, what == "short" ? 2 : 1);
    if (!l) return false;
    Item* op = A.h_items.data() + l->first;
    Launch& up = *(l + 1);
    if (what == "short") {
        int q = 0;
        while (op[q].s == op[0].s) ++q;
        const int s = op[q].s, moved = op[q].d - op[q].d / 5;
        for (; q < l->count && op[q].s == s; ++q) op[q].d = moved;
        for (int t = 0; t < up.count; ++t)
            if (A.h_items[up.first + t].s == s) A.h_items[up.first + t].d = moved;
        return true;
    }
    if (what == "units") {
        l->units -= l->units / 5;
        return true;
    }
    if (what == "workspace") {
        A.dmma_ws_units -= A.dmma_ws_units / 5;
        return true;
    }
    if (what == "brows") {  // the front's last 128 rows: some tile takes them as its columns
        for (size_t k = 0; k + 1 < A.plan_factor.size(); ++k) {
            Launch& o = A.plan_factor[k];
            if (o.kind != K_DMMA_SCALE || o.count < 2) continue;
            for (int q = 1; q < o.count; ++q) {
                Item& it = A.h_items[o.first + q];
                if (it.s == A.h_items[o.first + q - 1].s) {
                    it.b = A.h_items[o.first + q - 1].b;
                    return true;
                }
            }
        }
        return false;
    }
    if (what == "group") {
        A.h_items[up.first].a += kTcPanel;
        return true;
    }
    return false;
}

aphi_analysis_options options() {
    aphi_analysis_options o{};
    o.relax_small = 4;
    o.relax_fill = 0.05;
    o.relax_max_width = 256;
    o.small_front = 96;
    o.group4_rows = o.tc_group4_rows = 600;  // groups of one, two and four panels
    o.group2_rows = o.tc_group2_rows = 300;
    return o;
}

int check(aphi_analysis* A, const std::string& plant) {
    if (!plant.empty() && !plant_mistake(*A, plant)) {
        std::printf("nothing to plant: %s\n", plant.c_str());
        return 2;
    }
    const std::vector<Launch>* plans[2] = {&A->plan_factor, &A->plan_factor_tc};
    const long long ws[2] = {A->dmma_ws_units, A->tc_ws_units};
    int bad = 0;
    for (int p = 0; p < 2; ++p) {
        const Counts n = check_plan(*A, *plans[p], kForms[p], ws[p]);
        std::printf("%s launches %lld pieces %lld tiles %lld outside %lld twice %lld unwritten %lld %s\n", kForms[p].name,
                    n.launches, n.pieces, n.tiles, n.outside, n.twice, n.unwritten, n.ok() ? "ok" : "FAIL");
        bad += !n.ok();
    }
    analysis_destroy(A);
    return bad ? 1 : 0;
}

}  // namespace

int main(int argc, char** argv) {
    try {
        const std::string mode = argc > 1 ? argv[1] : "";
        if (mode == "cylinder" && (argc == 3 || argc == 4)) {
            Workload w;
            build_cylinder(w, std::atoi(argv[2]), 1.0, 0);
            std::vector<int> perm(w.num_total);
            reference_amd(w.num_total, w.row_ptr.data(), w.col_idx.data(), perm.data());
            return check(analysis_create(w.num_total, w.row_ptr.data(), w.col_idx.data(), perm.data(), nullptr, nullptr,
                                         options()),
                         argc == 4 ? argv[3] : "");
        }
        if (mode == "fronts" && (argc == 5 || argc == 6)) {
            std::mt19937 rng(static_cast<unsigned>(std::atoi(argv[2])));
            const int count = std::atoi(argv[3]), most = std::atoi(argv[4]);
            std::vector<int> rows(count), widths(count);
            for (int k = 0; k < count; ++k) {
                rows[k] = 97 + static_cast<int>(rng() % std::max(1, most - 96));
                widths[k] = 1 + static_cast<int>(rng() % (rows[k] - 1));
            }
            return check(analysis_create_fronts(count, rows.data(), widths.data(), options()), argc == 6 ? argv[5] : "");
        }
        std::fprintf(stderr, "usage: %s cylinder <cells> [mistake] | fronts <seed> <count> <max_rows> [mistake]\n", argv[0]);
        return 2;
    } catch (const std::exception& e) {
        std::fprintf(stderr, "region_check: %s\n", e.what());
        return 2;
    }
}
