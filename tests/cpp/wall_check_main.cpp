// Host-only driver of the wall table and its index check (built by
// tests/test_wall_table.py with g++ from the library's host sources): reads a
// deck directory, builds the table as the solver does, checks it (expects a
// pass), then plants one bad entry per array and expects each to be caught.
// Prints the counts and exits 0 when every case behaved.
#include <cstdio>
#include <functional>
#include <vector>

#include "gbte_internal.h"

using namespace gbte;

int main(int argc, char **argv) {
    Deck D;
    if (argc < 2 || read_deck(argv[1], D).code) return 2;
    D.bands.kappa.assign(D.bands.nmat, 1.0);
    D.bands.capb.assign(D.bands.nmat, 1.0);
    FlatMesh m;
    if (build_flat_mesh(D.mesh, D.bcs, D.bands, m).code) return 2;
    WallTable built;
    build_wall_table(m, built);
    int bad = 0;
    auto run = [&](const char *name, bool expect_pass, const std::function<void(WallTable &)> &plant) {
        WallTable w = built;
        plant(w);
        long long n = 0;
        const Error r = check_walls(m, w, n);
        const bool passed = r.code == 0;
        std::printf("%s: %s %s\n", name, passed ? "pass" : "caught", r.msg.c_str());
        if (passed != expect_pass || (!passed && r.code != -7)) bad++;
    };
    run("built", true, [](WallTable &) {});
    run("cf_slot past the slots", false, [](WallTable &w) {
        for (int &s : w.cf_slot)
            if (s >= 0) {
                s = w.nslots;
                break;
            }
    });
    run("slot on an interior face", false, [&](WallTable &w) {
        for (size_t k = 0; k < w.cf_slot.size(); k++)
            if (m.cf_bound[k] < 0) {
                w.cf_slot[k] = 0;
                break;
            }
    });
    run("side past the sides", false, [&](WallTable &w) { w.side.back() = m.nbs(); });
    run("side listed twice", false, [](WallTable &w) { w.side.back() = w.side.front(); });
    run("side not listed", false, [](WallTable &w) { w.side.pop_back(), w.slot.pop_back(); });
    run("slot of another face", false, [](WallTable &w) { w.slot[0] = w.slot[1]; });
    long long n = 0;
    std::vector<int> col = {0, 1, 2, 2};
    if (check_columns("columns", col, 4, 3, n).code != 0) bad++;
    col[3] = 3;
    if (check_columns("columns", col, 4, 3, n).code != -7 || check_columns("columns", col, 5, 4, n).code != -7) bad++;
    std::printf("slots %d walls %zu %s\n", built.nslots, built.side.size(), bad ? "FAILED" : "OK");
    return bad ? 1 : 0;
}
