// Host-side check of the list places (compiled and run by
// tests/test_pair_places_host.py, no GPU): pair_first gives every cell room
// for its pairs, cell after cell, and never more places than there are atoms,
// over dense, dilute, empty and clustered cells.
#include <cstdio>
#include <random>
#include <vector>

#include "../../nexusmd_gb300/csrc/nxm_view.h"

using namespace nxm;

static bool check(const char *what, const std::vector<int> &count) {
    int start = 0, atoms = 0;
    for (int n : count) atoms += n;
    bool ok = pair_first(0, 0) == 0;
    for (size_t c = 0; c < count.size(); ++c) {
        const int n = count[c], room = pair_first(start + n, (int)c + 1) - pair_first(start, (int)c);
        ok = ok && room >= (n + 1) / 2;
        start += n;
    }
    const int places = pair_first(atoms, (int)count.size());
    ok = ok && places <= atoms && places <= (int)((atoms + count.size()) / 2);
    std::printf("%s: %d atoms, %zu cells, %d places%s\n", what, atoms, count.size(), places, ok ? "" : " WRONG");
    return ok;
}

int main() {
    std::mt19937 g(5);
    bool ok = check("none", std::vector<int>(1000, 0)) && check("one cell", {1}) && check("one full cell", {77});
    auto filled = [&](size_t cells, double mean) {
        std::vector<int> c(cells);
        std::poisson_distribution<int> p(mean);
        for (int &n : c) n = p(g);
        return c;
    };
    for (double mean : {0.001, 0.02, 0.3, 0.9, 1.0, 1.1, 3.0, 16.0}) ok = check("even", filled(20000, mean)) && ok;
    // a droplet in a large box: the cells before it, in it and behind it
    for (size_t at : {(size_t)0, (size_t)9000, (size_t)19000}) {
        std::vector<int> c(20000, 0), d = filled(1000, 12.0);
        for (size_t k = 0; k < d.size(); ++k) c[at + k] = d[k];
        ok = check("droplet", c) && ok;
        for (size_t k = 0; k < c.size(); k += 7) c[k] += 1;
        ok = check("droplet in vapour", c) && ok;
    }
    std::printf("%s\n", ok ? "OK" : "FAILED");
    return ok ? 0 : 1;
}
