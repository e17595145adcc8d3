// packed_slots against the packings themselves, on random instances of every kind.
#include "../../analogsat_b200/csrc/as_problem.h"

#include <cstdio>
#include <random>

using namespace asb;

int main() {
    std::mt19937 rng(7);
    for (int t = 0; t < 60; t++) {
        const int n = t < 8 ? 1 + t * 11 : 20 + (int)(rng() % (t < 50 ? 700 : 40000));
        const int kmax = 1 + (int)(rng() % 6), m = 1 + (int)(rng() % (4 * n));
        std::vector<int32_t> lits, lens;
        for (int j = 0; j < m; j++) {
            const int k = t % 3 ? kmax : 1 + (int)(rng() % kmax);
            lens.push_back(k);
            for (int i = 0; i < k; i++) {  // some variables far more often than others, repeats allowed
                const int v = t % 2 ? 1 + (int)(rng() % n) : 1 + (int)((unsigned long long)(rng() % n) * (rng() % n) / n);
                lits.push_back(rng() % 2 ? v : -v);
            }
        }
        HostProblem p;
        p.add_clauses(lits.data(), lens.data(), m);
        for (int mode = 0; mode < 3; mode++) {
            if (n > 10000 && mode) continue;
            if (pack(p, mode).nslots != packed_slots(p)) {
                std::printf("instance %d mode %d\n", t, mode);
                return 1;
            }
        }
    }
    std::puts("slots ok");
    return 0;
}
