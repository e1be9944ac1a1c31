// Host check of below_fraction (gp_refine_small.cuh) against the host loop's
// long double comparison, on random and boundary pairs.
#include <cmath>
#include <cstdio>
#include <random>

#include "../horkxg_b200/csrc/gp_refine_small.cuh"

int main() {
    const gp::u64 fraction = static_cast<gp::u64>(std::ldexp(0.999L, 64));
    std::mt19937_64 rng(7);
    long bad = 0, checked = 0;
    auto check = [&](gp::u64 current, gp::u64 best) {
        const bool want = static_cast<long double>(current) < 0.999L * best;
        bad += gp::below_fraction(current, best, fraction) != want;
        ++checked;
    };
    for (gp::u64 best : {0ULL, 1ULL, 2ULL, 999ULL, 1000ULL, 1001ULL, 1ULL << 32, 1ULL << 63, ~0ULL})
        for (gp::u64 current : {0ULL, 1ULL, 998ULL, 999ULL, 1000ULL, 1ULL << 32, ~0ULL - 1, ~0ULL}) check(current, best);
    for (int i = 0; i < 2000000; ++i) {
        const gp::u64 best = rng() >> (rng() % 64);
        const gp::u64 edge = static_cast<gp::u64>(0.999L * best);   // where the answer turns
        check(edge - 1 + rng() % 3, best);
        check(rng() >> (rng() % 64), best);
    }
    std::printf("%ld checked, %ld differ\n", checked, bad);
    return bad != 0;
}
