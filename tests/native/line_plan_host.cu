// Host-side check of the radix plans of tr_lines_part.cuh and of their register butterflies.
// Prints, for each supported length, its threads and radices, and for each further radix and both
// directions the inputs and outputs of Dft<R>::run.  Built by nvcc as a plain host program.
#include <cmath>
#include <cstdio>

#include "tr_lines_part.cuh"

template <int R>
static void check() {
    for (int inv = 0; inv < 2; ++inv) {
        float2 v[R];
        for (int n = 0; n < R; ++n) v[n] = make_float2(std::sin(1.3f * n + R), std::cos(0.7f * n * R + 0.1f));
        std::printf("R %d %d\n", R, inv);
        for (int n = 0; n < R; ++n) std::printf("%.9g %.9g\n", v[n].x, v[n].y);
        tr::Dft<R>::run(v, inv != 0);
        for (int n = 0; n < R; ++n) std::printf("%.9g %.9g\n", v[n].x, v[n].y);
    }
}

int main() {
    for (int L = 1; L <= 330; ++L)
        if (tr::lp_supported(L)) {
            std::printf("L %d %d", L, tr::lp_threads(L));
            for (int s = 0; s < tr::lp_stages(L); ++s) std::printf(" %d", tr::lp_radix(L, s));
            std::printf("\n");
        }
    check<6>();
    check<9>();
    check<12>();
    check<14>();
    check<15>();
    check<18>();
    check<21>();
    return 0;
}
