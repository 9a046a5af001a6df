// sl3_near against the general retraction (host builds of fm_lie.cuh) over
// random G with ||G - I||_inf up to the given bound: prints the largest
// entry difference, and the largest one outside the few draws whose Newton
// stop test (residual 1e-12) falls on different sides.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "fm_lie.cuh"

using namespace fm::lie;

int main(int argc, char** argv) {
    const double lim = atof(argv[1]);
    const int n = argc > 2 ? atoi(argv[2]) : 20000;
    std::mt19937_64 g(1);
    std::normal_distribution<double> nd;
    std::uniform_real_distribution<double> U(0, 1);
    double worst = 0, inner = 0;
    int flips = 0;
    for (int t = 0; t < n; ++t) {
        M3 E;
        for (int i = 0; i < 9; ++i) E.a[i] = nd(g);
        if (t % 3 == 0) {  // rank one (simple shear among them)
            double u[3], v[3];
            for (int i = 0; i < 3; ++i) u[i] = nd(g), v[i] = nd(g);
            for (int i = 0; i < 9; ++i) E.a[i] = u[i % 3] * v[i / 3];
        }
        if (t % 7 == 0)  // axis-aligned compression
            for (int i = 0; i < 9; ++i) E.a[i] = (i % 4 == 0) ? -std::fabs(nd(g)) : 0.0;
        const double f = lim * (t % 2 ? 1.0 : U(g)) / inf_norm(E);
        M3 F;
        for (int i = 0; i < 9; ++i) F.a[i] = E.a[i] * f + (i % 4 == 0);
        if (!(inf_norm(sub(F, ident())) < kNear)) continue;
        const M3 A = sl3_retraction(F), B = sl3_near(F);
        double w = 0;
        for (int i = 0; i < 9; ++i) w = fmax(w, fabs(A.a[i] - B.a[i]));
        worst = fmax(worst, w);
        if (w > 2e-14) ++flips;
        else inner = fmax(inner, w);
    }
    std::printf("%.3e %.3e %d\n", worst, inner, flips);
    return 0;
}
