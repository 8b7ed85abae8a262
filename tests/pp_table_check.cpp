// Host check of md-force-routines_b200/csrc/p3m_pp_table.h: for every triple
// kappa alpha rc on the command line, the interval count the library takes (0:
// none) and the largest relative errors of psi and g = psi - r psi' between the
// points the builder looks at, against the closed form in extended precision.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "p3m_pp_table.h"

using namespace p3m;

static void closed_form(long double r, long double k, long double a, long double *psi, long double *g)
{
    const long double ep = expl(k * r) * erfcl(a * r + 0.5L * k / a), em = expl(-k * r) * erfcl(a * r - 0.5L * k / a);
    const long double gauss = expl(-a * a * r * r - 0.25L * k * k / (a * a));
    *psi = 0.5L * (ep + em);
    *g = 0.5L * (ep * (1.0L - k * r) + em * (1.0L + k * r)) +
         2.0L * a * r * gauss / sqrtl(3.141592653589793238462643383279502884L);
}

int main(int argc, char **argv)
{
    std::vector<double> tab(PP64_MAX_N * PP64_COEF);
    for (int c = 1; c + 2 < argc; c += 3) {
        const double kappa = atof(argv[c]), alpha = atof(argv[c + 1]), rc = atof(argv[c + 2]);
        int N = PP64_MIN_N;
        while (N <= PP64_MAX_N && !(build_pp_table64(kappa, alpha, rc, N, PP64_LIMIT, tab.data()) <= PP64_LIMIT)) N *= 2;
        if (N > PP64_MAX_N) {
            printf("0 0 0\n");
            continue;
        }
        double epsi = 0.0, eg = 0.0;
        const int points = 50021;
        for (int s = 0; s < points; ++s) {
            const long double t = N * (s + 0.5L) / points;
            const int i = (int)t;
            const long double u = t - (i + 0.5L);
            long double p = 0.0L, d = 0.0L, psi, g;
            for (int q = PP64_COEF - 1; q >= 0; --q) {
                d = d * u + p;
                p = p * u + tab[pp64_at(N, i, q)];
            }
            closed_form(t * ((long double)rc / N), kappa, alpha, &psi, &g);
            epsi = fmax(epsi, (double)(fabsl(p - psi) / psi));
            eg = fmax(eg, (double)(fabsl(p - t * d - g) / g));
        }
        printf("%d %.3e %.3e\n", N, epsi, eg);
    }
    return 0;
}
