// The fixed-point corner forces (v.1.1_gb300/csrc/msx_fixed.cuh) compiled for the
// host, over arrays of tets: X, u and f hold [tet][node][component].  taken[k]
// tells whether the element kernel would use the fixed-point form for tet k.
#include "../v.1.1_gb300/csrc/msx_fixed.cuh"

using namespace msx;

static void edges(const double *X, double *E)
{
    for (int b = 0; b < 3; b++)
        for (int i = 0; i < 3; i++) E[3 * b + i] = X[3 * (b + 1) + i] - X[i];
}

static void nodes(const double *u, double (*ua)[3])
{
    for (int a = 0; a < 4; a++)
        for (int i = 0; i < 3; i++) ua[a][i] = u[3 * a + i];
}

static void store(const FixedElem &q, const int64_t *f, double *out)
{
    for (int i = 0; i < 3; i++) {
        double s = 0;
        for (int a = 0; a < 3; a++) s += out[3 * (a + 1) + i] = std::ldexp((double)f[3 * a + i], q.x0 - q.lw[a]);
        out[i] = -s;
    }
}

extern "C" void fixed_cnh(long long n, const double *X, const double *u, double lambda, double mu, double *f, int *taken)
{
    int64_t kq[kFixTerms];
    int ks;
    fixed_series(lambda, mu, kq, &ks);
    const double ksw = 0.166666666667 * std::ldexp(1.0, ks);
    for (long long k = 0; k < n; k++) {
        FixedElem q;
        double E[9], ua[4][3];
        Limbs nb[9];
        int moved;
        int64_t fi[9];
        edges(X + 12 * k, E);
        nodes(u + 12 * k, ua);
        const auto scalar = [&](double J) {
            return J > 0 ? (int64_t)std::fmin((mu - lambda * std::log(J)) * ksw / J, 0x1p62) : INT64_MAX;
        };
        taken[k] = fixed_setup(E, kq[0], ks, q) && fixed_edges(q, ua, nb, moved) && fixed_forces(q, nb, kq, scalar, fi);
        if (taken[k]) store(q, fi, f + 12 * k);
    }
}

extern "C" void fixed_svk(long long n, const double *X, const double *u, int linear, double lambda, double mu2, double *f,
                          int *taken)
{
    int64_t kq;
    int ks;
    fixed_kappa(mu2, lambda, &kq, &ks);
    for (long long k = 0; k < n; k++) {
        FixedElem q;
        double E[9], ua[4][3];
        Limbs du[9];
        int moved;
        int64_t fi[9];
        edges(X + 12 * k, E);
        nodes(u + 12 * k, ua);
        taken[k] = fixed_setup_svk(E, 0.5 * mu2, ks, q) && fixed_edges<true>(q, ua, du, moved) &&
                   fixed_forces_svk(q, du, linear != 0, kq, ks, fi);
        if (taken[k]) store(q, fi, f + 12 * k);
    }
}
