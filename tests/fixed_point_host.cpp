// The fixed-point corner forces (v.1.1_gb300/csrc/msx_fixed.cuh) compiled for the
// host, over arrays of tets: X, u and f hold [tet][node][component].  taken[k]
// tells whether the element kernel would use the fixed-point form for tet k.
#include <algorithm>

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
        int s = 0, hi = 0;
        int64_t fi[9];
        edges(X + 12 * k, E);
        nodes(u + 12 * k, ua);
        double x[9];
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) {
                x[3 * a + i] = ua[a + 1][i] - ua[0][i];
                hi = std::max(hi, (int)(double_bits(std::fabs(x[3 * a + i])) >> 32));
            }
        taken[k] = fixed_setup_svk(E, 0.5 * mu2, ks, q) && fixed_motion(q, x, hi, linear != 0, du, s) &&
                   fixed_forces_svk(q, du, linear != 0, kq, ks, fi, s);
        q.x0 += s;
        if (taken[k]) store(q, fi, f + 12 * k);
    }
}

// The same corner forces in FP64, as the plain FP64 mode computes them for the
// elements that fixed point leaves out: law 2 St-Venant-Kirchhoff, 3 linear elastic.
extern "C" void fp64_svk(long long n, const double *X, const double *u, int linear, double lambda, double mu2, double *f)
{
    for (long long k = 0; k < n; k++) {
        double E[9], ua[4][3], G[9], F[9], P[9], du[9];
        edges(X + 12 * k, E);
        nodes(u + 12 * k, ua);
        double c[9];
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) {
                const double *p = E + 3 * ((a + 1) % 3), *q = E + 3 * ((a + 2) % 3);
                c[3 * a + i] = p[(i + 1) % 3] * q[(i + 2) % 3] - p[(i + 2) % 3] * q[(i + 1) % 3];
            }
        const double det = E[0] * c[0] + E[1] * c[1] + E[2] * c[2], wJ = 0.166666666667 * std::fabs(det);
        for (int j = 0; j < 9; j++) G[j] = c[j] / det;
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) du[3 * a + i] = ua[a + 1][i] - ua[0][i];
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++)
                F[3 * i + j] = std::fma(du[i], G[j], std::fma(du[3 + i], G[3 + j],
                                        i == j ? std::fma(du[6 + i], G[6 + j], 1.0) : du[6 + i] * G[6 + j]));
        if (linear) {
            const double h = mu2 * wJ, e0 = F[0] - 1.0, e1 = F[4] - 1.0, e2 = F[8] - 1.0, dg = lambda * ((e0 + e1) + e2) * wJ;
            P[0] = std::fma(h, e0, dg);
            P[4] = std::fma(h, e1, dg);
            P[8] = std::fma(h, e2, dg);
            P[1] = P[3] = 0.5 * h * (F[1] + F[3]);
            P[2] = P[6] = 0.5 * h * (F[2] + F[6]);
            P[5] = P[7] = 0.5 * h * (F[5] + F[7]);
        } else {
            double C[9], S[9];
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++)
                    C[3 * i + j] = std::fma(F[6 + i], F[6 + j], std::fma(F[i], F[j], F[3 + i] * F[3 + j]));
            const double tr = 0.5 * ((C[0] - 1.0) + (C[4] - 1.0) + (C[8] - 1.0)), h = 0.5 * mu2 * wJ, dg = lambda * tr * wJ;
            for (int j = 0; j < 9; j++) S[j] = j % 4 ? h * C[j] : std::fma(h, C[j] - 1.0, dg);
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++)
                    P[3 * i + j] = std::fma(F[3 * i + 2], S[6 + j], std::fma(F[3 * i], S[j], F[3 * i + 1] * S[3 + j]));
        }
        double *o = f + 12 * k;
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++)
                o[3 * (a + 1) + i] = std::fma(P[3 * i + 2], G[3 * a + 2], std::fma(P[3 * i], G[3 * a], P[3 * i + 1] * G[3 * a + 1]));
        for (int i = 0; i < 3; i++) o[i] = -(o[3 + i] + o[6 + i] + o[9 + i]);
    }
}

// Compressible neo-Hookean from the deformed edges, e_b = E_b + (u_b - u_0)
extern "C" void fp64_cnh(long long n, const double *X, const double *u, double lambda, double mu, double *f)
{
    for (long long k = 0; k < n; k++) {
        double E[9], ua[4][3], e[9], c[9], C[9], M[9];
        edges(X + 12 * k, E);
        nodes(u + 12 * k, ua);
        for (int b = 0; b < 3; b++)
            for (int i = 0; i < 3; i++) e[3 * b + i] = E[3 * b + i] + (ua[b + 1][i] - ua[0][i]);
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) {
                const int p = 3 * ((a + 1) % 3), q = 3 * ((a + 2) % 3), y = (i + 1) % 3, z = (i + 2) % 3;
                C[3 * a + i] = std::fma(E[p + y], E[q + z], -(E[p + z] * E[q + y]));
                c[3 * a + i] = std::fma(e[p + y], e[q + z], -(e[p + z] * e[q + y]));
            }
        const double D0 = std::fma(E[2], C[2], std::fma(E[0], C[0], E[1] * C[1])),
                     D = std::fma(e[2], c[2], std::fma(e[0], c[0], e[1] * c[1]));
        for (int j = 0; j < 9; j++) C[j] /= D0;
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++)
                M[3 * a + b] = std::fma(C[3 * a + 2], C[3 * b + 2], std::fma(C[3 * a], C[3 * b], C[3 * a + 1] * C[3 * b + 1]));
        const double wJ = 0.166666666667 * std::fabs(D0), J = D * (1.0 / D0), c1 = mu * wJ, c2 = (lambda * std::log(J) - mu) * (wJ / D);
        double *o = f + 12 * k;
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) {
                const double Fg = std::fma(e[6 + i], M[3 * a + 2], std::fma(e[i], M[3 * a], e[3 + i] * M[3 * a + 1]));
                o[3 * (a + 1) + i] = std::fma(c1, Fg, c2 * c[3 * a + i]);
            }
        for (int i = 0; i < 3; i++) o[i] = -(o[3 + i] + o[6 + i] + o[9 + i]);
    }
}

extern "C" double to_fp64(long long x, int k) { return fixed_to_fp64(x, k); }
