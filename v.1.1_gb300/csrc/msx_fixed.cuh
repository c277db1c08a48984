// msx_fixed.cuh -- corner forces of a tet in 64-bit fixed point: compressible
// neo-Hookean (here), St-Venant-Kirchhoff and linear elastic (fixed_setup_svk).
//
// The FP64 pipe of this GPU issues one warp instruction per scheduler in 64-80
// cycles, the integer pipes one in 1-2 (multiply-add of two 32-bit limbs into
// 64 bits: 2.2), so a product of two 60-bit numbers in three limb products
// costs a tenth of an FP64 product and carries more bits.  With e_b the
// deformed edges, g_a the gradients of shape functions 1..3, J = det e / det E
// and W = 0.166666666667 the quadrature weight, the corner forces are
//     f_a = S_a1 e_1 + S_a2 e_2 + S_a3 e_3 + c2 (e_c x e_d),  f_0 = -(f_1 + f_2 + f_3),
//     S_ab = W |det E| mu g_a.g_b,   c2 = -W (mu - lambda ln J) / J:
// sums of products of numbers whose size the reference element tells.  Each
// edge has its own power-of-two unit w_b, so accuracy does not depend on the
// element's aspect ratio: with e_b = w_b n_b and row a scaled by w_a,
//     f_a w_a = sum_b (S_ab w_a w_b) n_b + (c2 w_1 w_2 w_3) (n_c x n_d)
// has one unit for the nine products of a kind.
//
// Sizes.  |E_b| < 2^57 w_b, components of n_b below 2^58 - 2^32 (a stretch of two
// at least); cross products in units of 2^57, below 2^60 - 2^34; S below 2^57 and c2
// below 2^59; sums of a force in units of 2^58, below 2^61.3.  Numbers are split into a high and a signed 29-bit low limb,
// whose products fit 64-bit accumulators.  Products of two low limbs are left
// out; with the final shifts that drops half a unit of 2^-55 to 2^-56 of the
// products summed, less than the FP64 sum it replaces rounds.  An element that
// leaves these sizes is left to the FP64 arithmetic of its caller.
//
// Integer C that also compiles for the host.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define MSX_HD __host__ __device__ __forceinline__
#else
#define MSX_HD inline
#endif

namespace msx {

constexpr int kFixTerms = 16;   // coefficients of c2's series in 1 - J: |1 - J| < 2^-4
constexpr int kFixShort = 9;    // those that |1 - J| < 2^-7 needs
// A tet of det E >= kFixFlat |E_1||E_2||E_3| (0.41 for the six tets of a cube):
// in flatter ones the truncations of the cross products grow towards FP64's
// rounding.  Corner-force error against quad precision over that of the same
// formulas in FP64, 5000 random tets a case, nu 0 to 0.49, strains to 3 %: 0.3
// to 0.5 (0.05 undeformed) above 0.25, 0.4 to 0.8 around 0.15, 1.1 at 0.06.
constexpr double kFixFlat = 0.12;
constexpr int kFixMotionLeast = 64;   // exponent field of a motion that fixed_motion takes

struct Limbs {
    int32_t h, l;   // h 2^29 + l, |l| <= 2^28
};

MSX_HD Limbs limbs(int64_t x)
{
    return {(int32_t)((x + (1 << 28)) >> 29), (int32_t)((uint32_t)x << 3) >> 3};
}

MSX_HD Limbs limbs_neg(Limbs a) { return {-a.h, -a.l}; }

// a b = hh 2^58 + mid 2^29 + a.l b.l, summed without the last
MSX_HD int64_t mad_wide(int32_t a, int32_t b, int64_t c)
{
#ifdef __CUDA_ARCH__
    int64_t r;   // spelled out: from C the compiler splits many of these into a product and an addition
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return (int64_t)a * b + c;
#endif
}

MSX_HD void mac(int64_t &hh, int64_t &mid, Limbs a, Limbs b)
{
    hh = mad_wide(a.h, b.h, hh);
    mid = mad_wide(a.h, b.l, mid);
    mid = mad_wide(a.l, b.h, mid);
}

// hh 2^58 + mid 2^29 in units of 2^(58 - k), rounded to nearest when mid began
// at mac_half(k)
MSX_HD int64_t mac_sum(int64_t hh, int64_t mid, int k) { return (int64_t)((uint64_t)hh << k) + (mid >> (29 - k)); }
MSX_HD int64_t mac_half(int k) { return 1 << (28 - k); }

MSX_HD int64_t mulhi64(int64_t a, int64_t b)
{
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}

// a b 2^-64 to two units, for the series (a = h 2^32 + 2 l with l >= 0, h = a >> 32)
MSX_HD int64_t mulhi_near(int32_t h, int32_t l, int64_t b)
{
    const int32_t bh = (int32_t)(b >> 32), bl = (int32_t)((uint32_t)b >> 1);
    const int64_t t = mad_wide(l, bh, mad_wide(h, bl, 0));
    return mad_wide(h, bh, t >> 31);
}

MSX_HD uint32_t abs32(int32_t x)   // 2^31 for -2^31
{
#ifdef __CUDA_ARCH__
    return (uint32_t)abs(x);   // one instruction; with shift and exclusive or 2 % off a step of 6M tets
#else
    return x < 0 ? 0u - (uint32_t)x : (uint32_t)x;
#endif
}

MSX_HD int top_bit_u(uint64_t x)   // floor(log2 x), x > 0
{
#ifdef __CUDA_ARCH__
    return 63 - __clzll((long long)x);
#else
    return 63 - __builtin_clzll((unsigned long long)x);
#endif
}

MSX_HD int top_bit(int64_t x) { return top_bit_u((uint64_t)x); }

MSX_HD uint64_t double_bits(double x)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
#endif
}

MSX_HD double bits_double(uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}

MSX_HD double pow2_double(int k)   // 2^k, -1022 <= k <= 1023
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)(k + 1023) << 52);
#else
    return ldexp(1.0, k);
#endif
}

MSX_HD uint64_t shr64(uint64_t x, int s)   // zero for s < 0 and s > 63
{
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
#else
    return (unsigned)s > 63 ? 0 : x >> s;
#endif
}

// The fixed-point value of x in units of 2^lw, truncated toward zero: |x| < 2^62
// 2^lw.
MSX_HD int64_t fixed_from(double x, int lw)
{
    const uint64_t v = double_bits(x);
    const uint32_t hi = (uint32_t)(v >> 32);
    const int ex = (int)((hi >> 20) & 0x7FFu);
    const uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | 0x100000u) << 32 | (uint32_t)v) << 9;   // below 2^62
    const int64_t sg = (int64_t)((int32_t)hi >> 31);
    return ((int64_t)shr64(m, lw + (1075 + 9) - ex) ^ sg) - sg;
}

// x 2^k rounded to nearest (halves away from zero), on the integer pipes (a
// conversion takes the FP64 pipe as long as a product): the result has to be a
// normal number or zero.
MSX_HD double fixed_to_fp64(int64_t x, int k)
{
    const uint64_t m = x < 0 ? 0 - (uint64_t)x : (uint64_t)x;
    if (m == 0) return 0.0;
    const int lead = 63 - top_bit_u(m);
    const uint64_t v = m << lead;
    const uint64_t b = ((uint64_t)(1085 - lead + k) << 52) + (v >> 11) + ((v >> 10) & 1);
    return bits_double(b | (x < 0 ? 1ull << 63 : 0));
}

// c = n_a x n_b in units of 2^57
MSX_HD void fixed_cross(const Limbs *a, const Limbs *b, int64_t *c)
{
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        int64_t hh = 0, mid = mac_half(1);
        mac(hh, mid, a[j], b[k]);
        mac(hh, mid, limbs_neg(a[k]), b[j]);
        c[i] = mac_sum(hh, mid, 1);
    }
}

// n_1 . (n_2 x n_3) in units of 2^(57 + 57); cr: the limbs of the cross product
MSX_HD int64_t fixed_det(const Limbs *n1, const Limbs *cr)
{
    int64_t hh = 0, mid = mac_half(1);
#pragma unroll
    for (int i = 0; i < 3; i++) mac(hh, mid, n1[i], cr[i]);
    return mac_sum(hh, mid, 1);
}

// The element's static data: the reference edges E_b in units of the smallest
// w (with half a unit of w_b added, so that the shift to w_b rounds to nearest);
// S_ab w_a w_b 2^t (in the order 11 12 13 22 23 33); det E as fixed_det gives
// it; 2^(62 + ds) / det E for ds = floor(log2 det E); exponents.
struct FixedElem {
    int64_t E[9];
    Limbs S[6];
    int64_t d0, rd;
    int32_t lw[3];   // log2 w_b
    int32_t x0;      // log2 of f_a's unit = x0 - lw_a
    int32_t cs;      // c2's series (MatParams::kq) << cs is c2 w_1 w_2 w_3 2^(57 + t); StVK: headroom hr and gradient unit gs, hr | gs << 2
    int32_t ds;
};

MSX_HD int fixed_lw_min(const FixedElem &q)
{
    const int a = q.lw[0] < q.lw[1] ? q.lw[0] : q.lw[1];
    return a < q.lw[2] ? a : q.lw[2];
}

// The exponents as two words in device memory.  A zero first word (ds is at
// least 40) sends the element to FP64.
MSX_HD void fixed_pack(const FixedElem &q, uint32_t *w)
{
    w[0] = (uint32_t)q.ds | (uint32_t)(q.cs + 32) << 6 | (uint32_t)(q.lw[0] + 2048) << 12;
    w[1] = (uint32_t)(q.lw[1] - q.lw[0] + 64) | (uint32_t)(q.lw[2] - q.lw[0] + 64) << 7 | (uint32_t)(q.x0 + 4096) << 14;
}

MSX_HD void fixed_unpack(uint32_t w0, uint32_t w1, FixedElem &q)
{
    q.ds = (int)(w0 & 63u);
    q.cs = (int)((w0 >> 6) & 63u) - 32;
    q.lw[0] = (int)(w0 >> 12) - 2048;
    q.lw[1] = q.lw[0] + (int)(w1 & 127u) - 64;
    q.lw[2] = q.lw[0] + (int)((w1 >> 7) & 127u) - 64;
    q.x0 = (int)(w1 >> 14) - 4096;
}

// The deformed edges n_b = (E_b + u_b - u_0) / w_b in limbs, exact up to the
// final rounding and the bits of u below the smallest w; false for a component
// of 2^58 - 2^32 and more (judged before limbs(), whose high half is the value
// modulo 2^61), a motion of 2^62 of the smallest w and more, infinities and NaN.
// Displacements beyond 2^62 of the smallest w
// (32 edge lengths at least) are taken in a unit 2^k times larger, whose lost
// bits lie 2^-9 below u's own last one.  moved: an upper bound of
// max |u_b - u_0| component by component, in units of 2^32 of the smallest w.
MSX_HD bool fixed_edges(const FixedElem &q, const double (*u)[3], Limbs *n, int &moved)
{
    const int lw = fixed_lw_min(q);
    int emax = 0;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int ex = (int)((double_bits(u[a][i]) >> 52) & 0x7FF);
            emax = emax > ex ? emax : ex;
        }
    int k = emax - (lw + 1075 + 9);   // 2^k 2^lw is the unit of u
    k = k > 0 ? k : 0;
    if (k > 40) return false;
    int64_t U[4][3];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int i = 0; i < 3; i++) U[a][i] = fixed_from(u[a][i], lw + k);
    if (k > 0) {   // back to units of 2^lw, as differences (the common part of a far motion is gone)
        bool far = false;
#pragma unroll
        for (int i = 0; i < 3; i++) {
#pragma unroll
            for (int b = 1; b < 4; b++) {
                const int64_t d = U[b][i] - U[0][i];
                far = far || d >= (1LL << (60 - k)) || d <= -(1LL << (60 - k));
                U[b][i] = (int64_t)((uint64_t)d << k);
            }
            U[0][i] = 0;
        }
        if (far) return false;
    }
    uint32_t m = 0, most = 0;
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const int d = q.lw[b] - lw;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int64_t du = U[b + 1][i] - U[0][i];
            const uint32_t da = abs32((int)(du >> 32));
            m = m > da ? m : da;
            const int64_t x = (int64_t)((uint64_t)q.E[3 * b + i] + (uint64_t)du) >> d;
            const uint32_t xa = abs32((int)(x >> 32));
            most = most > xa ? most : xa;
            n[3 * b + i] = limbs(x);
        }
    }
    moved = m < (1u << 30) ? (int)m + 1 : 1 << 30;
    return m < (1u << 30) && most < (1u << 26) - 1;
}

// Corner forces f_1..f_3 (f[3(a-1) + i]) as integers in units of
// 2^(x0 - lw_a); false when the element leaves the sizes above.  n: the deformed
// edges (fixed_edges); kq: c2's series.  scalar(J) gives -c2 in kq's units for
// |1 - J| >= 2^-4, in FP64.  f_0 = -(f_1 + f_2 + f_3) is left to the caller, in
// FP64: its rounding to nearest has no preferred sign (a sum of shifted integers
// has, and pushes the whole body).
template <typename SCALAR>
MSX_HD bool fixed_forces(const FixedElem &q, const Limbs *n, const int64_t *kq, SCALAR scalar, int64_t *f)
{
    Limbs cr[9];   // cr_1 = n_2 x n_3, cr_2 = n_3 x n_1, cr_3 = n_1 x n_2
#pragma unroll
    for (int a = 0; a < 3; a++) {
        int64_t c[3];
        fixed_cross(n + 3 * ((a + 1) % 3), n + 3 * ((a + 2) % 3), c);
#pragma unroll
        for (int i = 0; i < 3; i++) cr[3 * a + i] = limbs(c[i]);
    }
    const int64_t D = fixed_det(n, cr);
    const int64_t y = q.d0 - D;   // d0 (1 - J)
    int64_t c2;
    if (y < (q.d0 >> 4) && y > -(q.d0 >> 4)) {
        const int64_t ys = (int64_t)((uint64_t)y << (66 - q.ds));
        const int64_t yq = mulhi_near((int32_t)(ys >> 32), (int32_t)((uint32_t)ys >> 1), q.rd);   // (1 - J) 2^64
        const int32_t yh = (int32_t)(yq >> 32), yl = (int32_t)((uint32_t)yq >> 1);
        const bool near1 = yq < (1LL << 57) && yq > -(1LL << 57);
        c2 = near1 ? kq[kFixShort - 1] : kq[kFixTerms - 1];
        if (!near1)
#pragma unroll
            for (int k = kFixTerms - 2; k >= kFixShort - 1; k--) c2 = kq[k] + mulhi_near(yh, yl, c2);
#pragma unroll
        for (int k = kFixShort - 2; k >= 0; k--) c2 = kq[k] + mulhi_near(yh, yl, c2);
    } else {
        c2 = scalar(1.0 - (double)y / (double)q.d0);
    }
    const int64_t most = q.cs >= 0 ? (1LL << 59) >> q.cs : (q.cs > -3 ? (1LL << 59) << -q.cs : INT64_MAX);
    if (c2 >= most || c2 <= -most) return false;
    c2 = q.cs >= 0 ? (int64_t)((uint64_t)c2 << q.cs) : c2 >> -q.cs;
    const Limbs lc = limbs(-c2);
    const int mi[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            int64_t hh = 0, mid = mac_half(0);
            mac(hh, mid, lc, cr[3 * a + i]);
#pragma unroll
            for (int b = 0; b < 3; b++) mac(hh, mid, q.S[mi[a * 3 + b]], n[3 * b + i]);
            f[3 * a + i] = mac_sum(hh, mid, 0);
        }
    return true;
}

// ds and rd = 2^(62 + ds) / d0: the FP64 quotient, corrected once
MSX_HD void fixed_reciprocal(FixedElem &q)
{
    q.ds = top_bit(q.d0);
    q.rd = (int64_t)(0x1p62 / ((double)q.d0 * pow2_double(-q.ds)));
    const __int128 res = ((__int128)1 << (62 + q.ds)) - (__int128)q.rd * q.d0;   // below 2^66
    q.rd += mulhi64((int64_t)(res >> 8), q.rd) >> (q.ds - 10);
}

// The static data from the reference edges E (E[3(b-1) + i]), the law's c2
// series' first coefficient kq0 and exponent ks (fixed_series).  With the
// integers of the reference element itself, n_a x n_b as c_a and det E as d0,
//     S_ab w_a w_b = W mu w_1 w_2 w_3 (c_a . c_b) / d0,
// so S and c2 carry the same truncations of the cross products and cancel to
// the last bits in the undeformed state.  false: the element is left to FP64 (a
// non-positive volume, too flat an element, numbers near the ends of the FP64
// range).
MSX_HD bool fixed_setup(const double *E, int64_t kq0, int ks, FixedElem &q)
{
    Limbs n[9], cl[9];
    int64_t c[9], v[6], vm = 0;
    int sum = 0;
    double vol = kFixFlat * kFixFlat;
    for (int b = 0; b < 3; b++) {
        const double l2 = E[3 * b] * E[3 * b] + E[3 * b + 1] * E[3 * b + 1] + E[3 * b + 2] * E[3 * b + 2];
        if (!(l2 < 1e100) || !(l2 > 1e-100)) return false;
        const int ex2 = (int)(double_bits(l2) >> 52) - 1023;
        q.lw[b] = (ex2 >> 1) + 1 - 57;   // floor(log2 |E_b|) + 1 - 57
        sum += q.lw[b];
        vol *= l2 * pow2_double(-2 * q.lw[b]);
    }
    const int d1 = q.lw[1] - q.lw[0], d2 = q.lw[2] - q.lw[0];
    if (d1 < -4 || d1 > 4 || d2 < -4 || d2 > 4 || d2 - d1 < -4 || d2 - d1 > 4) return false;   // E fits 2^61 of the smallest w
    const int lw = fixed_lw_min(q);
    for (int b = 0; b < 3; b++)
        for (int i = 0; i < 3; i++) {
            const int d = q.lw[b] - lw;
            q.E[3 * b + i] = fixed_from(E[3 * b + i], lw) + (d ? 1LL << (d - 1) : 0);
            n[3 * b + i] = limbs(q.E[3 * b + i] >> d);
        }
    for (int a = 0; a < 3; a++) {
        fixed_cross(n + 3 * ((a + 1) % 3), n + 3 * ((a + 2) % 3), c + 3 * a);
        for (int i = 0; i < 3; i++) cl[3 * a + i] = limbs(c[3 * a + i]);
    }
    q.d0 = fixed_det(n, cl);
    const double det = (double)q.d0 * 0x1p114;
    if (q.d0 < (1LL << 48) || q.d0 >= (1LL << 62) || !(det * det >= vol)) return false;
    fixed_reciprocal(q);
    __int128 dot[6], dm = 0;
    int k = 0;
    for (int a = 0; a < 3; a++)
        for (int b = a; b < 3; b++, k++) {
            dot[k] = (__int128)c[3 * a] * c[3 * b] + (__int128)c[3 * a + 1] * c[3 * b + 1] +
                     (__int128)c[3 * a + 2] * c[3 * b + 2];
            if (a == b && dot[k] > dm) dm = dot[k];   // the largest is on the diagonal
        }
    const int64_t dh = (int64_t)(dm >> 56);   // below 2^62
    if (dh < 1) return false;
    const int cs = 56 + top_bit(dh) - 61;   // dot >> cs below 2^62
    for (k = 0; k < 6; k++) {
        v[k] = mulhi64((int64_t)(dot[k] >> cs), q.rd);   // (c_a . c_b / 2^cs) / d0 2^(ds - 2)
        const int64_t m = v[k] < 0 ? -v[k] : v[k];
        vm = vm > m ? vm : m;
    }
    if (kq0 < (1LL << 32) || vm < (1LL << 32)) return false;
    if (vm >= (1LL << 62)) return false;
    const int z = 61 - top_bit(kq0), kv = 61 - top_bit(vm), kc = kv - cs + 56;   // kq0 and the largest v to [2^61, 2^62)
    // S_ab w_a w_b 2^t = mulhi(kq0 << z, v << kv) >> sh, below 2^57, and
    // kq0 << cs = c2 w_1 w_2 w_3 2^(57 + t) at J = 1, below 2^57 too
    const int64_t top = mulhi64(kq0 << z, vm << kv);   // below 2^60
    int sh = top >= (1LL << 59) ? 3 : (top >= (1LL << 58) ? 2 : 1);
    if (q.ds + kc - 60 > sh) sh = q.ds + kc - 60;
    const int t = ks + z - sum - 122 + q.ds + kc - sh;
    for (k = 0; k < 6; k++)
        q.S[k] = limbs((mulhi64(kq0 << z, (int64_t)((uint64_t)v[k] << kv)) + (1LL << (sh - 1))) >> sh);
    q.x0 = 58 - t;
    q.cs = -ks + sum + 57 + t;
    if (sh > 20 || q.cs < -31 || q.cs > 20) return false;
    const int lmax = q.lw[0] + (d1 > d2 ? (d1 > 0 ? d1 : 0) : (d2 > 0 ? d2 : 0));
    const int lmin = q.lw[0] + (d1 < d2 ? (d1 < 0 ? d1 : 0) : (d2 < 0 ? d2 : 0));
    return q.x0 - lmin <= 900 && q.x0 - lmax >= -900;   // forces stay normal FP64 numbers
}

// St-Venant-Kirchhoff and linear elasticity: the displacement gradient and the
// stress in the axes of space, as in FP64 (products of the edges would lose
// accuracy with the square of an element's flatness).  With the shape
// functions' gradients g_a, one unit w for all three edges, and a unit 2^s for
// the strain that follows from the largest |u_b - u_0| (a state of strain 1e-9
// has all its bits; in linear elasticity it also grows with the motion), a unit
// 2^gs for flat elements' gradients, du_b = (u_b - u_0) / (w 2^(s - gs)) and
// f_a = f_a' 2^(s + gs) |det E| W mu / w:
//     H = sum_b du_b (w g_b / 2^gs),  G = H + H^T + 2^s H^T H (linear: without H^T H),
//     S = scale (G + kappa tr(G) I),  kappa = lambda / (2 mu),
//     P = S + 2^s H S (linear: S),  f_a' = P (w g_a / 2^gs),
// where scale 2^(x0 - gs) w = |det E| W mu, 1/2 <= scale < 1.  Units: du 2^-57, w g
// 2^-111, H to P 2^-55, scale 2^-57, du so small that |H| < 2^57 (by hr bits).
// G and what follows it take a unit 2^t larger where kappa tr(G) asks for it.
// An error of one unit in H, S or P is 2^-55 of the largest of them, against
// 2^-53 of 1 for F's diagonal in FP64, whatever the strain.  Corner-force error
// against extended precision over that of the FP64 form, grids of hexes of
// 1:1:0.4 to 1:1:3, six tets each, jittered and not, nu 0 to 0.49, strains 1e-14
// to 0.3: median 0.002 (linear) and 0.0004; above 1 only where both are below 1.5
// roundings of the result (grids whose sides are powers of two, on which FP64's
// own products can be exact) or, to 1.3, at strains of 0.3.  One StVK step of 264,000 shuffled
// tets: 64.7 us, 63.0 with a unit set by the element alone, whose error at a
// shear of 1e-5 on a cubic grid was 8,700 (linear) and 4.4 times FP64's.  With
// products of edges instead, E_b . E_c and their metric, the error is 2 to 8
// times FP64's on cubes and grows with the square of the flatness.  E holds w g
// in limbs, S[0] the scale, both rounded from 128-bit products.  gs up to 7
// takes hexes down to 1:1:0.02; without it (w g below 8 / |E| alone) hexes
// flatter than 1:1:0.2 went to FP64: 1M jittered tets of 1:1:0.2, StVK, 140 us a
// step, 348 without, 308 with all elements in FP64.
MSX_HD int64_t limbs_pack(Limbs x) { return (int64_t)((uint64_t)(uint32_t)x.h << 32 | (uint32_t)x.l); }
MSX_HD Limbs limbs_unpack(int64_t x) { return {(int32_t)(x >> 32), (int32_t)x}; }

// kappa as kq 2^(ks - 57) with |kappa| < 2^ks, in limbs; ks < 0 where there is none
inline void fixed_kappa(double mu2, double lambda, int64_t *kq, int *ks)
{
    const double kappa = lambda / mu2;
    *kq = 0;
    *ks = -1;
    if (!(mu2 > 0) || !(std::fabs(kappa) < 0x1p20)) return;
    *ks = 0;
    while (std::fabs(kappa) >= std::ldexp(1.0, *ks)) ++*ks;
    *kq = limbs_pack(limbs((int64_t)std::rint(std::ldexp(kappa, 57 - *ks))));
}

// false: the element is left to FP64 (see fixed_setup; w g beyond 2^7 times 4 to 8)
MSX_HD bool fixed_setup_svk(const double *E, double mu, int ks, FixedElem &q)
{
    int64_t n[9], c[9];
    double l2 = 0;
    for (int b = 0; b < 3; b++) {
        const double x = E[3 * b] * E[3 * b] + E[3 * b + 1] * E[3 * b + 1] + E[3 * b + 2] * E[3 * b + 2];
        if (!(x < 1e100) || !(x > 1e-100)) return false;
        l2 = l2 > x ? l2 : x;
    }
    const int lw = (((int)(double_bits(l2) >> 52) - 1023) >> 1) + 1 - 57;
    q.lw[0] = q.lw[1] = q.lw[2] = lw;
    // edges in units of w 2^-5 and cross products of w^2 2^51, below 2^62 and 2^63; det E of w^3 2^46
    for (int k = 0; k < 9; k++) n[k] = fixed_from(E[k], lw - 5);
    __int128 det = 0;
    for (int a = 0; a < 3; a++)
        for (int i = 0; i < 3; i++) {
            const int64_t *p = n + 3 * ((a + 1) % 3), *r = n + 3 * ((a + 2) % 3);
            const int y = (i + 1) % 3, z = (i + 2) % 3;
            c[3 * a + i] = (int64_t)(((__int128)p[y] * r[z] - (__int128)p[z] * r[y] + ((__int128)1 << 60)) >> 61);
            if (a == 0) det += (__int128)n[i] * c[i];
        }
    // det E = d0 2^dx w^3, d0 of 62 bits
    const int64_t dh = (int64_t)(det >> 63);
    if (dh < (1LL << 40)) return false;   // below 2^-21 |E|^3 (or not positive)
    const int down = top_bit(dh) + 2, dx = down + 46;
    q.d0 = (int64_t)(det >> down);
    fixed_reciprocal(q);
    // w g = c 2^51 / (d0 2^dx) = c rd 2^-sh in units of 2^-111; 2^gs times larger where that leaves 2^57
    const int sh = 62 + q.ds + dx - 51 - 111;
    int gs = 0;
    for (int k = 0; k < 9; k++) {
        const int64_t a = mulhi64(c[k] < 0 ? -c[k] : c[k], q.rd);
        const int over = a ? top_bit(a) + 64 - sh - 56 : 0;
        gs = over > gs ? over : gs;
    }
    if (gs > 7) return false;
    int64_t sum[3] = {0, 0, 0};
    for (int k = 0; k < 9; k++) {
        const int64_t g = (int64_t)(((__int128)c[k] * q.rd + ((__int128)1 << (sh + gs - 1))) >> (sh + gs));
        sum[k % 3] += g < 0 ? -g : g;
        q.E[k] = limbs_pack(limbs(g));
    }
    // |du| < 2^(57 - hr) makes |H| < 2^57: sum_b |w g_b| <= 2^(56 + hr), component by component
    int hr = 0;
    while (sum[0] > 1LL << (56 + hr) || sum[1] > 1LL << (56 + hr) || sum[2] > 1LL << (56 + hr)) hr++;
    q.cs = hr | gs << 2;   // at most 31
    // |det E| W mu = scale 2^x w^3, 1/2 <= scale < 1, to the scale's 57 bits
    if (ks < 0 || !(mu < 1e100) || !(mu > 1e-100)) return false;
    const int xm = (int)(double_bits(mu) >> 52) - 1022;
    const int64_t wm = (int64_t)(((__int128)fixed_from(0.166666666667, -64) * fixed_from(mu, xm - 62)) >> 62);
    const int64_t v = (int64_t)(((__int128)wm * (q.d0 << (62 - q.ds))) >> 62);   // W mu det E 2^(64 - xm - ds - dx) / w^3
    const int tv = top_bit(v);   // 59 to 62
    q.S[0] = limbs((v + (1LL << (tv - 57))) >> (tv - 56));
    q.x0 = tv + 1 - 64 + xm + q.ds + dx + 3 * lw - 109 + gs;
    return q.x0 - lw <= 900 && q.x0 - lw >= -900;
}

// x 2^-r rounded to nearest, 0 <= r <= 61, |x| < 2^62.9
MSX_HD int64_t shift_round(int64_t x, int r) { return (x + (int64_t)((1ull << r) >> 1)) >> r; }

MSX_HD int32_t high_word(int64_t x) { return (int32_t)(x >> 32); }

// The motion x[3(b-1) + i] = u_b - u_0 in limbs and the exponent s of H's unit; hi: the largest high word of |x|.  s <= 0 with H^T H, whose elements
// larger motions leave to FP64.  false: infinities, NaN, a motion beyond 2^58
// of w 2^-gs, forces near the ends of the FP64 range.
MSX_HD bool fixed_motion(const FixedElem &q, const double *x, int hi, bool linear, Limbs *du, int &s)
{
    if (hi < kFixMotionLeast << 20) {   // at rest, or nearly
        uint64_t any = 0;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            any |= double_bits(x[k]) << 1;
            du[k] = {0, 0};
        }
        s = 0;
        return any == 0;
    }
    const int e = (hi >> 20) - 1022;   // |x| < 2^e
    const int gs = q.cs >> 2;
    int lu = e - 57 + (linear ? 0 : q.cs & 3);
    if (!linear && lu > q.lw[0] - gs) lu = q.lw[0] - gs;
    s = lu - q.lw[0] + gs;
    const int unit = q.x0 + s - q.lw[0];
#pragma unroll
    for (int k = 0; k < 9; k++) du[k] = limbs(fixed_from(x[k], lu));
    return hi < 0x7FF << 20 && e - lu <= 58 && unit <= 870 && unit >= -870;
}

// Corner forces f_1..f_3 (f[3(a-1) + i]) as integers in units of
// 2^(x0 - lw + s), s as it returns; du, s: fixed_motion; kq, ks: fixed_kappa.
// false: beyond the sizes above.  Every bound is judged on 64-bit values.
MSX_HD bool fixed_forces_svk(const FixedElem &q, const Limbs *du, bool linear, int64_t kq, int ks, int64_t *f, int &s)
{
    Limbs g[9], H[9], S[6];
    uint32_t out = 0;
    // the products of H, when there are any, go 2^r below G's unit; half of that unit begins their sums
    const int r = s < -61 ? 61 : -s;
    const int64_t half_hh = r > 36 ? 1LL << (r - 4) : 0, half_mid = r > 36 ? 0 : 1LL << (25 + r);
#pragma unroll
    for (int k = 0; k < 9; k++) g[k] = limbs_unpack(q.E[k]);
    int64_t h[9], G[6];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            int64_t hh = 0, mid = mac_half(2);
#pragma unroll
            for (int b = 0; b < 3; b++) mac(hh, mid, du[3 * b + i], g[3 * b + j]);
            h[3 * i + j] = mac_sum(hh, mid, 2);
            H[3 * i + j] = limbs(h[3 * i + j]);
            out |= (uint32_t)(high_word(h[3 * i + j]) + (1 << 25));   // 2^57
        }
    if (!linear && out >= (1u << 26)) return false;
    int k = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) G[k++] = h[3 * i + j] + h[3 * j + i];
    if (!linear) {
        k = 0;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = i; j < 3; j++) {
                int64_t hh = half_hh, mid = half_mid;
#pragma unroll
                for (int b = 0; b < 3; b++) mac(hh, mid, H[3 * b + i], H[3 * b + j]);
                G[k++] += mac_sum(hh, mid, 3) >> r;
            }
    } else {   // |H| < 2^(57 + cs): G to 2^58, by up to 25 bits where a spin cancelled in it
        uint32_t any = 1;
#pragma unroll
        for (k = 0; k < 6; k++) any |= abs32(high_word(G[k]));
        const int d = top_bit(any) - 25, right = d > 0 ? d : 0, left = right - d;
#pragma unroll
        for (k = 0; k < 6; k++) G[k] = (int64_t)((uint64_t)shift_round(G[k], right) << left);
        s += d;
    }
    const int64_t tr = G[0] + G[3] + G[5], ta = tr < 0 ? -tr : tr;
    if (ta >= (1LL << 60) - (1LL << 29)) return false;
    // kappa tr < 2^(ks + 1 + top bit of tr), below 2^57 in a unit 2^t larger; rounded to
    // nearest (a truncation is a pressure on every element of the body)
    int t = ta ? ks + top_bit(ta) - 56 : 0;
    t = t > 0 ? t : 0;
    const int kk = 1 + ks - t, kd = kk < 0 ? -kk : 0;   // kk >= -2
    int64_t th = 0, tm = 1LL << (28 - kk);
    mac(th, tm, limbs(tr), limbs_unpack(kq));
    const int64_t kt = mac_sum(th, tm, kk + kd) >> kd;
    if (t > 0) {
        s += t;
#pragma unroll
        for (k = 0; k < 6; k++) G[k] = shift_round(G[k], t);
    }
    out = 0;
#pragma unroll
    for (k = 0; k < 6; k++) {
        const int64_t x = G[k] + (k == 0 || k == 3 || k == 5 ? kt : 0);
        out |= (uint32_t)(high_word(x) + (1 << 27));   // 2^59
        int64_t hh = 0, mid = mac_half(1);
        mac(hh, mid, limbs(x), q.S[0]);
        G[k] = mac_sum(hh, mid, 1);
        S[k] = limbs(G[k]);
    }
    const int mi[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    Limbs P[9];
    if (linear) {
#pragma unroll
        for (k = 0; k < 9; k++) P[k] = S[mi[k]];
    } else {
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                int64_t hh = half_hh, mid = half_mid;
#pragma unroll
                for (int b = 0; b < 3; b++) mac(hh, mid, H[3 * i + b], S[mi[3 * b + j]]);
                const int64_t x = G[mi[3 * i + j]] + (mac_sum(hh, mid, 3) >> r);
                out |= (uint32_t)(high_word(x) + (1 << 27));
                P[3 * i + j] = limbs(x);
            }
    }
    if (out >= (1u << 28)) return false;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int i = 0; i < 3; i++) {
            int64_t hh = 0, mid = mac_half(1);
#pragma unroll
            for (int j = 0; j < 3; j++) mac(hh, mid, P[3 * i + j], g[3 * a + j]);
            f[3 * a + i] = mac_sum(hh, mid, 1);
        }
    return true;
}

// kq and ks of a material: (mu + lambda H_n) W 2^ks, n = 0..15 (H_n the harmonic
// numbers), as integers below 2^61.
inline void fixed_series(double lambda, double mu, int64_t *kq, int *ks)
{
    double c[kFixTerms], H = 0, big = 0;
    for (int n = 0; n < kFixTerms; n++) {
        if (n) H += 1.0 / n;
        c[n] = (mu + lambda * H) * 0.166666666667;
        if (std::fabs(c[n]) > big) big = std::fabs(c[n]);
    }
    *ks = 60 - std::ilogb(big);
    for (int n = 0; n < kFixTerms; n++) kq[n] = (int64_t)std::rint(std::ldexp(c[n], *ks));
}

}  // namespace msx
