// msx_device.cuh -- device code of the explicit C3D4 step.
//
// Included by one translation unit per numeric mode.  msx_exact.cu is built
// with --fmad=false and instantiates the reference-order kernels; msx_fast.cu
// is built with contraction on and instantiates the FP64 and mixed kernels.
#pragma once
#include <cfloat>
#include <cmath>
#include "msx_internal.h"

namespace msx {

#define MSX_INF_BITS 0x7FF0000000000000ULL

// ---------------------------------------------------------------------------
// Reference-order arithmetic (src/mathematics/maths.cpp, geometry.cpp and the
// laws).  These compile to plain mul/add only when contraction is off.
// ---------------------------------------------------------------------------
// maths.cpp:1564-1577 determinantTensor
__device__ __forceinline__ double det3_ref(const double *A)
{
    return A[0] * (A[4] * A[8] - A[7] * A[5]) - A[1] * (A[3] * A[8] - A[6] * A[5]) +
           A[2] * (A[3] * A[7] - A[6] * A[4]);
}

// maths.cpp:2749-2785 inverse
__device__ __forceinline__ void inv3_ref(const double *A, double *Ai)
{
    double idet = 1.0 / det3_ref(A);
    Ai[0] = idet * (A[4] * A[8] - A[5] * A[7]);
    Ai[3] = -idet * (A[3] * A[8] - A[5] * A[6]);
    Ai[6] = idet * (A[3] * A[7] - A[4] * A[6]);
    Ai[1] = -idet * (A[1] * A[8] - A[2] * A[7]);
    Ai[4] = idet * (A[0] * A[8] - A[2] * A[6]);
    Ai[7] = -idet * (A[0] * A[7] - A[1] * A[6]);
    Ai[2] = idet * (A[1] * A[5] - A[2] * A[4]);
    Ai[5] = -idet * (A[0] * A[5] - A[2] * A[3]);
    Ai[8] = idet * (A[0] * A[4] - A[1] * A[3]);
}

// geometry.cpp:90-136 areaTriangle (3D) of triangle (p, q, r): 0.5*|(p-r)x(q-r)|
__device__ __forceinline__ double area_tri_ref(const double *p, const double *q, const double *r)
{
    double A0 = p[0] - r[0], A1 = p[1] - r[1], A2 = p[2] - r[2];
    double B0 = q[0] - r[0], B1 = q[1] - r[1], B2 = q[2] - r[2];
    double C0 = A1 * B2 - A2 * B1;
    double C1 = A2 * B0 - A0 * B2;
    double C2 = A0 * B1 - A1 * B0;
    return 0.5 * sqrt(C0 * C0 + C1 * C1 + C2 * C2);
}

// geometry.cpp:264-301 inscribedSphere x 2 (classLinearTetrahedra.cpp:146-163);
// *det_edges (when given) receives the determinant of the edge rows p1-p0,
// p2-p0, p3-p0 that the volume comes from.
__device__ __forceinline__ double char_length_ref(const double *x, double *det_edges = nullptr)
{
    const double *p0 = x, *p1 = x + 3, *p2 = x + 6, *p3 = x + 9;
    double s1 = area_tri_ref(p0, p1, p2);
    double s2 = area_tri_ref(p1, p2, p3);
    double s3 = area_tri_ref(p0, p2, p3);
    double s4 = area_tri_ref(p0, p1, p3);
    double A = fabs(s1) + fabs(s2) + fabs(s3) + fabs(s4);
    double M[9] = {p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2], p2[0] - p0[0], p2[1] - p0[1],
                   p2[2] - p0[2], p3[0] - p0[0], p3[1] - p0[1], p3[2] - p0[2]};
    const double D = det3_ref(M);
    if (det_edges) *det_edges = D;
    double V = 1.0 / 6.0 * fabs(D);
    double r = 3.0 * V / A;
    return 2 * r;
}

// The reference's sums start from 0, as (0 + a) + b + ...: bit for bit that is
// a + b + ... with -0 made +0.  Once 0 is added no partial sum is -0, so the two
// can only differ where every term is -0.  A mask in place of an FP64 addition,
// 46 of them a StVK element: 384,000 tets in exact mode 4.78 -> 4.29 ms for 20
// steps (bound by the FP64 pipe).
__device__ __forceinline__ double no_minus_zero(double x)
{
    return __double_as_longlong(x) == (long long)(1ull << 63) ? 0.0 : x;
}

// First Piola stress in the reference's operation order:
// hyperElasticNeoHookean.cpp:84-127 (Neo-Hookean), :235-259 (compressible),
// hyperElasticStVenantKirchhoff.cpp:64-101,219-222 (StVK), linearElastic.cpp
// :58-82,114-145 (linear elastic: the small-strain stress is returned as P).
__device__ __forceinline__ void stress_ref(const MatParams &m, const double *F, double *P)
{
    if (m.law == 1) {
        double J = det3_ref(F), C[9], iC[9], S[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                C[i * 3 + j] = no_minus_zero(F[i] * F[j] + F[3 + i] * F[3 + j] + F[6 + i] * F[6 + j]);
            }
        inv3_ref(C, iC);
        double alpha = m.lambda * log(J) - m.mu;
#pragma unroll
        for (int i = 0; i < 9; i++) S[i] = i % 4 ? no_minus_zero(alpha * iC[i]) : no_minus_zero(m.mu) + alpha * iC[i];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                P[i * 3 + j] = no_minus_zero(F[i * 3] * S[j] + F[i * 3 + 1] * S[3 + j] + F[i * 3 + 2] * S[6 + j]);
            }
    } else if (m.law == 0) {
        double B[9], iF[9], Ca[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                B[i * 3 + j] = no_minus_zero(F[i * 3] * F[j * 3] + F[i * 3 + 1] * F[j * 3 + 1] + F[i * 3 + 2] * F[j * 3 + 2]);
            }
        double J = det3_ref(F);
        inv3_ref(F, iF);
        const double trB = B[0] + B[4] + B[8];   // no -0 among them
        double fact1 = pow(J, 5.0 / 3.0);
        double fact2 = m.mu / fact1;
#pragma unroll
        for (int i = 0; i < 9; i++) Ca[i] = no_minus_zero(fact2 * B[i]);
        double fact3 = -(m.mu / 3.0) * trB / fact1 + m.K1 * (J - 1.0);
        // Ca_ij += fact3 delta_ij: off the diagonal fact3 * 0 adds nothing while fact3 is finite
        const double off = isfinite(fact3) ? 0.0 : fact3 * 0.0;
        if (off != 0.0)   // NaN
#pragma unroll
            for (int i = 0; i < 9; i++)
                if (i % 4) Ca[i] += off;
#pragma unroll
        for (int i = 0; i < 9; i += 4) Ca[i] += fact3;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                P[i * 3 + j] = no_minus_zero(Ca[i * 3] * iF[j * 3] * J + Ca[i * 3 + 1] * iF[j * 3 + 1] * J + Ca[i * 3 + 2] * iF[j * 3 + 2] * J);
            }
    } else if (m.law == 3) {
        // linearElastic.cpp:71-76 E = (F + F^T)/2 - I, :114-145 P = mu2 E + lam tr(E) I
        double E[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) E[i * 3 + j] = 0.5 * (F[i * 3 + j] + F[j * 3 + i] - 2. * (i == j ? 1. : 0.));
        const double trE = no_minus_zero(E[0] + E[4] + E[8]);
#pragma unroll
        for (int i = 0; i < 9; i++) P[i] = E[i] * m.mu2;
#pragma unroll
        for (int i = 0; i < 3; i++) P[i * 3 + i] += m.lam_stvk * trE;
    } else {
        double C[9], S[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                C[i * 3 + j] = no_minus_zero(F[i] * F[j] + F[3 + i] * F[3 + j] + F[6 + i] * F[6 + j]);
            }
#pragma unroll
        for (int i = 0; i < 9; i++) S[i] = 0.5 * (C[i] - ((i % 4) == 0 ? 1.0 : 0.0));
        const double trE = no_minus_zero(S[0] + S[4] + S[8]);
#pragma unroll
        for (int i = 0; i < 9; i++) S[i] = S[i] * m.mu2;
#pragma unroll
        for (int i = 0; i < 3; i++) S[i * 3 + i] += m.lam_stvk * trE;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                P[i * 3 + j] = no_minus_zero(F[i * 3] * S[j] + F[i * 3 + 1] * S[3 + j] + F[i * 3 + 2] * S[6 + j]);
            }
    }
}

// ---------------------------------------------------------------------------
// Shared pieces
// ---------------------------------------------------------------------------
__device__ __forceinline__ const MatParams &mat_of(const Problem &p, long long e)
{
    return p.mats[p.mat ? p.mat[e] : 0];
}

// Element birth (the reference's *ACTIVATION option: solvers.cpp:403-433 with
// the laws' checkActivation): a St-Venant-Kirchhoff or linear-elastic element
// is alive once its activation time is <= t; a dead element adds no internal
// force (solverExplicit.cpp:370-371).  act_t is null without the option.
__device__ __forceinline__ bool elem_dead(const Problem &p, long long e, double t)
{
    return p.act_t && mat_of(p, e).law >= 2 && t < p.act_t[e];
}

// Block-wide min of a positive double, then one integer atomicMin on its bit
// pattern (monotone for non-negative doubles; exact and order independent).
__device__ __forceinline__ void block_min_to(double v, unsigned long long *slot)
{
    __shared__ double wmin[32];
    if (!(v >= 0.0)) v = INFINITY;    // NaN or negative: ignored
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) wmin[w] = v;
    __syncthreads();
    if (w == 0) {
        int nw = (blockDim.x + 31) >> 5;
        v = l < nw ? wmin[l] : INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (l == 0 && v < INFINITY) atomicMin(slot, (unsigned long long)__double_as_longlong(v));
    }
    __syncthreads();   // wmin may be reused by the next call
}

// The control decision of the node kernel: derived identically in every
// thread from the previous slot (solverExplicit.cpp:217-276).
struct StepDecision {
    Ctrl next;
    bool run;
};

__device__ __forceinline__ StepDecision decide_step(const Problem &p, const Ctrl &cp, int parity)
{
    StepDecision d;
    d.next = cp;
    d.next.ran = 0;
    d.run = false;
    const unsigned long long dtmin = p.dtmin[parity];   // with the flag and the slot: one latency
    const int flag = p.flags[parity];
    if (cp.stop) return d;
    if (cp.ran && flag) {        // uK[1] not finite after the last step
        d.next.status = 4;
        d.next.stop = 1;
        return d;
    }
    if (cp.t < p.tf - 1E-12 && cp.step < cp.limit) {
        double t = cp.t, dt = cp.dt;
        if (t + dt > p.tf) {
            dt = p.tf - t;
            t = p.tf;
        } else {
            t += dt;
        }
        double dtn = __longlong_as_double((long long)dtmin);
        dtn = dtn * p.sf;
        d.next.t = t;
        if (dtn < 1E-20) {
            d.next.status = 3;
            d.next.stop = 1;
            d.next.dt = dtn;
        } else {
            d.next.dt = dtn;
            d.next.step = cp.step + 1;
            d.next.ran = 1;
            d.run = true;
        }
    } else {
        // stopped at tf or at the step limit: keep the CFL min of the next step
        // so that a later call can resume the block where it left off
        d.next.stop = 1;
        d.next.pending = dtmin;
    }
    return d;
}

// Dirichlet increment of one entry at block step `step` (solverExplicit.cpp:545-575)
__device__ __forceinline__ double bc_increment(const BCEntry &b, double dt, long long step)
{
    if (b.mode == 1) return step == 1 ? b.val : 0.0;
    if (b.mode == 2) {
        double r = (b.ramp_steps > 0 && step < b.ramp_steps) ? (double)step / (double)b.ramp_steps : 1.0;
        return b.val * r * dt;
    }
    return b.val * dt;
}

// ---------------------------------------------------------------------------
// Node kernel: post-update of step n-1 (a = -f_int/m, v += dt (a_prev+a)/2,
// nonlinearSystem.cpp:1034-1117), control of step n, prediction
// u += dt v + dt^2/2 a (nonlinearSystem.cpp:1186-1200) and Dirichlet values.
// One thread per node, three components.
// ---------------------------------------------------------------------------
// Dirichlet records of node i: per component (first entry, count); count 0 = active.
__device__ __forceinline__ void node_bc_records(const Problem &p, long long i, int2 *br)
{
    br[0] = br[1] = br[2] = make_int2(0, 0);
    int rec = p.node_bc[i];
    if (rec >= 0) {
        br[0] = p.bc_rec[rec * 3 + 0];
        br[1] = p.bc_rec[rec * 3 + 1];
        br[2] = p.bc_rec[rec * 3 + 2];
    }
}

// External force of DOF d at time t (the step being completed): its terms in
// deck order, summed from 0 as NeumannBCManagement fills the force vector
// (boundaryConditions.cpp:75-138; nodal forces m t inside [t0, tf],
// classNodes.h:101-109).
__device__ __forceinline__ double ext_force_dof(const Problem &p, long long d, double t)
{
    double fx = 0.0;
    for (int k = p.ext_ptr[d]; k < p.ext_ptr[d + 1]; k++) {
        const unsigned term = p.ext_term[k], idx = term & ((1u << kExtIndexBits) - 1u);
        double v;
        switch (term >> kExtIndexBits) {
        case EXT_FORCE: {
            const ForceEntry f = p.nfs[idx];
            v = (t >= f.t0 && t <= f.tf) ? f.m * t : 0;
            break;
        }
        case EXT_GRAV_ELEM: v = p.grav_e[idx]; break;
        case EXT_GRAV_NODE: v = p.grav_n[idx]; break;
        default: v = p.fcon[idx]; break;
        }
        fx += v;
    }
    return fx;
}

// One DOF: post-update of step n-1 with the gathered internal force s and
// external force fx (a = (fx - s)/m, v += dt (a_prev + a)/2), then the
// prediction (active) or the Dirichlet values (constrained) of step n.  The
// reference-order mode keeps the reference's operations; the others use
// v += (dt/2)(a_prev + a) and u += dt (v + (dt/2) a) with 1/m.
template <int MODE>
__device__ __forceinline__ void dof_update(const Problem &p, long long dof, double ui, double vi, double ai, double s,
                                           double fx, bool loads, int2 br, const Ctrl &cp, const StepDecision &d,
                                           double mass, double minv)
{
    const bool act = br.y == 0;
    bool changed = false;
    if (cp.ran && act) {
        double an;
        if (MODE == MODE_EXACT) {
            double val = -s + fx;
            double rhs = 0;
            rhs += val;
            an = rhs / mass;
            vi += cp.dt * ((1. - 0.5) * ai + 0.5 * an);
        } else {
            an = (loads ? fx - s : -s) * minv;
            vi = fma(0.5 * cp.dt, ai + an, vi);
        }
        ai = an;
        changed = true;
    }
    if (d.run) {
        const double dtn = d.next.dt;
        if (act) {
            if (MODE == MODE_EXACT) ui += dtn * vi + 0.5 * dtn * dtn * ai;
            else ui = fma(dtn, fma(0.5 * dtn, ai, vi), ui);
        } else {
            for (int k = br.x; k < br.x + br.y; k++) {
                double Ud = bc_increment(p.bcs[k], dtn, d.next.step);
                ui += Ud;
                vi = Ud;
                ai = 0.;
            }
        }
        changed = true;
    }
    if (changed) {
        p.u[dof] = ui;
        p.v[dof] = vi;
        p.a[dof] = ai;
        if (MODE == MODE_MIXED) {
            float hi = (float)ui;
            p.uhl[dof] = make_float2(hi, (float)(ui - (double)hi));
        }
    }
}

// Node kernel body, one thread per node (reference-order mode): corner forces
// of the incident elements summed in element order, then the three DOFs.
template <int MODE>
__device__ __forceinline__ void node_body(const Problem &p, long long i, const Ctrl &cp, const StepDecision &d)
{
    int2 br[3];
    node_bc_records(p, i, br);
    double s[3] = {0.0, 0.0, 0.0};
    if (cp.ran && (br[0].y == 0 || br[1].y == 0 || br[2].y == 0)) {
        for (int k = p.node_ptr[i]; k < p.node_ptr[i + 1]; k++) {
            const double *f = p.fe + (long long)p.node_inc[k] * 3;
            s[0] += f[0];
            s[1] += f[1];
            s[2] += f[2];
        }
    }
    double fx[3] = {0.0, 0.0, 0.0};
    if (cp.ran && p.ext_ptr)
        for (int c = 0; c < 3; c++) fx[c] = ext_force_dof(p, i + c * p.nn, cp.t);
    const double mass = MODE == MODE_EXACT ? p.mass[i] : 0.0, minv = MODE == MODE_EXACT ? 0.0 : p.minv[i];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const long long dof = i + c * p.nn;
        dof_update<MODE>(p, dof, p.u[dof], p.v[dof], p.a[dof], s[c], fx[c], true, br[c], cp, d, mass, minv);
    }
}

// Rounding error of s = fl(a + b): a + b = s + err exactly (Knuth's TwoSum).
__device__ __forceinline__ float two_sum_err(float a, float b, float s)
{
    float bp = s - a;
    return (a - (s - bp)) + (b - bp);
}

// Neumaier merge of two compensated FP32 partial sums (lo first).
__device__ __forceinline__ void neumaier_merge(float &sh, float &sc, float oh, float oc)
{
    float t = sh + oh;
    float e = fabsf(sh) >= fabsf(oh) ? (sh - t) + oh : (oh - t) + sh;
    sh = t;
    sc = (sc + oc) + e;
}

// ---------------------------------------------------------------------------
// Double-word ("double-float") arithmetic: a value is a pair (hi, lo) of FP32
// numbers with value hi + lo and |lo| <= ulp(hi)/2, about 48 significant
// bits.  The mixed mode keeps the nodal state u, v, a in this form while a
// block runs, so its node update runs on the FP32 pipe (on this GPU the FP64
// pipe issues about 1/64 of the FP32 rate).  Algorithms: TwoSum (Knuth),
// Fast2Sum (Dekker), and the accurate double-word sum and double-word product
// of Joldes, Muller and Popescu, "Tight and rigorous error bounds for basic
// building blocks of double-word arithmetic", ACM TOMS 44 (2017), Algs. 6, 12.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 df_fast2sum(float a, float b)   // needs |a| >= |b| (or a = 0)
{
    float s = a + b;
    return make_float2(s, b - (s - a));
}

__device__ __forceinline__ float2 df_two_sum(float a, float b)
{
    float s = a + b;
    return make_float2(s, two_sum_err(a, b, s));
}

__device__ __forceinline__ float2 df_add(float2 x, float2 y)
{
    float2 s = df_two_sum(x.x, y.x), t = df_two_sum(x.y, y.y);
    float2 v = df_fast2sum(s.x, s.y + t.x);
    return df_fast2sum(v.x, t.y + v.y);
}

__device__ __forceinline__ float2 df_mul(float2 x, float2 y)
{
    float ch = x.x * y.x;
    float cl1 = fmaf(x.x, y.x, -ch);
    float cl2 = fmaf(x.y, y.x, fmaf(x.x, y.y, x.y * y.y));
    return df_fast2sum(ch, cl1 + cl2);
}

__device__ __forceinline__ float2 df_neg(float2 x) { return make_float2(-x.x, -x.y); }

// nearest double-word to an FP64 value (FP64 pipe: control values and loads only)
__device__ __forceinline__ float2 df_from(double x)
{
    float hi = (float)x;
    return make_float2(hi, (float)(x - (double)hi));
}

// Writes the new control slot and clears the slots the element kernel fills.
__device__ __forceinline__ void publish_step(const Problem &p, const StepDecision &d, int parity)
{
    p.ctrl[parity] = d.next;
    p.dtmin[parity ^ 1] = MSX_INF_BITS;
    p.dtmin[2 + (parity ^ 1)] = p.dtmin[4];   // the undeformed CFL minimum bounds every step's
    p.flags[parity ^ 1] = 0;
}

// Per-solve quantities of the node kernel, derived once per block and solve
// from the solve's control slot (not once per tile).
struct NodeStep {
    bool ran, run, loads;       // step n-1 ran / step n runs / external loads present
    long long step;             // block step number of step n
    double t;                   // time of step n-1 (external forces)
    double hdt, dtn, hdtn;      // dt/2 of the step being completed; dt, dt/2 of the next
    float2 hdt2, dtn2, hdtn2;   // the same as double-words (mixed)
};

template <int MODE>
__device__ __forceinline__ void node_step(const Problem &p, int parity, bool publish, NodeStep &ns)
{
    const Ctrl cp = p.ctrl[parity ^ 1];
    const StepDecision d = decide_step(p, cp, parity);
    if (publish) publish_step(p, d, parity);
    ns.ran = cp.ran;
    ns.run = d.run;
    ns.step = d.next.step;
    ns.t = cp.t;
    ns.hdt = 0.5 * cp.dt;
    ns.dtn = d.next.dt;
    ns.hdtn = 0.5 * ns.dtn;
    if (MODE == MODE_MIXED || MODE == MODE_DW) {
        ns.hdt2 = df_from(ns.hdt);
        ns.dtn2 = df_from(ns.dtn);
        ns.hdtn2 = df_from(ns.hdtn);
    }
    ns.loads = p.ext_ptr != nullptr;
}

// Node kernel bodies of the tiled FP64 and mixed kernels: four lanes per node.
// The node's corner forces sit in its CSR slots [node_ptr[i], node_ptr[i+1]),
// in element order; lane q sums slots k0+q, k0+q+4, ...  The lane sums l_q
// are combined as (l0 + l1) + (l2 + l3) for every component (addition and
// the compensated merge are commutative, so the result does not depend on
// which lane adds): each lane receives only what it or the lane it serves
// next needs.  Lane c < 3 then updates DOF c: a = (f_ext - f_int)/m,
// v += (dt/2)(a_prev + a), u += dt (v + (dt/2) a), or the Dirichlet values.
// The DOF state, mass and Dirichlet record are loaded before the gather so
// their latency overlaps it.  All 32 lanes of a warp call these together
// (valid = false past the tile's end).
template <typename T>
__device__ __forceinline__ T pick3(int c, T a, T b, T d) { return c == 0 ? a : (c == 1 ? b : d); }

__device__ __forceinline__ double node_fext(const Problem &p, long long i, int q, const NodeStep &ns)
{
    return ext_force_dof(p, i + (long long)q * p.nn, ns.t);
}

// The high word of |x|: ordered as |x| to its first 20 mantissa bits.
__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7FFFFFFF; }

// Adds x as an integer multiple of 2^(E - 1075 - H), truncated toward zero, to
// a, for R = E + 10 - H, 0 <= H <= 10, and E >= kFixedLeast at least x's exponent
// field and not 0x7FF.  Zeros and subnormals, which take the implicit bit too,
// lie 2^64 below E's unit and shift out.
constexpr int kFixedLeast = 75;
__device__ __forceinline__ void add_fixed(long long &a, double x, int R)
{
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned h = (__funnelshift_l(xl, xh, 10) & 0x3FFFFFFFu) | 0x40000000u;   // the significand's 53 bits << 10
    unsigned long long t = (unsigned long long)h << 32 | (xl << 10);
    asm("{\n\t.reg .pred p;\n\t"
        "shr.u64 %1, %1, %2;\n\t"   // beyond 63: zero
        "setp.lt.s32 p, %3, 0;\n\t"
        "@p sub.s64 %0, %0, %1;\n\t"
        "@!p add.s64 %0, %0, %1;\n\t}"
        : "+l"(a), "+l"(t)
        : "r"(R - (int)((xh & 0x7FFFFFFFu) >> 20)), "r"((int)xh));
}

// x * 2^k for an integer-valued x (|x| < 2^63) and -1085 <= k <= 971: exact
// unless the product is subnormal, then rounded once (the first factor of the
// two-step case keeps x * 2^-600 normal and exact).
__device__ __forceinline__ double pow2_scale(double x, int k)
{
    if (k < -1022) {
        x *= __longlong_as_double((long long)(1023 - 600) << 52);
        k += 600;
    }
    return x * __longlong_as_double((long long)(k + 1023) << 52);
}

// A 24-byte corner slot of the FP64 layout (slot k at byte 24 k: 16-byte
// aligned for even k) in one 16-byte and one 8-byte access instead of three
// 8-byte ones: the 16-byte half holds values 0-1 of an even slot, 1-2 of an
// odd one.  The selects keep the warp on one path.
__device__ __forceinline__ void st_slot24(double *base, long long k, double x, double y, double z)
{
    const bool odd = k & 1;
    double *s = base + 3 * k;
    *reinterpret_cast<double2 *>(s + (odd ? 1 : 0)) = odd ? make_double2(y, z) : make_double2(x, y);
    s[odd ? 0 : 2] = odd ? x : z;
}

// A node's first 4 kBatch corner-force slots go to registers in one batch when
// BATCH (kernels whose grid has a block for every tile): few warps are resident
// then, and slot after slot costs a memory latency each.
constexpr int kBatch = 8;

// A value of the state or the corner forces.  DEP: the kernel may be under way
// while the one before it still writes them (programmatic dependent launch, see
// pdl_wait), where the read-only path promises nothing; without, that path takes
// 2 % off a step of 6M tets.
template <bool DEP, typename T>
__device__ __forceinline__ T ld_step(const T *x)
{
    return DEP ? *x : __ldg(x);
}

template <bool BATCH>
__device__ __forceinline__ void node_quad_fp64(const Problem &p, long long i, bool valid, const NodeStep &ns, int2 slots)
{
    const int q = threadIdx.x & 3;
    const bool odd = q & 1;
    const bool own = valid && q < 3;   // this lane updates DOF q of node i
    const long long dof = i + (long long)q * p.nn;
    double ui = 0, vi = 0, ai = 0, minv = 0;
    int rec = -1;
    if (own) {
        ui = p.u[dof];
        vi = p.v[dof];
        ai = p.a[dof];
        minv = p.minv[i];
        rec = p.node_bc[i];
    }
    const int k0 = slots.x, k1 = slots.y;
    // The node's f_int per component as one exact integer sum, rounded once:
    // each term's 53-bit significand aligned to the largest exponent E of that
    // component among the node's terms, with H guard bits below it, summed in
    // int64 on the integer pipes instead of ~24 dependent FP64 additions.  With
    // n terms, H = 10 - ceil(log2 n) keeps the sum below 2^63; bits below the
    // guard bits are truncated (at most one unit of 2^(E - 1075 - H) per term).
    // The sum does not depend on the order of the terms.  Nodes with an
    // infinite or NaN term, a component whose largest term is below 2^-948 but
    // not 0 (subnormals below 2^-1042 count as 0), or too many terms for H >= 0
    // (and the other nodes of their warp), add in FP64.
    // A lane's slots are all even or all odd, so it adds the three values in
    // the order they lie in its two loads (xyz, or yzx) and turns the sums, not
    // the values: 6M tets, node kernel 181 -> 174 us with this and add_fixed (the ALU
    // pipe was 63 % busy); 6000 tets 14.8 -> 13.2 us a step.
    const int n = k1 - k0;   // the same for the node's four lanes
    const bool turned = (k0 + q) & 1;
    const double *at = p.fe + 3LL * (k0 + q), *at2 = at + (turned ? 1 : 0), *at1 = at + (turned ? 0 : 2);
    int zx = 0, zy = 0, zw = 0;
    constexpr int NB = BATCH ? kBatch : 0;
    double2 g2[NB + 1];
    double g1[NB + 1];
    if (BATCH) {
#pragma unroll
        for (int j = 0; j < NB; j++) {
            g2[j] = make_double2(0.0, 0.0);
            g1[j] = 0.0;
            if (k0 + q + 4 * j < k1) {
                g2[j] = ld_step<BATCH>(reinterpret_cast<const double2 *>(at2 + 12 * j));
                g1[j] = ld_step<BATCH>(at1 + 12 * j);
            }
        }
#pragma unroll
        for (int j = 0; j < NB; j++) {
            zx = max(zx, abs_hi(g2[j].x));
            zy = max(zy, abs_hi(g2[j].y));
            zw = max(zw, abs_hi(g1[j]));
        }
    }
    for (int k = k0 + q + 4 * NB, o = 12 * NB; k < k1; k += 4, o += 12) {
        const double2 f = ld_step<BATCH>(reinterpret_cast<const double2 *>(at2 + o));
        zx = max(zx, abs_hi(f.x));
        zy = max(zy, abs_hi(f.y));
        zw = max(zw, abs_hi(ld_step<BATCH>(at1 + o)));
    }
    int z0 = turned ? zw : zx, z1 = turned ? zx : zy, z2 = turned ? zy : zw;
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        z0 = max(z0, __shfl_xor_sync(0xffffffffu, z0, o));
        z1 = max(z1, __shfl_xor_sync(0xffffffffu, z1, o));
        z2 = max(z2, __shfl_xor_sync(0xffffffffu, z2, o));
    }
    const int H = 10 - (n > 1 ? 32 - __clz(n - 1) : 0);
    const auto in_range = [](int z) { return z == 0 || (z >= kFixedLeast << 20 && z < 0x7FF << 20); };
    // one path for the whole warp: both use shuffles over all 32 lanes (lanes
    // past the tile's end have no terms and vote for the integer path)
    const bool fixed = __all_sync(0xffffffffu, H >= 0 && in_range(z0) && in_range(z1) && in_range(z2));
    double s;
    if (fixed) {
        // a component of zeros: every term shifts out
        const int r0 = (z0 ? z0 >> 20 : 4000) + 10 - H, r1 = (z1 ? z1 >> 20 : 4000) + 10 - H,
                  r2 = (z2 ? z2 >> 20 : 4000) + 10 - H;
        const int rx = turned ? r1 : r0, ry = turned ? r2 : r1, rw = turned ? r0 : r2;
        long long ax = 0, ay = 0, aw = 0;
        if (BATCH) {
#pragma unroll
            for (int j = 0; j < NB; j++) {
                add_fixed(ax, g2[j].x, rx);
                add_fixed(ay, g2[j].y, ry);
                add_fixed(aw, g1[j], rw);
            }
        }
        for (int k = k0 + q + 4 * NB, o = 12 * NB; k < k1; k += 4, o += 12) {
            const double2 f = ld_step<BATCH>(reinterpret_cast<const double2 *>(at2 + o));
            const double w = ld_step<BATCH>(at1 + o);
            add_fixed(ax, f.x, rx);
            add_fixed(ay, f.y, ry);
            add_fixed(aw, w, rw);
        }
        long long a0 = turned ? aw : ax, a1 = turned ? ax : ay, a2 = turned ? ay : aw;
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, o);
            a1 += __shfl_xor_sync(0xffffffffu, a1, o);
            a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        if (!own) return;
        s = pow2_scale(__ll2double_rn(pick3(q, a0, a1, a2)), (pick3(q, z0, z1, z2) >> 20) - 1075 - H);
    } else {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (int k = k0 + q; k < k1; k += 4) {
            const double *f = p.fe + (long long)k * 3;
            s0 += f[0];
            s1 += f[1];
            s2 += f[2];
        }
        // pairs (0,1), (2,3): even lanes need components 0 and 2, odd lanes 1
        double x = __shfl_xor_sync(0xffffffffu, odd ? s0 : s1, 1), y = __shfl_xor_sync(0xffffffffu, s2, 1);
        if (odd) {
            s1 += x;
        } else {
            s0 += x;
            s2 += y;
        }
        // across pairs: lanes 0 <-> 2 exchange components 2 / 0, lane 1 <- 3 component 1
        double z = __shfl_xor_sync(0xffffffffu, odd ? s1 : (q == 0 ? s2 : s0), 2);
        if (!own) return;
        s = pick3(q, s0, s1, s2) + z;
    }
    const int2 br = rec >= 0 ? p.bc_rec[rec * 3 + q] : make_int2(0, 0);
    const bool act = br.y == 0;
    bool changed = false;
    if (ns.ran && act) {
        const double an = (ns.loads ? node_fext(p, i, q, ns) - s : -s) * minv;
        vi = fma(ns.hdt, ai + an, vi);
        ai = an;
        changed = true;
    }
    if (ns.run) {
        if (act) {
            ui = fma(ns.dtn, fma(ns.hdtn, ai, vi), ui);
        } else {
            for (int k = br.x; k < br.x + br.y; k++) {
                double Ud = bc_increment(p.bcs[k], ns.dtn, ns.step);
                ui += Ud;
                vi = Ud;
                ai = 0.;
            }
        }
        changed = true;
    }
    if (changed) {
        p.u[dof] = ui;
        p.v[dof] = vi;
        p.a[dof] = ai;
        if (p.u4) p.u4[4LL * i + q] = ui;
    }
}

// The mixed mode's acceleration, one FP32 per DOF in the storage of ahl: a is
// recomputed every step from the FP32 corner forces (compensated sum / m), so
// FP32 holds all it carries; u and v, the accumulated state, stay double-words.
__device__ __forceinline__ float *mixed_a32(const Problem &p) { return reinterpret_cast<float *>(p.ahl); }

template <bool BATCH>
__device__ __forceinline__ void node_quad_mixed(const Problem &p, long long i, bool valid, const NodeStep &ns, int2 slots)
{
    const int q = threadIdx.x & 3;
    const bool odd = q & 1;
    const bool own = valid && q < 3;
    const long long dof = i + (long long)q * p.nn;
    float2 uq = make_float2(0.f, 0.f), vq = uq, aq = uq, minv = uq;
    int rec = -1;
    if (own) {
        uq = p.uhl[dof];
        vq = p.vhl[dof];
        aq = make_float2(mixed_a32(p)[dof], 0.f);
        minv = p.minv2[i];
        rec = p.node_bc[i];
    }
    const int k0 = slots.x, k1 = slots.y;
    // compensated FP32 sums (Neumaier) of the FP32 corner forces
    const float4 *fe = reinterpret_cast<const float4 *>(p.fe32);
    float h0 = 0.f, h1 = 0.f, h2 = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f;
    int k = k0 + q;
    constexpr int NB = BATCH ? kBatch : 0;
    float4 g[NB + 1];
    if (BATCH) {
#pragma unroll
        for (int j = 0; j < NB; j++)
            if (k + 4 * j < k1) g[j] = fe[k + 4 * j];
#pragma unroll
        for (int j = 0; j < NB; j++) {
            if (k >= k1) break;
            if (j == 0) {
                h0 = g[0].x;
                h1 = g[0].y;
                h2 = g[0].z;
            } else {
                neumaier_merge(h0, c0, g[j].x, 0.0f);
                neumaier_merge(h1, c1, g[j].y, 0.0f);
                neumaier_merge(h2, c2, g[j].z, 0.0f);
            }
            k += 4;
        }
    } else if (k < k1) {
        const float4 f = fe[k];
        h0 = f.x;
        h1 = f.y;
        h2 = f.z;
        k += 4;
    }
    for (; k < k1; k += 4) {
        const float4 f = fe[k];
        neumaier_merge(h0, c0, f.x, 0.0f);
        neumaier_merge(h1, c1, f.y, 0.0f);
        neumaier_merge(h2, c2, f.z, 0.0f);
    }
    float ah = odd ? h0 : h1, ac = odd ? c0 : c1;
    float xh = __shfl_xor_sync(0xffffffffu, ah, 1), xc = __shfl_xor_sync(0xffffffffu, ac, 1);
    float yh = __shfl_xor_sync(0xffffffffu, h2, 1), yc = __shfl_xor_sync(0xffffffffu, c2, 1);
    if (odd) {
        neumaier_merge(h1, c1, xh, xc);
    } else {
        neumaier_merge(h0, c0, xh, xc);
        neumaier_merge(h2, c2, yh, yc);
    }
    float sh = odd ? h1 : (q == 0 ? h2 : h0), sc = odd ? c1 : (q == 0 ? c2 : c0);
    float zh = __shfl_xor_sync(0xffffffffu, sh, 2), zc = __shfl_xor_sync(0xffffffffu, sc, 2);
    float mh = pick3(q, h0, h1, h2), mc = pick3(q, c0, c1, c2);
    neumaier_merge(mh, mc, zh, zc);
    if (!own) return;
    const float2 s = df_two_sum(mh, mc);
    const int2 br = rec >= 0 ? p.bc_rec[rec * 3 + q] : make_int2(0, 0);
    const bool act = br.y == 0;
    bool changed = false;
    if (ns.ran && act) {
        const float2 f = ns.loads ? df_add(df_from(node_fext(p, i, q, ns)), df_neg(s)) : df_neg(s);
        const float2 an = df_mul(f, minv);
        vq = df_add(vq, df_mul(ns.hdt2, df_add(aq, an)));
        aq = make_float2(__fadd_rn(an.x, an.y), 0.f);   // as stored: the prediction uses what a later call reads
        changed = true;
    }
    if (ns.run) {
        if (act) {
            uq = df_add(uq, df_mul(ns.dtn2, df_add(vq, df_mul(ns.hdtn2, aq))));
        } else {
            for (int k = br.x; k < br.x + br.y; k++) {
                const float2 Ud = df_from(bc_increment(p.bcs[k], ns.dtn, ns.step));
                uq = df_add(uq, Ud);
                vq = Ud;
                aq = make_float2(0.f, 0.f);
            }
        }
        changed = true;
    }
    if (changed) {
        p.uhl[dof] = uq;
        p.vhl[dof] = vq;
        mixed_a32(p)[dof] = aq.x;
    }
}

template <int MODE>
__global__ void __launch_bounds__(kNodeBlock) node_kernel(Problem p, int parity)
{
    const Ctrl cp = p.ctrl[parity ^ 1];
    StepDecision d = decide_step(p, cp, parity);
    if (blockIdx.x == 0 && threadIdx.x == 0) publish_step(p, d, parity);
    if (!cp.ran && !d.run) return;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.nn) node_body<MODE>(p, i, cp, d);
}

// ---------------------------------------------------------------------------
// Element kernels: F, P, wJ B^T P corner forces and the deformed CFL length.
// ---------------------------------------------------------------------------

// Reference operation order (used with contraction off).
__device__ __forceinline__ float f32_trunc(double x);
__device__ __forceinline__ float gate_moved(float Lr, float d, float inv_c);
__device__ __forceinline__ float cfl_screen(const Problem &p, long long e, const float *g, const float *du,
                                            const MatParams &m);

// Exact CFL value of one element, min(L_ref, L(X+u)) / c, in the reference's
// order (solvers.cpp:304-317: deformed inscribed sphere).
__device__ __forceinline__ double cfl_exact_ref(const Problem &p, long long e)
{
    const long long nn = p.nn;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double x[12];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            x[a * 3 + k] = p.X[k * nn + nd[a]];
            x[a * 3 + k] += p.u[nd[a] + k * nn];
        }
    double dist = char_length_ref(x);
    double Lr = p.Lref[e];
    double mlen = (dist < Lr) ? dist : Lr;
    return mlen / mat_of(p, e).c;
}

// SCREEN: return the FP32 screen value of the CFL (cfl_screen) instead of the
// exact one; the caller rechecks the elements near its block's minimum.
template <bool FORCE_ONLY, bool SCREEN = false, bool VISC = false>
__device__ __forceinline__ double elem_body_exact(const Problem &p, long long e, int parity, float gmin = 0.0f)
{
    const long long ne = p.ne, nn = p.nn;
    double vmin = INFINITY;
    {
        int4 cn = p.conn[e];
        int nd[4] = {cn.x, cn.y, cn.z, cn.w};
        double dphi[12];
#pragma unroll
        for (int k = 0; k < 9; k++) dphi[3 + k] = p.G[k * ne + e];
#pragma unroll
        for (int j = 0; j < 3; j++) dphi[j] = (-dphi[3 + j] - dphi[6 + j]) - dphi[9 + j];
        double ue[12];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int i = 0; i < 3; i++) ue[a * 3 + i] = p.u[nd[a] + i * nn];
        // constitutiveManager.cpp:151-164: each entry's sum starts from 0, then 1 on the diagonal
        double F[9], P[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                double c = i == j ? 1. + dphi[j] * ue[i] : dphi[j] * ue[i];
#pragma unroll
                for (int a = 1; a < 4; a++) c += dphi[a * 3 + j] * ue[a * 3 + i];
                F[i * 3 + j] = i == j ? c : no_minus_zero(c);
            }
        const MatParams &m = mat_of(p, e);
        stress_ref(m, F, P);
        // constitutiveAlgorithms.cpp:46-56
        double wJ = p.wJ[e];
        double *fe = p.fe + e * 12;
        const bool dead = !FORCE_ONLY && elem_dead(p, e, p.ctrl[parity].t);
        double Pv[9];
        if (VISC && !FORCE_ONLY) {
            // bulkViscosity in the reference's order (solverExplicit.cpp:514-541; sumTensorTensor,
            // multiSTensorScalar, getTrace, multSTensor3SecondTranspose: maths.cpp:1169-1175,
            // 1604-1610, 2257-2286); F_prev's diagonal rolls to F's
            double *f0 = p.visc_f0;
            const double dt = p.ctrl[parity].dt;
            double Fd[3] = {0., 0., 0.};
            if (dt != 0) {
                const double r = 1 / dt;
#pragma unroll
                for (int c = 0; c < 3; c++) Fd[c] = (F[c * 4] + (-1) * f0[c * ne + e]) * r;
            }
            double trD = 0;
#pragma unroll
            for (int c = 0; c < 3; c++) trD += Fd[c];
#pragma unroll
            for (int c = 0; c < 3; c++) f0[c * ne + e] = F[c * 4];
            const double J1 = det3_ref(F);
            const double Rho_1 = m.rho / J1;
            const double qBV = Rho_1 * p.visc_h *
                               (p.visc_c1 * p.visc_c1 * p.visc_h * fabs(trD) * ((trD < 0.) ? trD : 0.) +
                                p.visc_cl * p.visc_c0 * trD);
            double Cv[9], iF[9];
#pragma unroll
            for (int k = 0; k < 9; k++) Cv[k] = (k % 4 == 0) ? -1 * qBV : 0.0;
            inv3_ref(F, iF);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    double s = 0;
#pragma unroll
                    for (int k = 0; k < 3; k++) s += Cv[i * 3 + k] * iF[j * 3 + k];
                    Pv[i * 3 + j] = s * (-1 * J1);
                }
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int i = 0; i < 3; i++) {
                double f = no_minus_zero(wJ * P[i * 3] * dphi[a * 3] + wJ * P[i * 3 + 1] * dphi[a * 3 + 1] +
                                         wJ * P[i * 3 + 2] * dphi[a * 3 + 2]);
                if (VISC && !FORCE_ONLY)   // the viscous pass's terms, as computeInternalForce adds them
#pragma unroll
                    for (int J = 0; J < 3; J++) f += wJ * Pv[i * 3 + J] * dphi[a * 3 + J];
                fe[a * 3 + i] = dead ? 0.0 : f;
            }
        if (!FORCE_ONLY && SCREEN) {
            if (e == 0 && !isfinite(p.u[1])) atomicOr(p.flags + (parity ^ 1), 1);
            // the gate takes FP32 differences of the truncated displacements: off by 2^-22 |u|
            float u32[12], d2 = 0.0f, um = 0.0f;
#pragma unroll
            for (int k = 0; k < 12; k++) {
                u32[k] = f32_trunc(ue[k]);
                um = fmaxf(um, fabsf(u32[k]));
            }
#pragma unroll
            for (int a = 1; a < 4; a++) {
                float q = 0.0f;
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const float w = u32[a * 3 + i] - u32[i];
                    q += w * w;
                }
                d2 = fmaxf(d2, q);
            }
            float dm;
            asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(dm) : "f"(d2));
            if (gate_moved(__ldg(p.Lref32 + e), dm + 0x1p-20f * um, m.inv_c_f) > gmin) return INFINITY;
            float du32[9];
#pragma unroll
            for (int a = 1; a < 4; a++)
#pragma unroll
                for (int i = 0; i < 3; i++) du32[(a - 1) * 3 + i] = f32_trunc(ue[a * 3 + i] - ue[i]);
            float g32[9];
#pragma unroll
            for (int k = 0; k < 9; k++) g32[k] = f32_trunc(dphi[3 + k]);
            vmin = (double)cfl_screen(p, e, g32, du32, m);
        } else if (!FORCE_ONLY) {
            // solvers.cpp:304-317: deformed inscribed sphere
            double x[12];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    x[a * 3 + k] = p.X[k * nn + nd[a]];
                    x[a * 3 + k] += ue[a * 3 + k];
                }
            double dist = char_length_ref(x);
            double Lr = p.Lref[e];
            double mlen = (dist < Lr) ? dist : Lr;
            vmin = mlen / m.c;
            if (e == 0 && !isfinite(p.u[1])) atomicOr(p.flags + (parity ^ 1), 1);
        }
    }
    return vmin;
}

template <bool FORCE_ONLY>
__global__ void __launch_bounds__(kElemBlock) elem_kernel_exact(Problem p, int parity)
{
    if (!FORCE_ONLY && !p.ctrl[parity].ran) return;
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double v = e < p.ne ? elem_body_exact<FORCE_ONLY>(p, e, parity) : INFINITY;
    if (!FORCE_ONLY) block_min_to(v, p.dtmin + (parity ^ 1));
}

// Plain FP64 with contraction: H from node differences, laws written through
// the cofactor of F (F C^-1 = F^-T = cof(F)/J), the 4th corner force as minus
// the sum of the other three.  Same algebra as the reference, fewer FP64
// operations.
__device__ __forceinline__ void cofactor(const double *F, double *K)
{
    K[0] = F[4] * F[8] - F[5] * F[7];
    K[1] = F[5] * F[6] - F[3] * F[8];
    K[2] = F[3] * F[7] - F[4] * F[6];
    K[3] = F[2] * F[7] - F[1] * F[8];
    K[4] = F[0] * F[8] - F[2] * F[6];
    K[5] = F[1] * F[6] - F[0] * F[7];
    K[6] = F[1] * F[5] - F[2] * F[4];
    K[7] = F[2] * F[3] - F[0] * F[5];
    K[8] = F[0] * F[4] - F[1] * F[3];
}

// Artificial bulk viscosity (the second pass of computeInternalForce,
// solverExplicit.cpp:381-421, with bulkViscosity, :514-541): the viscous
// Cauchy stress -qBV I maps to the Piola stress J qBV F^-T = qBV cof(F), with
// qBV = rho/J h (c1^2 h |trD| min(0, trD) + cl c0 trD) and trD = tr(Fdot),
// Fdot = (F - F_prev)/dt.  Only F_prev's diagonal enters, so that is what an
// element keeps; h and c0 stand for the reference's solvers::_elementSize and
// _c0.  FP64 form; the mixed and reference-order forms sit in their bodies.
__device__ __forceinline__ double visc_q(const Problem &p, double rho, double J, double trD)
{
    return rho / J * p.visc_h * (p.visc_c1 * p.visc_c1 * p.visc_h * fabs(trD) * fmin(0.0, trD) +
                                 p.visc_cl * p.visc_c0 * trD);
}

// P += wJ qBV cof(F) for F in FP64 (FP64 and double-word modes); rolls the
// element's F_prev diagonal to F's.
__device__ __forceinline__ void visc_bulk_fp64(const Problem &p, long long e, const double *F, double wJ, double rho,
                                               double idt, double *Pv)
{
    const long long ne = p.ne;
    double *f0 = p.visc_f0;
    const double trD = ((F[0] - f0[e]) + (F[4] - f0[ne + e]) + (F[8] - f0[2 * ne + e])) * idt;
    f0[e] = F[0];
    f0[ne + e] = F[4];
    f0[2 * ne + e] = F[8];
    double K[9];
    cofactor(F, K);
    const double J = F[0] * K[0] + F[1] * K[1] + F[2] * K[2];
    const double w = wJ * visc_q(p, rho, J, trD);
#pragma unroll
    for (int k = 0; k < 9; k++) Pv[k] = w * K[k];
}

// ln J for J = det F in FP64.  For |J - 1| < 2^-7 (the usual case) the
// series of log1p(x), x = J - 1, to x^9 by Horner's rule: truncation below
// |x|^10/10 < 1e-22 |x|, so its error is that of the rounded coefficients,
// about 1 ulp of ln J; x itself carries J's rounding, as log(J) does.
// Otherwise the library log.
__device__ __forceinline__ double log_near1(double J)
{
    const double x = J - 1.0;
    if (!(fabs(x) < 0.0078125)) return log(J);
    double q = 1.0 / 9.0;
    q = fma(q, -x, 1.0 / 8.0);
    q = fma(q, -x, 1.0 / 7.0);
    q = fma(q, -x, 1.0 / 6.0);
    q = fma(q, -x, 1.0 / 5.0);
    q = fma(q, -x, 1.0 / 4.0);
    q = fma(q, -x, 1.0 / 3.0);
    q = fma(q, -x, 1.0 / 2.0);
    q = fma(q, -x, 1.0);
    return q * x;
}

// wJ * P written through the cofactor; the quadrature weight is folded into
// the law's scalar coefficients instead of scaling the nine entries of P.
__device__ __forceinline__ void stress_fast(const MatParams &m, const double *F, double wJ, double *P)
{
    if (m.law == 3) {
        // linear elastic: wJ P = wJ (mu2 E + lam tr(E) I), E = (F + F^T)/2 - I
        const double h = m.mu2 * wJ;
        const double E00 = F[0] - 1.0, E11 = F[4] - 1.0, E22 = F[8] - 1.0;
        const double dg = m.lam_stvk * ((E00 + E11) + E22) * wJ;
        P[0] = h * E00 + dg;
        P[4] = h * E11 + dg;
        P[8] = h * E22 + dg;
        P[1] = P[3] = 0.5 * h * (F[1] + F[3]);
        P[2] = P[6] = 0.5 * h * (F[2] + F[6]);
        P[5] = P[7] = 0.5 * h * (F[5] + F[7]);
        return;
    }
    if (m.law == 2) {
        // S = mu2 E + lam tr(E) I, E = (F^T F - I)/2; wJ P = F (wJ S)
        double C00 = F[0] * F[0] + F[3] * F[3] + F[6] * F[6];
        double C11 = F[1] * F[1] + F[4] * F[4] + F[7] * F[7];
        double C22 = F[2] * F[2] + F[5] * F[5] + F[8] * F[8];
        double C01 = F[0] * F[1] + F[3] * F[4] + F[6] * F[7];
        double C02 = F[0] * F[2] + F[3] * F[5] + F[6] * F[8];
        double C12 = F[1] * F[2] + F[4] * F[5] + F[7] * F[8];
        double trE = 0.5 * ((C00 - 1.0) + (C11 - 1.0) + (C22 - 1.0));
        double h = 0.5 * m.mu2 * wJ, dg = m.lam_stvk * trE * wJ;
        double S00 = h * (C00 - 1.0) + dg, S11 = h * (C11 - 1.0) + dg, S22 = h * (C22 - 1.0) + dg;
        double S01 = h * C01, S02 = h * C02, S12 = h * C12;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            double f0 = F[i * 3], f1 = F[i * 3 + 1], f2 = F[i * 3 + 2];
            P[i * 3 + 0] = f0 * S00 + f1 * S01 + f2 * S02;
            P[i * 3 + 1] = f0 * S01 + f1 * S11 + f2 * S12;
            P[i * 3 + 2] = f0 * S02 + f1 * S12 + f2 * S22;
        }
        return;
    }
    double K[9];
    cofactor(F, K);
    double J = F[0] * K[0] + F[1] * K[1] + F[2] * K[2];
    double iJ = 1.0 / J;
    double a1, g;
    if (m.law == 1) {
        // P = mu F + (lambda ln J - mu) F^-T
        a1 = m.mu * wJ;
        g = (m.lambda * log_near1(J) - m.mu) * iJ * wJ;
    } else {
        // P = mu J^-2/3 F + (-mu/3 trB J^-5/3 + K1 (J-1)) cof(F)
        double r = rcbrt(J);
        double j23 = r * r;
        double trB = 0;
#pragma unroll
        for (int k = 0; k < 9; k++) trB += F[k] * F[k];
        a1 = m.mu * j23 * wJ;
        g = (-(m.mu / 3.0) * trB * j23 * iJ + m.K1 * (J - 1.0)) * wJ;
    }
#pragma unroll
    for (int k = 0; k < 9; k++) P[k] = a1 * F[k] + g * K[k];
}

// Inscribed-sphere diameter from the three edge vectors at vertex 0:
// 2 r = 2 |e1.(e2 x e3)| / (|e1xe2| + |e1xe3| + |e2xe3| + |(e2-e1)x(e3-e1)|).
template <typename T>
__device__ __forceinline__ T char_length_edges(const T *e1, const T *e2, const T *e3)
{
    T A0 = e1[1] * e2[2] - e1[2] * e2[1], A1 = e1[2] * e2[0] - e1[0] * e2[2], A2 = e1[0] * e2[1] - e1[1] * e2[0];
    T B0 = e1[1] * e3[2] - e1[2] * e3[1], B1 = e1[2] * e3[0] - e1[0] * e3[2], B2 = e1[0] * e3[1] - e1[1] * e3[0];
    T C0 = e2[1] * e3[2] - e2[2] * e3[1], C1 = e2[2] * e3[0] - e2[0] * e3[2], C2 = e2[0] * e3[1] - e2[1] * e3[0];
    T D0 = C0 + A0 - B0, D1 = C1 + A1 - B1, D2 = C2 + A2 - B2;
    T s = sqrt(A0 * A0 + A1 * A1 + A2 * A2) + sqrt(B0 * B0 + B1 * B1 + B2 * B2) +
          sqrt(C0 * C0 + C1 * C1 + C2 * C2) + sqrt(D0 * D0 + D1 * D1 + D2 * D2);
    T v6 = fabs(e1[0] * C0 + e1[1] * C1 + e1[2] * C2);
    return T(2) * v6 / s;
}

// Exact FP64 CFL value of one element, min(L_ref, L(X+u)) / c, for the elements
// the FP32 screen keeps (solvers.cpp:296-320), by four lanes of a warp (q = lane
// & 3, all four with the same e): lane q loads node q and takes one face, so
// the chain of FP64 instructions -- 68 cycles each, whatever the number of
// active lanes -- is half that of one lane doing the four faces.  All 32 lanes
// call this together; `pairs`: u as (hi, lo) pairs.  Every lane gets the value.
__device__ __forceinline__ double cfl_quad(const Problem &p, long long e, bool pairs)
{
    const long long nn = p.nn;
    const int q = threadIdx.x & 3;
    const int4 cn = p.conn[e];
    const int nd = q == 0 ? cn.x : (q == 1 ? cn.y : (q == 2 ? cn.z : cn.w));
    const double Lr = p.Lref[e], c = mat_of(p, e).c;
    double x[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        double u;
        if (pairs) {
            const float2 w = p.uhl[k * nn + nd];
            u = (double)w.x + (double)w.y;
        } else {
            u = p.u[k * nn + nd];
        }
        x[k] = p.X[k * nn + nd] + u;
    }
    // lanes 0-2: e1 x e2, e1 x e3, e2 x e3; lane 3 the fourth face, (e2 - e1) x
    // (e3 - e1) as their sum e2 x e3 + e1 x e2 - e1 x e3 (char_length_edges, with
    // its products and sums spelled out so that every caller gets the same bits)
    const int ia = q < 2 ? 1 : 2, ib = q == 0 ? 2 : 3;
    double a[3], b[3], d[3], f[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double e0 = __shfl_sync(0xffffffffu, x[k], 0, 4), w = x[k] - e0;   // edge q
        a[k] = __shfl_sync(0xffffffffu, w, ia, 4);
        b[k] = __shfl_sync(0xffffffffu, w, ib, 4);
        d[k] = __shfl_sync(0xffffffffu, w, 1, 4);
    }
    f[0] = fma(a[1], b[2], -__dmul_rn(a[2], b[1]));
    f[1] = fma(a[2], b[0], -__dmul_rn(a[0], b[2]));
    f[2] = fma(a[0], b[1], -__dmul_rn(a[1], b[0]));
    const double v6 = __shfl_sync(0xffffffffu, fabs(fma(d[2], f[2], fma(d[0], f[0], __dmul_rn(d[1], f[1])))), 2, 4);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double A = __shfl_sync(0xffffffffu, f[k], 0, 4), B = __shfl_sync(0xffffffffu, f[k], 1, 4),
                     C = __shfl_sync(0xffffffffu, f[k], 2, 4);
        if (q == 3) f[k] = __dadd_rn(__dadd_rn(C, A), -B);
    }
    const double r = sqrt(fma(f[2], f[2], fma(f[0], f[0], __dmul_rn(f[1], f[1]))));
    double s = __dadd_rn(__shfl_sync(0xffffffffu, r, 0, 4), __shfl_sync(0xffffffffu, r, 1, 4));
    s = __dadd_rn(s, __shfl_sync(0xffffffffu, r, 2, 4));
    s = __dadd_rn(s, __shfl_sync(0xffffffffu, r, 3, 4));
    const double dist = __dmul_rn(2.0, v6) / s;
    return ((dist < Lr) ? dist : Lr) / c;
}

// The same value, bit for bit, by one lane: half the instructions of four lanes
// an element, for blocks with candidates for every lane.
static __device__ __noinline__ double cfl_lane(const Problem &p, long long e, bool pairs)
{
    const long long nn = p.nn;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double x0[3], e1[3], e2[3], e3[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        double x[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            double u;
            if (pairs) {
                const float2 w = p.uhl[k * nn + nd[q]];
                u = (double)w.x + (double)w.y;
            } else {
                u = p.u[k * nn + nd[q]];
            }
            x[q] = p.X[k * nn + nd[q]] + u;
        }
        x0[k] = x[0];
        e1[k] = x[1] - x0[k];
        e2[k] = x[2] - x0[k];
        e3[k] = x[3] - x0[k];
    }
    const auto face = [](const double *a, const double *b, double *f) {
        f[0] = fma(a[1], b[2], -__dmul_rn(a[2], b[1]));
        f[1] = fma(a[2], b[0], -__dmul_rn(a[0], b[2]));
        f[2] = fma(a[0], b[1], -__dmul_rn(a[1], b[0]));
    };
    const auto norm = [](const double *f) { return sqrt(fma(f[2], f[2], fma(f[0], f[0], __dmul_rn(f[1], f[1])))); };
    double A[3], B[3], C[3], D[3];
    face(e1, e2, A);
    face(e1, e3, B);
    face(e2, e3, C);
#pragma unroll
    for (int k = 0; k < 3; k++) D[k] = __dadd_rn(__dadd_rn(C[k], A[k]), -B[k]);
    const double v6 = fabs(fma(e1[2], C[2], fma(e1[0], C[0], __dmul_rn(e1[1], C[1]))));
    double s = __dadd_rn(norm(A), norm(B));
    s = __dadd_rn(s, norm(C));
    s = __dadd_rn(s, norm(D));
    const double dist = __dmul_rn(2.0, v6) / s, Lr = p.Lref[e];
    return ((dist < Lr) ? dist : Lr) / mat_of(p, e).c;
}

// x rounded toward zero to FP32 with integer operations only (the FP64->FP32
// conversion instruction would take the FP64 pipe): relative error below
// 2^-23 in FP32's normal range, signed zero below it, signed infinity above.
__device__ __forceinline__ float f32_trunc(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned sign = hi & 0x80000000u;
    const int ex = (int)((hi >> 20) & 0x7FFu) - (1023 - 127);
    const unsigned mant = ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    const unsigned r = ex <= 0 ? sign : (ex >= 255 ? (sign | 0x7F800000u) : (sign | ((unsigned)ex << 23) | mant));
    return __uint_as_float(r);
}

// The gate before the CFL screen.  An element whose nodes moved by at most d
// relative to its first node keeps an inscribed sphere of diameter
// L_ref - 2 d: ||F - I|| <= sum_b |u_b - u_0| / h_b <= max_b |u_b - u_0| / r
// (heights h_b, 1/r = sum of the four 1/h), and the reference sphere of radius
// r goes to an ellipsoid with half axes of at least (1 - ||F - I||) r inside
// the tet.  gate = that bound with ||F - I||_F at hand, or with max |u_b - u_0|,
// over the sound speed.  Elements above (1 + 2^-8) times the solve's running
// minimum cannot hold the step's minimum and skip the screen: about 200 FP32
// instructions an element, for 12 to 30.  A reference sliver (negative Lref32)
// and NaN never skip it.  Element kernels with and without: mixed, 6M tets 0.164
// and 0.185 ms; reference order, 384 K tets 0.208 and 0.247; FP64, 6M tets 0.621
// and 0.647; double-word, 1.57M tets 0.1165 and 0.1214.  (On a mesh of equal
// elements everything is near the minimum and passes to the screen as before.)
__device__ __forceinline__ float gate_frobenius(float Lr, float hh, float inv_c)
{
    float s;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(hh));
    // the margin covers sqrt.approx and the rounding of H; s times |L_ref|, so that no motion makes a sliver's
    // negative length a large gate
    return (Lr * 0.9995f - fabsf(Lr) * s) * inv_c;
}

__device__ __forceinline__ float gate_moved(float Lr, float d, float inv_c) { return (Lr - 2.002f * d) * inv_c; }

// An upper bound of max_k |x_k| of FP64 values from the largest of their high
// words m; infinite (or NaN) when it leaves FP32's range.
__device__ __forceinline__ float abs_bound_hi(int m)
{
    // high word: 11 exponent bits biased by 1023, 20 of the mantissa's; modulo 2^32
    const unsigned f = ((unsigned)(m + 1) << 3) - ((unsigned)(1023 - 127) << 23);
    return m >= ((1023 + 100) << 20) ? INFINITY : (m <= ((1023 - 100) << 20) ? 0x1p-99f : __uint_as_float(f));
}

template <int N>
__device__ __forceinline__ float abs_bound(const double *x)
{
    int m = 0;
#pragma unroll
    for (int k = 0; k < N; k++) m = max(m, abs_hi(x[k]));
    return abs_bound_hi(m);
}

// FP32 estimate of an element's CFL value: the reference edges X_b - X_0 are
// the columns of G^-1 (g: the rows of G, the gradients of shape functions
// 1-3, in FP32), cof(G)^T / det G, plus the displacement differences du.  Its
// relative error stays below ~3e-4 unless the tet is a sliver (6V below
// 0.063 |e1||e2||e3|, where the FP32 inverse loses accuracy) or a reference
// sliver (a negative Lref32, set at set-up); those are returned as -1 so that
// the caller always recomputes them in FP64.  The same screen as the mixed
// kernel's, with no streamed edge data.
__device__ __forceinline__ float cfl_screen_edges(const Problem &p, long long e, const float *e1, const float *e2,
                                                  const float *e3, const MatParams &m)
{
    const float C0 = e2[1] * e3[2] - e2[2] * e3[1], C1 = e2[2] * e3[0] - e2[0] * e3[2],
                C2 = e2[0] * e3[1] - e2[1] * e3[0];
    const float v6 = fabsf(e1[0] * C0 + e1[1] * C1 + e1[2] * C2);
    const float l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
    const float l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
    const float l3 = e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2];
    const float dist = char_length_edges<float>(e1, e2, e3);
    const float Lr = __ldg(p.Lref32 + e);
    const float dt = ((dist < Lr) ? dist : Lr) * m.inv_c_f;
    const bool sliver = !(v6 * v6 >= 4e-3f * l1 * l2 * l3) || !(dt > 0.0f);
    return sliver ? -1.0f : dt;
}

__device__ __forceinline__ float cfl_screen(const Problem &p, long long e, const float *g, const float *du,
                                            const MatParams &m)
{
    float C[9];
    C[0] = g[4] * g[8] - g[5] * g[7];
    C[1] = g[5] * g[6] - g[3] * g[8];
    C[2] = g[3] * g[7] - g[4] * g[6];
    C[3] = g[2] * g[7] - g[1] * g[8];
    C[4] = g[0] * g[8] - g[2] * g[6];
    C[5] = g[1] * g[6] - g[0] * g[7];
    C[6] = g[1] * g[5] - g[2] * g[4];
    C[7] = g[2] * g[3] - g[0] * g[5];
    C[8] = g[0] * g[4] - g[1] * g[3];
    const float idet = 1.0f / (g[0] * C[0] + g[1] * C[1] + g[2] * C[2]);
    float e1[3], e2[3], e3[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        e1[i] = C[i] * idet + du[i];
        e2[i] = C[3 + i] * idet + du[3 + i];
        e3[i] = C[6 + i] * idet + du[6 + i];
    }
    return cfl_screen_edges(p, e, e1, e2, e3, m);
}

// What the fixed-point bodies return for an element they leave to FP64
// (elem_left_out), whose forces are not written yet.
constexpr float kLeftOut = -2.0f;

// 2^k in FP32, infinite outside its normal range
__device__ __forceinline__ float pow2f_or_inf(int k)
{
    return k >= -126 && k <= 127 ? __int_as_float((k + 127) << 23) : INFINITY;
}

// x 2^k for an integer x: the exponent is added to the converted integer's
// (|x| < 2^63 and -900 <= k <= 900, so the result is a normal number or zero)
__device__ __forceinline__ double fixed_to_double(long long x, int k)
{
    const double d = __ll2double_rn(x);
    const int hi = __double2hiint(d);
    return __hiloint2double(hi ? hi + (k << 20) : 0, __double2loint(d));
}

template <bool DEP>
__device__ __forceinline__ void gather_u4(const double *u4, const int *nd, double (*ua)[3])
{
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const double2 xy = ld_step<DEP>(reinterpret_cast<const double2 *>(u4) + 2LL * nd[a]);
        ua[a][0] = xy.x;
        ua[a][1] = xy.y;
        ua[a][2] = ld_step<DEP>(u4 + 4LL * nd[a] + 2);
    }
}

// The displacements of an element's four nodes.
template <bool FORCE_ONLY>
__device__ __forceinline__ void gather_u(const Problem &p, const int *nd, double (*ua)[3])
{
    if (!FORCE_ONLY && p.u4 && !p.dependent) {
        gather_u4<false>(p.u4, nd, ua);
    } else if (!FORCE_ONLY && p.u4) {
        gather_u4<true>(p.u4, nd, ua);
    } else {
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int i = 0; i < 3; i++) ua[a][i] = p.u[nd[a] + i * p.nn];
    }
}

// The corner forces of fixed-point sums f[3(a-1) + i], a = 1..3, in units of
// 2^(x0 - lw_a); f_0 = -(f_1 + f_2 + f_3) in FP64.
template <bool FORCE_ONLY>
__device__ __forceinline__ void store_fixed_forces(const Problem &p, long long e, int parity, const FixedElem &q,
                                                   const int64_t *f)
{
    if (!FORCE_ONLY && e == 0 && !isfinite(p.u[1])) atomicOr(p.flags + (parity ^ 1), 1);
    const int4 sl = __ldg(p.slot + e);
    const int ks[4] = {sl.x, sl.y, sl.z, sl.w};
    double fa[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int i = 0; i < 3; i++) fa[a][i] = fixed_to_double(f[a * 3 + i], q.x0 - q.lw[a]);
    st_slot24(p.fe, ks[0], -(fa[0][0] + fa[1][0] + fa[2][0]), -(fa[0][1] + fa[1][1] + fa[2][1]),
              -(fa[0][2] + fa[1][2] + fa[2][2]));
#pragma unroll
    for (int a = 0; a < 3; a++) st_slot24(p.fe, ks[a + 1], fa[a][0], fa[a][1], fa[a][2]);
}

// Plain FP64 mode, compressible neo-Hookean: the deformed edges
// e_b = E_b + (u_b - u_0) and the corner forces from them in 64-bit fixed point
// (msx_fixed.cuh), rounded to FP64 at the end; nine conversions and the six
// additions of f_0 are left to the FP64 pipe, against 115 operations of the same
// formulas in FP64.
// Per warp of 32 elements on the 6M-tet cube (ncu): 115 FP64 instructions and
// 1020 others took 1.290 ms, FP64 pipe 86 % busy; now 18 and 1350 take 0.450 ms,
// ALU pipe 49 % busy.
template <bool FORCE_ONLY>
__device__ __forceinline__ float elem_body_fp64_cnh(const Problem &p, long long e, int parity, const MatParams &m,
                                                    const int *nd, float gmin)
{
    const long long ne = p.ne;
    double ua[4][3];
    gather_u<FORCE_ONLY>(p, nd, ua);
    const uint2 w = __ldg(p.fxw + e);
    if (w.x == 0) return kLeftOut;
    FixedElem q;
    fixed_unpack(w.x, w.y, q);
#pragma unroll
    for (int k = 0; k < 9; k++) q.E[k] = __ldg(p.fxE + k * ne + e);
    Limbs n[9];
    int moved;
    if (!fixed_edges(q, ua, n, moved)) return kLeftOut;
    float scr = INFINITY;
    if (!FORCE_ONLY && !(gate_moved(__ldg(p.Lref32 + e), 1.7321f * ((float)moved * pow2f_or_inf(fixed_lw_min(q) + 32)), m.inv_c_f) > gmin)) {
        float e32[9];
#pragma unroll
        for (int k = 0; k < 9; k++) e32[k] = (float)n[k].h * pow2f_or_inf(q.lw[k / 3] + 29);
        scr = cfl_screen_edges(p, e, e32, e32 + 3, e32 + 6, m);
    }
    const longlong2 dd = __ldg(p.fxD + e);
    q.d0 = dd.x;
    q.rd = dd.y;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const int2 x = __ldg(p.fxS + k * ne + e);
        q.S[k] = {x.x, x.y};
    }
    int64_t f[9];
    if (!fixed_forces(q, n, m.kq, [&](double J) { return (int64_t)__double2ll_rn((m.mu - m.lambda * log(J)) * m.ksw / J); }, f))
        return kLeftOut;
    store_fixed_forces<FORCE_ONLY>(p, e, parity, q, f);
    return scr;
}

// Plain FP64 mode, St-Venant-Kirchhoff and linear elasticity: the node
// differences, the displacement gradient and the stress in 64-bit fixed point
// (msx_fixed.cuh); 99 products of limb pairs in place of about 190 FP64
// operations.  264,000 shuffled tets, StVK: 86 us in FP64, the FP64 pipe its
// bound, 44 us now, bound by the integer pipes and the scattered slot writes.
// ACT: element birth, whose dead elements have no force.
template <bool FORCE_ONLY, bool ACT>
__device__ __forceinline__ float elem_body_fp64_svk(const Problem &p, long long e, int parity, double t,
                                                    const MatParams &m, const int *nd, float gmin)
{
    const long long ne = p.ne;
    double ua[4][3];
    gather_u<FORCE_ONLY>(p, nd, ua);
    const uint2 w = __ldg(p.fxw + e);
    if (w.x == 0) return kLeftOut;
    FixedElem q;
    fixed_unpack(w.x, w.y, q);
#pragma unroll
    for (int k = 0; k < 9; k++) q.E[k] = __ldg(p.fxE + k * ne + e);
    q.S[0] = limbs_unpack(__ldg(&p.fxD[e].x));
    double x[9];
    int hi = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        x[k] = ua[k / 3 + 1][k % 3] - ua[0][k % 3];
        hi = max(hi, abs_hi(x[k]));
    }
    float scr = INFINITY;
    if (!FORCE_ONLY && !(gate_moved(__ldg(p.Lref32 + e), 1.7321f * abs_bound_hi(hi), m.inv_c_f) > gmin)) {
        float du32[9], g32[9];
#pragma unroll
        for (int k = 0; k < 9; k++) {
            du32[k] = f32_trunc(x[k]);
            g32[k] = (float)limbs_unpack(q.E[k]).h * pow2f_or_inf(29 - 111 + (q.cs >> 2) - q.lw[0]);
        }
        scr = cfl_screen(p, e, g32, du32, m);
    }
    Limbs du[9];
    int64_t f[9];
    int s;
    if (!fixed_motion(q, x, hi, m.law == 3, du, s) || !fixed_forces_svk(q, du, m.law == 3, m.kq[0], m.ks, f, s))
        return kLeftOut;
    q.x0 += s;
    if (ACT && elem_dead(p, e, t))
#pragma unroll
        for (int k = 0; k < 9; k++) f[k] = 0;
    store_fixed_forces<FORCE_ONLY>(p, e, parity, q, f);
    return scr;
}

// Plain FP64 with contraction: H from node differences, laws through the
// cofactor (F C^-1 = F^-T = cof(F)/J), wJ folded into the law's coefficients,
// the 4th corner force as minus the sum of the other three.  Same algebra as
// the reference, about half its FP64 operations.  Returns the FP32 CFL screen
// value (see cfl_screen).
template <bool FORCE_ONLY, bool ACT, bool VISC>
__device__ __forceinline__ float elem_cofactor_fp64(const Problem &p, long long e, int parity, double t, double idt,
                                                    const MatParams &m, const int *nd, const double *G, float gmin)
{
    double ua[4][3], du[9];
    gather_u<FORCE_ONLY>(p, nd, ua);
#pragma unroll
    for (int a = 1; a < 4; a++)
#pragma unroll
        for (int i = 0; i < 3; i++) du[(a - 1) * 3 + i] = ua[a][i] - ua[0][i];
    double F[9], P[9];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            // the identity enters the FMA chain (no separate 0 + x or 1 + x)
            F[i * 3 + j] = fma(du[i], G[j], fma(du[3 + i], G[3 + j], i == j ? fma(du[6 + i], G[6 + j], 1.0)
                                                                             : du[6 + i] * G[6 + j]));
    float scr = INFINITY;
    // the CFL screen first, so du dies before the stress
    if (!FORCE_ONLY && !(gate_moved(__ldg(p.Lref32 + e), 1.7321f * abs_bound<9>(du), m.inv_c_f) > gmin)) {
        float du32[9], g32[9];
#pragma unroll
        for (int k = 0; k < 9; k++) {
            du32[k] = f32_trunc(du[k]);
            g32[k] = f32_trunc(G[k]);
        }
        scr = cfl_screen(p, e, g32, du32, m);
    }
    stress_fast(m, F, __ldg(p.wJ + e), P);
    if (VISC && !FORCE_ONLY) {
        double Pv[9];
        visc_bulk_fp64(p, e, F, __ldg(p.wJ + e), m.rho, idt, Pv);
#pragma unroll
        for (int k = 0; k < 9; k++) P[k] += Pv[k];
    }
    double f[12];
#pragma unroll
    for (int a = 1; a < 4; a++)
#pragma unroll
        for (int i = 0; i < 3; i++)
            f[a * 3 + i] = P[i * 3] * G[(a - 1) * 3] + P[i * 3 + 1] * G[(a - 1) * 3 + 1] + P[i * 3 + 2] * G[(a - 1) * 3 + 2];
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = -(f[3 + i] + f[6 + i] + f[9 + i]);
    if (ACT && elem_dead(p, e, t))
#pragma unroll
        for (int k = 0; k < 12; k++) f[k] = 0.0;
    const int4 sl = __ldg(p.slot + e);
    const int ks[4] = {sl.x, sl.y, sl.z, sl.w};
#pragma unroll
    for (int a = 0; a < 4; a++) st_slot24(p.fe, ks[a], f[a * 3], f[a * 3 + 1], f[a * 3 + 2]);
    if (FORCE_ONLY) return 0.0f;
    if (e == 0 && !isfinite(p.u[1])) atomicOr(p.flags + (parity ^ 1), 1);
    return scr;
}

__device__ __forceinline__ void load_G(const Problem &p, long long e, double *G)
{
#pragma unroll
    for (int k = 0; k < 9; k++) G[k] = __ldg(p.G + k * p.ne + e);
}

// An element that fixed point leaves out, in the FP64 cofactor form.  The form
// from the deformed edges (f_a = sum_b S_ab e_b + c2 e_c x e_d, 110 operations
// for 130) is a little faster, but compressible neo-Hookean elements are left
// out because they are flat, and there its error is 5 to 10 times this one's
// (hexes of 1:1:0.1, strain 1e-4: 2e-11 to 4e-11 of the forces, 4e-12 here).
// One function for all kernels: which product of a b + c d is fused is the
// compiler's choice, and would differ between instantiations.
template <bool FORCE_ONLY, bool ACT>
static __device__ __noinline__ float elem_left_out(const Problem &p, long long e, int parity, double t, float gmin)
{
    const long long ne = p.ne;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    const MatParams &m = mat_of(p, e);
    double G[9];
    if (m.law == 1) {
        load_G(p, e, G);
    } else {   // the gradients, FP64 bits or limbs of w g 2^(111 - gs)
        const uint2 w = __ldg(p.fxw + e);
        FixedElem q;
        fixed_unpack(w.x, w.y, q);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const long long x = __ldg(p.fxE + k * ne + e);
            const Limbs g = limbs_unpack(x);
            G[k] = w.x == 0 ? bits_double((uint64_t)x)
                            : fixed_to_fp64(((int64_t)g.h << 29) + g.l, (q.cs >> 2) - 111 - q.lw[0]);
        }
    }
    return elem_cofactor_fp64<FORCE_ONLY, ACT, false>(p, e, parity, t, 0.0, m, nd, G, gmin);
}

template <bool FORCE_ONLY, bool ACT = false, bool VISC = false, int FIXED = FIXED_NONE>
__device__ __forceinline__ float elem_body_fp64(const Problem &p, long long e, int parity, double t = 0.0,
                                                double idt = 0.0, float gmin = 0.0f, int4 cn_ahead = make_int4(0, 0, 0, 0))
{
    const int4 cn = FIXED ? cn_ahead : p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    const MatParams &m = mat_of(p, e);
    if (FIXED == FIXED_CNH || (!FIXED && !VISC && p.fxE && m.law == 1))   // never dead
        return elem_body_fp64_cnh<FORCE_ONLY>(p, e, parity, m, nd, gmin);
    if (FIXED == FIXED_SVK || (!VISC && p.fxE && m.law >= 2))
        return elem_body_fp64_svk<FORCE_ONLY, ACT>(p, e, parity, t, m, nd, gmin);
    double G[9];
    load_G(p, e, G);
    return elem_cofactor_fp64<FORCE_ONLY, ACT, VISC>(p, e, parity, t, idt, m, nd, G, gmin);
}

// corner forces only (internal-force hook); three CTAs an SM in spite of the
// registers of the left-out elements' FP64 form (80 instead of 114: a call of
// 1.3M tets 334 us, 341 with two, 322 with that form inside the warps)
static __global__ void __launch_bounds__(kElemBlock, 3) elem_force_kernel_fp64(Problem p, int parity)
{
    __shared__ int left[kElemBlock], s_nleft;   // left out by fixed point: by consecutive threads at the end
    if (threadIdx.x == 0) s_nleft = 0;
    __syncthreads();
    const long long b = (long long)blockIdx.x * blockDim.x, e = b + threadIdx.x;
    if (e < p.ne && elem_body_fp64<true>(p, e, parity) == kLeftOut) left[atomicAdd(&s_nleft, 1)] = threadIdx.x;
    __syncthreads();
    if ((int)threadIdx.x < s_nleft) elem_left_out<true, false>(p, b + left[threadIdx.x], parity, 0.0, 0.0f);
}

// ---------------------------------------------------------------------------
// Mixed precision: FP32 kinematics, stress and B^T P written in terms of the
// displacement gradient H = F - I (no 1 - 1 cancellation in FP32); J - 1 and
// ln J in FP32 with an exactly summed trace; FP32 corner forces; an FP32
// screen of the CFL values whose near-minimum elements are recomputed in FP64
// (cfl_quad), so the stable dt is the FP64 minimum.
// cof(I + H) = I + D with D = (tr H + I2) I - (1 + tr H) H^T + (H^2)^T.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void stress_mixed(const MatParams &m, const float *H, float Jm1, float lnJ,
                                             float t, float I2, float *P)
{
    if (m.law == 3) {
        // linear elastic: P = mu2 E + lam tr(E) I with E = (H + H^T)/2
        const float dg = m.lam_stvk_f * t;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                P[i * 3 + j] = m.mu2_f * (0.5f * (H[i * 3 + j] + H[j * 3 + i])) + (i == j ? dg : 0.0f);
        return;
    }
    if (m.law == 2) {
        // E = (H + H^T + H^T H)/2, S = mu2 E + lam tr(E) I, P = (I + H) S
        float E[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                E[i * 3 + j] = 0.5f * (H[i * 3 + j] + H[j * 3 + i] +
                                       (H[i] * H[j] + H[3 + i] * H[3 + j] + H[6 + i] * H[6 + j]));
        float trE = E[0] + E[4] + E[8];
        float S[9];
#pragma unroll
        for (int k = 0; k < 9; k++) S[k] = m.mu2_f * E[k];
        S[0] += m.lam_stvk_f * trE;
        S[4] += m.lam_stvk_f * trE;
        S[8] += m.lam_stvk_f * trE;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                P[i * 3 + j] = S[i * 3 + j] + (H[i * 3] * S[j] + H[i * 3 + 1] * S[3 + j] + H[i * 3 + 2] * S[6 + j]);
        return;
    }
    // Products and sums are spelled out (fmaf, _rn) from here on: which product
    // of a*b + c*d is fused is otherwise the compiler's choice, and differs
    // between the instantiations of this body; a pooled solve has to give the
    // bits of the solve run alone.
    float D[9];
    const float a0 = t + I2, a1 = 1.0f + t;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            // (H^2)^T_ij = sum_k H_jk H_ki
            const float x = H[j * 3], X = H[i], y = H[j * 3 + 1], Y = H[3 + i], z = H[j * 3 + 2], Z = H[6 + i];
            float h2;
            if (i == 0 && j == 0) h2 = __fadd_rn(fmaf(x, X, __fmul_rn(y, Y)), __fmul_rn(z, Z));
            else if (i == 1 && j == 1) h2 = __fadd_rn(fmaf(y, Y, __fmul_rn(x, X)), __fmul_rn(z, Z));
            else if (i == 2 && j == 2) h2 = fmaf(z, Z, __fadd_rn(__fmul_rn(x, X), __fmul_rn(y, Y)));
            else h2 = fmaf(z, Z, fmaf(x, X, __fmul_rn(y, Y)));
            D[i * 3 + j] = __fadd_rn(i == j ? fmaf(-a1, H[j * 3 + i], a0) : -__fmul_rn(a1, H[j * 3 + i]), h2);
        }
    const float Jx = 1.0f + Jm1, iJ = 1.0f / Jx;
    if (m.law == 1) {
        // P = [mu (Jm1 I + (1+Jm1) H - D) + lambda lnJ (I + D)] / J
        const float lj = __fmul_rn(m.lambda_f, lnJ);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const float q = __fadd_rn(k % 4 == 0 ? fmaf(Jx, H[k], Jm1) : __fmul_rn(Jx, H[k]), -D[k]);
            P[k] = __fmul_rn(fmaf(lj, k % 4 == 0 ? __fadd_rn(1.0f, D[k]) : D[k], __fmul_rn(m.mu_f, q)), iJ);
        }
    } else {
        // P = mu J^-2/3 [(Jm1 - beta) I + (1+Jm1) H - (1+beta) D]/J + K Jm1 (I + D), beta = b3 / 3
        float hh = 0.0f;
#pragma unroll
        for (int k = 0; k < 9; k++) hh = fmaf(H[k], H[k], hh);
        const float b3 = fmaf(2.0f, t, hh), b1 = fmaf(b3, 1.0f / 3.0f, 1.0f), Jb = fmaf(-b3, 1.0f / 3.0f, Jm1);
        const float j23 = __fmul_rn(__fmul_rn(expf(__fmul_rn(-(2.0f / 3.0f), lnJ)), m.mu_f), iJ);
        const float kj = __fmul_rn(m.K1_f, Jm1);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const float q = fmaf(-b1, D[k], k % 4 == 0 ? fmaf(Jx, H[k], Jb) : __fmul_rn(Jx, H[k]));
            P[k] = fmaf(kj, k % 4 == 0 ? __fadd_rn(1.0f, D[k]) : D[k], __fmul_rn(j23, q));
        }
    }
}

template <bool FORCE_ONLY, bool ACT = false, bool VISC = false>
__device__ __forceinline__ float elem_body_mixed(const Problem &p, long long e, int parity, int4 cn, double t = 0.0,
                                                 float idtf = 0.0f, float gmin = 0.0f)
{
    const long long ne = p.ne, nn = p.nn;
    float vmin = INFINITY;
    {
        int nd[4] = {cn.x, cn.y, cn.z, cn.w};
        float G[9];
#pragma unroll
        for (int k = 0; k < 9; k++) G[k] = __ldg(p.G32 + k * ne + e);
        // du = u_a - u_0 from the (hi, lo) split: the hi difference is exact for
        // nearby values, the lo difference restores the bits FP32 drops
        float2 h0[3];
#pragma unroll
        for (int i = 0; i < 3; i++) h0[i] = p.uhl[nd[0] + i * nn];
        float du[9];
#pragma unroll
        for (int a = 1; a < 4; a++)
#pragma unroll
            for (int i = 0; i < 3; i++) {
                float2 ha = p.uhl[nd[a] + i * nn];
                du[(a - 1) * 3 + i] = (ha.x - h0[i].x) + (ha.y - h0[i].y);
            }
        float H[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                H[i * 3 + j] = fmaf(du[6 + i], G[6 + j], fmaf(du[i], G[j], __fmul_rn(du[3 + i], G[3 + j])));
        // J - 1 = tr H + (I2(H) + det H).  The trace carries J - 1 and may
        // cancel (nearly isochoric motion), so it is summed without rounding,
        // as s + err by TwoSum; I2 and det H are O(|H|^2) and their FP32
        // rounding lies far below the FP32 precision of J - 1.  So J - 1 is
        // good to FP32 relative precision, and so is ln J = log1p(J - 1);
        // F = I + H is never formed or reduced.
        float hh = 0.0f;   // ||H||_F^2, for the CFL gate
#pragma unroll
        for (int k = 0; k < 9; k++) hh = fmaf(H[k], H[k], hh);
        float tf = H[0] + H[4] + H[8];
        // spelled out, as in stress_mixed
        const float m48 = fmaf(H[4], H[8], -__fmul_rn(H[5], H[7])), m38 = fmaf(H[3], H[8], -__fmul_rn(H[5], H[6])),
                    m37 = fmaf(H[3], H[7], -__fmul_rn(H[4], H[6]));
        const float I2f = __fadd_rn(__fadd_rn(fmaf(H[0], H[4], -__fmul_rn(H[1], H[3])), m48),
                                    fmaf(H[0], H[8], -__fmul_rn(H[2], H[6])));
        const float I3f = fmaf(H[2], m37, fmaf(H[0], m48, -__fmul_rn(H[1], m38)));
        const float s1 = H[0] + H[4], s2 = s1 + H[8];
        const float terr = two_sum_err(H[0], H[4], s1) + two_sum_err(s1, H[8], s2);
        const float Jm1 = s2 + (terr + (I2f + I3f));
        const float lnJ = log1pf(Jm1);
        const MatParams &m = mat_of(p, e);
        float P[9];
        stress_mixed(m, H, Jm1, lnJ, tf, I2f, P);
        if (VISC && !FORCE_ONLY) {
            // bulk viscosity in FP32: P += qBV cof(I + H) = qBV (I + D), D as in stress_mixed
            float *h0 = p.visc_h0;
            const float trD = ((H[0] - h0[e]) + (H[4] - h0[ne + e]) + (H[8] - h0[2 * ne + e])) * idtf;
            h0[e] = H[0];
            h0[ne + e] = H[4];
            h0[2 * ne + e] = H[8];
            const float q = m.rho_f / (1.0f + Jm1) * p.visc_hf *
                            (p.visc_c1sq_hf * fabsf(trD) * fminf(0.0f, trD) + p.visc_clc0f * trD);
            const float a0 = tf + I2f, a1 = 1.0f + tf;
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const float h2 = H[j * 3] * H[i] + H[j * 3 + 1] * H[3 + i] + H[j * 3 + 2] * H[6 + i];
                    const float Dij = (i == j ? a0 : 0.0f) - a1 * H[j * 3 + i] + h2;
                    P[i * 3 + j] += q * ((i == j ? 1.0f : 0.0f) + Dij);
                }
        }
        float wJ = __ldg(p.wJ32 + e);
#pragma unroll
        for (int k = 0; k < 9; k++) P[k] *= wJ;
        float f[12];
#pragma unroll
        for (int a = 1; a < 4; a++)
#pragma unroll
            for (int i = 0; i < 3; i++)
                f[a * 3 + i] = fmaf(P[i * 3 + 2], G[(a - 1) * 3 + 2],
                                    fmaf(P[i * 3], G[(a - 1) * 3], __fmul_rn(P[i * 3 + 1], G[(a - 1) * 3 + 1])));
#pragma unroll
        for (int i = 0; i < 3; i++) f[i] = -(f[3 + i] + f[6 + i] + f[9 + i]);
        if (ACT && elem_dead(p, e, t))
#pragma unroll
            for (int k = 0; k < 12; k++) f[k] = 0.f;
        // one 16-byte store per corner (a padded slot) rather than three scalar ones
        const int4 sl = __ldg(p.slot + e);
        float4 *fe = reinterpret_cast<float4 *>(p.fe32);
        fe[sl.x] = make_float4(f[0], f[1], f[2], 0.f);
        fe[sl.y] = make_float4(f[3], f[4], f[5], 0.f);
        fe[sl.z] = make_float4(f[6], f[7], f[8], 0.f);
        fe[sl.w] = make_float4(f[9], f[10], f[11], 0.f);
        if (!FORCE_ONLY && e == 0 && !isfinite(p.uhl[1].x)) atomicOr(p.flags + (parity ^ 1), 1);
        if (!FORCE_ONLY && !(gate_frobenius(__ldg(p.Lref32 + e), hh, m.inv_c_f) > gmin)) {
            // reference edges X_b - X_0 = columns of G^-1 (G's rows are the
            // gradients of shape functions 1-3): cof(G)^T / det G in FP32,
            // instead of streaming them; only the CFL value uses them
            float C[9];
            C[0] = G[4] * G[8] - G[5] * G[7];
            C[1] = G[5] * G[6] - G[3] * G[8];
            C[2] = G[3] * G[7] - G[4] * G[6];
            C[3] = G[2] * G[7] - G[1] * G[8];
            C[4] = G[0] * G[8] - G[2] * G[6];
            C[5] = G[1] * G[6] - G[0] * G[7];
            C[6] = G[1] * G[5] - G[2] * G[4];
            C[7] = G[2] * G[3] - G[0] * G[5];
            C[8] = G[0] * G[4] - G[1] * G[3];
            const float idet = 1.0f / (G[0] * C[0] + G[1] * C[1] + G[2] * C[2]);
            float e1[3], e2[3], e3[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                e1[i] = C[i] * idet + du[i];
                e2[i] = C[3 + i] * idet + du[3 + i];
                e3[i] = C[6 + i] * idet + du[6 + i];
            }
            // FP32 screen of the CFL value, as cfl_screen: slivers (6V below
            // 0.063 |e1||e2||e3|, where the FP32 edges lose accuracy) and
            // reference slivers (a negative Lref32, set at set-up) come back
            // negative, so the caller recomputes them in FP64
            const float C0 = e2[1] * e3[2] - e2[2] * e3[1], C1 = e2[2] * e3[0] - e2[0] * e3[2],
                        C2 = e2[0] * e3[1] - e2[1] * e3[0];
            const float v6 = fabsf(e1[0] * C0 + e1[1] * C1 + e1[2] * C2);
            const float l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
            const float l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
            const float l3 = e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2];
            float dist = char_length_edges<float>(e1, e2, e3);
            float Lr = __ldg(p.Lref32 + e);
            vmin = ((dist < Lr) ? dist : Lr) * m.inv_c_f;
            if (!(v6 * v6 >= 4e-3f * l1 * l2 * l3) || !(vmin > 0.0f)) vmin = -1.0f;
        }
    }
    return vmin;
}

// corner forces only (internal-force hook)
static __global__ void __launch_bounds__(kElemBlock) elem_force_kernel_mixed(Problem p, int parity)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < p.ne) elem_body_mixed<true>(p, e, parity, p.conn[e]);
}


// ---------------------------------------------------------------------------
// Double-word mode: the algebra of elem_body_fp64 (F from node differences,
// the laws through cof(F), B^T P with wJ folded in) evaluated in double-word
// arithmetic on the FP32 pipe, with the nodal state and the corner forces as
// double-words too.  A double-word operation costs 4-20 FP32 operations and
// carries about 2^-47 relative error against FP64's 2^-53; on this GPU the
// FP64 pipe issues 1/64 of the FP32 rate, so the element work runs several
// times faster than in FP64 while results stay within a few 1e-13 of it.
// The error-free pieces (TwoSum, Fast2Sum, the FMA product split) use the
// _rn intrinsics, which the compiler never fuses into an FMA.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float dw_err(float a, float b, float s)   // a + b - s for s = fl(a + b)
{
    const float bb = __fsub_rn(s, a);
    return __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

__device__ __forceinline__ float2 dw_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    return make_float2(s, dw_err(a, b, s));
}

__device__ __forceinline__ float2 dw_fast(float a, float b)   // |a| >= |b| or a = 0
{
    const float s = __fadd_rn(a, b);
    return make_float2(s, __fsub_rn(b, __fsub_rn(s, a)));
}

__device__ __forceinline__ float2 dw_neg(float2 x) { return make_float2(-x.x, -x.y); }
__device__ __forceinline__ float2 dw_scale2(float2 x, float p2) { return make_float2(x.x * p2, x.y * p2); }  // p2 = 2^k

// Joldes, Muller, Popescu (2017) Alg. 6 (accurate sum), Alg. 12 (product),
// Alg. 4 (double-word + FP32), Alg. 9 (double-word * FP32).
__device__ __forceinline__ float2 dw_add(float2 x, float2 y)
{
    const float2 s = dw_two_sum(x.x, y.x), t = dw_two_sum(x.y, y.y);
    const float2 v = dw_fast(s.x, __fadd_rn(s.y, t.x));
    return dw_fast(v.x, __fadd_rn(t.y, v.y));
}

// x + y with absolute error a few 2^-48 (|x| + |y|) (the "sloppy" sum, JMP
// Alg. 5): enough where the inputs' own rounding is of that size, as for node
// differences and sums of corner forces; no bound relative to |x + y|.
__device__ __forceinline__ float2 dw_add_sloppy(float2 x, float2 y)
{
    const float2 s = dw_two_sum(x.x, y.x);
    return dw_fast(s.x, __fadd_rn(s.y, __fadd_rn(x.y, y.y)));
}

__device__ __forceinline__ float2 dw_mul(float2 x, float2 y)
{
    const float ch = __fmul_rn(x.x, y.x);
    const float cl1 = fmaf(x.x, y.x, -ch);
    const float cl2 = fmaf(x.y, y.x, fmaf(x.x, y.y, __fmul_rn(x.y, y.y)));
    return dw_fast(ch, __fadd_rn(cl1, cl2));
}

__device__ __forceinline__ float2 dw_add_f(float2 x, float y)
{
    const float2 s = dw_two_sum(x.x, y);
    return dw_fast(s.x, __fadd_rn(x.y, s.y));
}

__device__ __forceinline__ float2 dw_mul_f(float2 x, float y)
{
    const float ch = __fmul_rn(x.x, y);
    return dw_fast(ch, fmaf(x.y, y, fmaf(x.x, y, -ch)));
}

__device__ __forceinline__ float2 dw_from(double x)
{
    const float hi = (float)x;
    return make_float2(hi, (float)(x - (double)hi));
}

// Compensated dot products of double-words (Ogita, Rump, Oishi, "Accurate sum
// and dot product", SIAM J. Sci. Comput. 26 (2005), Dot2, with the low words'
// cross terms): each hi*hi product is split exactly by an FMA and summed with
// TwoSum; the product and sum errors and the hi*lo terms gather in one FP32
// correction c.  Result s + c by Fast2Sum (exact unless the sum cancels below
// |c|, where its error is still of the order 2^-48 sum |a_k b_k|); error a few
// 2^-48 sum |a_k b_k|, the size of FP64's 2^-53 sum |a_k b_k| times ~30.
__device__ __forceinline__ void dw_acc(float &s, float &c, float2 x, float2 y)
{
    const float p = __fmul_rn(x.x, y.x);
    c = fmaf(x.y, y.x, fmaf(x.x, y.y, c + fmaf(x.x, y.x, -p)));
    const float t = __fadd_rn(s, p);
    c += dw_err(s, p, t);
    s = t;
}

__device__ __forceinline__ float2 dw_dot2(float2 a0, float2 b0, float2 a1, float2 b1)
{
    float s = __fmul_rn(a0.x, b0.x);
    float c = fmaf(a0.y, b0.x, fmaf(a0.x, b0.y, fmaf(a0.x, b0.x, -s)));
    dw_acc(s, c, a1, b1);
    return dw_fast(s, c);
}

// init + a0 b0 + a1 b1 + a2 b2 (init an FP32 constant, e.g. the identity's 1)
__device__ __forceinline__ float2 dw_dot3(float2 a0, float2 b0, float2 a1, float2 b1, float2 a2, float2 b2,
                                          float init)
{
    float s, c;
    if (init == 0.0f) {   // a constant at every call: resolved at compile time
        s = __fmul_rn(a0.x, b0.x);
        c = fmaf(a0.y, b0.x, fmaf(a0.x, b0.y, fmaf(a0.x, b0.x, -s)));
    } else {
        s = init;
        c = 0.0f;
        dw_acc(s, c, a0, b0);
    }
    dw_acc(s, c, a1, b1);
    dw_acc(s, c, a2, b2);
    return dw_fast(s, c);
}

// ln(1 + x) for a double-word x.  For |x| < 2^-7: x - x^2/2 + x^3/3 in
// double-words plus the tail x^4 (-1/4 + x/5 - x^2/6 + x^3/7 - x^4/8) in FP32
// (|tail| < 2^-21 |x|, so its FP32 rounding stays below 2^-45 |x|; the next
// term is below 2^-56 |x|).  Otherwise the FP64 library log.
__device__ __forceinline__ float2 dw_log1p(float2 x)
{
    if (!(fabsf(x.x) < 0.0078125f)) return dw_from(log(1.0 + ((double)x.x + (double)x.y)));
    const float2 third = make_float2(0x1.555556p-2f, -0x1.555556p-27f);
    const float2 x2 = dw_mul(x, x), x3 = dw_mul(x2, x);
    const float2 lead = dw_add(dw_add(x, dw_scale2(x2, -0.5f)), dw_mul(x3, third));
    const float xf = x.x;
    const float tail = (x2.x * x2.x) * fmaf(xf, fmaf(xf, fmaf(xf, fmaf(xf, -0.125f, 1.0f / 7.0f), -1.0f / 6.0f), 0.2f), -0.25f);
    return dw_add_f(lead, tail);
}

// 1 / y: one Newton step from the FP32 reciprocal.
__device__ __forceinline__ float2 dw_rcp(float2 y)
{
    const float r0 = __frcp_rn(y.x);
    const float2 p = dw_mul_f(y, r0);                       // y r0 = 1 - e
    const float e = __fsub_rn(__fsub_rn(1.0f, p.x), p.y);
    return dw_fast(r0, __fmul_rn(r0, e));
}

// wJ * P through the cofactor, as stress_fast does in FP64.
__device__ __forceinline__ void stress_dw(const MatParams &m, const float2 *F, float2 wJ, float2 *P)
{
    if (m.law == 3) {
        // linear elastic: wJ P = wJ (mu2 E + lam tr(E) I), E = (F + F^T)/2 - I
        const float2 h = dw_mul(m.mu2_w, wJ);
        const float2 E00 = dw_add_f(F[0], -1.0f), E11 = dw_add_f(F[4], -1.0f), E22 = dw_add_f(F[8], -1.0f);
        const float2 dg = dw_mul(dw_mul(m.lam_stvk_w, dw_add(dw_add(E00, E11), E22)), wJ);
        P[0] = dw_add(dw_mul(h, E00), dg);
        P[4] = dw_add(dw_mul(h, E11), dg);
        P[8] = dw_add(dw_mul(h, E22), dg);
        P[1] = P[3] = dw_mul(h, dw_scale2(dw_add(F[1], F[3]), 0.5f));
        P[2] = P[6] = dw_mul(h, dw_scale2(dw_add(F[2], F[6]), 0.5f));
        P[5] = P[7] = dw_mul(h, dw_scale2(dw_add(F[5], F[7]), 0.5f));
        return;
    }
    if (m.law == 2) {
        // S = mu2 E + lam tr(E) I with E = (F^T F - I)/2; C_ii - 1 from the dot's initial -1
        const float2 C00 = dw_dot3(F[0], F[0], F[3], F[3], F[6], F[6], -1.0f);
        const float2 C11 = dw_dot3(F[1], F[1], F[4], F[4], F[7], F[7], -1.0f);
        const float2 C22 = dw_dot3(F[2], F[2], F[5], F[5], F[8], F[8], -1.0f);
        const float2 C01 = dw_dot3(F[0], F[1], F[3], F[4], F[6], F[7], 0.0f);
        const float2 C02 = dw_dot3(F[0], F[2], F[3], F[5], F[6], F[8], 0.0f);
        const float2 C12 = dw_dot3(F[1], F[2], F[4], F[5], F[7], F[8], 0.0f);
        const float2 trE = dw_scale2(dw_add(dw_add(C00, C11), C22), 0.5f);
        const float2 h = dw_scale2(dw_mul(m.mu2_w, wJ), 0.5f), dg = dw_mul(dw_mul(m.lam_stvk_w, trE), wJ);
        const float2 S00 = dw_add(dw_mul(h, C00), dg), S11 = dw_add(dw_mul(h, C11), dg),
                     S22 = dw_add(dw_mul(h, C22), dg);
        const float2 S01 = dw_mul(h, C01), S02 = dw_mul(h, C02), S12 = dw_mul(h, C12);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float2 f0 = F[i * 3], f1 = F[i * 3 + 1], f2 = F[i * 3 + 2];
            P[i * 3 + 0] = dw_dot3(f0, S00, f1, S01, f2, S02, 0.0f);
            P[i * 3 + 1] = dw_dot3(f0, S01, f1, S11, f2, S12, 0.0f);
            P[i * 3 + 2] = dw_dot3(f0, S02, f1, S12, f2, S22, 0.0f);
        }
        return;
    }
    float2 K[9];
    K[0] = dw_dot2(F[4], F[8], dw_neg(F[5]), F[7]);
    K[1] = dw_dot2(F[5], F[6], dw_neg(F[3]), F[8]);
    K[2] = dw_dot2(F[3], F[7], dw_neg(F[4]), F[6]);
    K[3] = dw_dot2(F[2], F[7], dw_neg(F[1]), F[8]);
    K[4] = dw_dot2(F[0], F[8], dw_neg(F[2]), F[6]);
    K[5] = dw_dot2(F[1], F[6], dw_neg(F[0]), F[7]);
    K[6] = dw_dot2(F[1], F[5], dw_neg(F[2]), F[4]);
    K[7] = dw_dot2(F[2], F[3], dw_neg(F[0]), F[5]);
    K[8] = dw_dot2(F[0], F[4], dw_neg(F[1]), F[3]);
    const float2 J = dw_dot3(F[0], K[0], F[1], K[1], F[2], K[2], 0.0f);
    const float2 x = dw_add_f(J, -1.0f);   // J - 1
    const float2 iJ = dw_rcp(J);
    float2 a1, g;
    if (m.law == 1) {
        // P = mu F + (lambda ln J - mu) cof(F) / J
        a1 = dw_mul(m.mu_w, wJ);
        g = dw_mul(dw_mul(dw_add(dw_mul(m.lambda_w, dw_log1p(x)), dw_neg(m.mu_w)), iJ), wJ);
    } else {
        // P = mu J^-2/3 F + (-mu/3 trB J^-5/3 + K1 (J-1)) cof(F); J^-2/3 from the FP64 library
        const double r = rcbrt((double)J.x + (double)J.y);
        const float2 j23 = dw_from(r * r);
        const float2 trB = dw_add(dw_add(dw_dot3(F[0], F[0], F[1], F[1], F[2], F[2], 0.0f),
                                         dw_dot3(F[3], F[3], F[4], F[4], F[5], F[5], 0.0f)),
                                  dw_dot3(F[6], F[6], F[7], F[7], F[8], F[8], 0.0f));
        a1 = dw_mul(dw_mul(m.mu_w, j23), wJ);
        g = dw_mul(dw_add(dw_neg(dw_mul(dw_mul(dw_mul(m.mu3_w, trB), j23), iJ)), dw_mul(m.K1_w, x)), wJ);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) P[k] = dw_dot2(a1, F[k], g, K[k]);
}

template <bool FORCE_ONLY, bool ACT = false, bool VISC = false>
__device__ __forceinline__ float elem_body_dw(const Problem &p, long long e, int parity, int4 cn, double t = 0.0,
                                              double idt = 0.0, float gmin = 0.0f)
{
    const long long ne = p.ne, nn = p.nn;
    int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    float2 G[9];
#pragma unroll
    for (int k = 0; k < 9; k++) G[k] = make_float2(__ldg(p.G32 + k * ne + e), __ldg(p.G32lo + k * ne + e));
    float2 u0[3], du[9];
#pragma unroll
    for (int i = 0; i < 3; i++) u0[i] = p.uhl[nd[0] + i * nn];
#pragma unroll
    for (int a = 1; a < 4; a++)
#pragma unroll
        for (int i = 0; i < 3; i++) du[(a - 1) * 3 + i] = dw_add_sloppy(p.uhl[nd[a] + i * nn], dw_neg(u0[i]));
    float2 F[9], P[9];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            F[i * 3 + j] = dw_dot3(du[i], G[j], du[3 + i], G[3 + j], du[6 + i], G[6 + j], i == j ? 1.0f : 0.0f);
    const MatParams &m = mat_of(p, e);
    float hh = 0.0f;   // ||F - I||_F^2, for the CFL gate
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const float h = k % 4 == 0 ? F[k].x - 1.0f : F[k].x;
        hh = fmaf(h, h, hh);
    }
    stress_dw(m, F, make_float2(__ldg(p.wJ32 + e), __ldg(p.wJ32lo + e)), P);
    if (VISC && !FORCE_ONLY) {
        // bulk viscosity in FP64 from the double-word F (exact as doubles), added as double-words
        double Fd[9], Pv[9];
#pragma unroll
        for (int k = 0; k < 9; k++) Fd[k] = (double)F[k].x + (double)F[k].y;
        visc_bulk_fp64(p, e, Fd, (double)__ldg(p.wJ32 + e) + (double)__ldg(p.wJ32lo + e), m.rho, idt, Pv);
#pragma unroll
        for (int k = 0; k < 9; k++) P[k] = dw_add(P[k], dw_from(Pv[k]));
    }
    float2 f[12];
#pragma unroll
    for (int a = 1; a < 4; a++)
#pragma unroll
        for (int i = 0; i < 3; i++)
            f[a * 3 + i] = dw_dot3(P[i * 3], G[(a - 1) * 3], P[i * 3 + 1], G[(a - 1) * 3 + 1], P[i * 3 + 2],
                                   G[(a - 1) * 3 + 2], 0.0f);
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = dw_neg(dw_add_sloppy(dw_add_sloppy(f[3 + i], f[6 + i]), f[9 + i]));
    if (ACT && elem_dead(p, e, t))
#pragma unroll
        for (int k = 0; k < 12; k++) f[k] = make_float2(0.f, 0.f);
    const int4 sl = __ldg(p.slot + e);
    const int ks[4] = {sl.x, sl.y, sl.z, sl.w};
    float2 *fe = reinterpret_cast<float2 *>(p.fe);
#pragma unroll
    for (int a = 0; a < 4; a++) {
        float2 *fk = fe + (long long)ks[a] * 3;
        fk[0] = f[a * 3];
        fk[1] = f[a * 3 + 1];
        fk[2] = f[a * 3 + 2];
    }
    if (FORCE_ONLY) return 0.0f;
    if (e == 0 && !isfinite(p.uhl[1].x)) atomicOr(p.flags + (parity ^ 1), 1);
    if (gate_frobenius(__ldg(p.Lref32 + e), hh, m.inv_c_f) > gmin) return INFINITY;
    float du32[9], g32[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
        du32[k] = du[k].x;
        g32[k] = G[k].x;
    }
    return cfl_screen(p, e, g32, du32, m);
}

// corner forces only (internal-force hook)
static __global__ void __launch_bounds__(kElemBlock) elem_force_kernel_dw(Problem p, int parity)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < p.ne) elem_body_dw<true>(p, e, parity, p.conn[e]);
}

// Node body of the double-word mode: the mixed mode's four-lane gather and
// update, with double-word corner forces summed as (s, c): s the FP32 sum of
// the high words by TwoSum, c the rounding errors plus the low words.
__device__ __forceinline__ void dw_sum_merge(float &s, float &c, float s2, float c2)
{
    const float t = __fadd_rn(s, s2);
    c = c + c2 + dw_err(s, s2, t);
    s = t;
}

template <bool BATCH>
__device__ __forceinline__ void node_quad_dw(const Problem &p, long long i, bool valid, const NodeStep &ns, int2 slots)
{
    const int q = threadIdx.x & 3;
    const bool odd = q & 1;
    const bool own = valid && q < 3;
    const long long dof = i + (long long)q * p.nn;
    float2 uq = make_float2(0.f, 0.f), vq = uq, aq = uq, minv = uq;
    int rec = -1;
    if (own) {
        uq = p.uhl[dof];
        vq = p.vhl[dof];
        aq = p.ahl[dof];
        minv = p.minv2[i];
        rec = p.node_bc[i];
    }
    const int k0 = slots.x, k1 = slots.y;
    const float2 *fe = reinterpret_cast<const float2 *>(p.fe);
    float h0 = 0.f, h1 = 0.f, h2 = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f;
    int k = k0 + q;
    constexpr int NB = BATCH ? kBatch : 0;
    float2 g[3 * NB + 1];
    if (BATCH) {
#pragma unroll
        for (int j = 0; j < NB; j++)
            if (k + 4 * j < k1) {
                const float2 *f = fe + (long long)(k + 4 * j) * 3;
                g[3 * j] = f[0];
                g[3 * j + 1] = f[1];
                g[3 * j + 2] = f[2];
            }
#pragma unroll
        for (int j = 0; j < NB; j++) {
            if (k >= k1) break;
            const float2 f0 = g[3 * j], f1 = g[3 * j + 1], f2 = g[3 * j + 2];
            if (j == 0) {
                h0 = f0.x, c0 = f0.y;
                h1 = f1.x, c1 = f1.y;
                h2 = f2.x, c2 = f2.y;
            } else {
                dw_sum_merge(h0, c0, f0.x, f0.y);
                dw_sum_merge(h1, c1, f1.x, f1.y);
                dw_sum_merge(h2, c2, f2.x, f2.y);
            }
            k += 4;
        }
    } else if (k < k1) {
        const float2 *f = fe + (long long)k * 3;
        const float2 f0 = f[0], f1 = f[1], f2 = f[2];
        h0 = f0.x, c0 = f0.y;
        h1 = f1.x, c1 = f1.y;
        h2 = f2.x, c2 = f2.y;
        k += 4;
    }
    for (; k < k1; k += 4) {
        const float2 *f = fe + (long long)k * 3;
        const float2 f0 = f[0], f1 = f[1], f2 = f[2];
        dw_sum_merge(h0, c0, f0.x, f0.y);
        dw_sum_merge(h1, c1, f1.x, f1.y);
        dw_sum_merge(h2, c2, f2.x, f2.y);
    }
    float ah = odd ? h0 : h1, ac = odd ? c0 : c1;
    float xh = __shfl_xor_sync(0xffffffffu, ah, 1), xc = __shfl_xor_sync(0xffffffffu, ac, 1);
    float yh = __shfl_xor_sync(0xffffffffu, h2, 1), yc = __shfl_xor_sync(0xffffffffu, c2, 1);
    if (odd) {
        dw_sum_merge(h1, c1, xh, xc);
    } else {
        dw_sum_merge(h0, c0, xh, xc);
        dw_sum_merge(h2, c2, yh, yc);
    }
    float sh = odd ? h1 : (q == 0 ? h2 : h0), sc = odd ? c1 : (q == 0 ? c2 : c0);
    float zh = __shfl_xor_sync(0xffffffffu, sh, 2), zc = __shfl_xor_sync(0xffffffffu, sc, 2);
    float mh = pick3(q, h0, h1, h2), mc = pick3(q, c0, c1, c2);
    dw_sum_merge(mh, mc, zh, zc);
    if (!own) return;
    const float2 s = dw_two_sum(mh, mc);
    const int2 br = rec >= 0 ? p.bc_rec[rec * 3 + q] : make_int2(0, 0);
    const bool act = br.y == 0;
    bool changed = false;
    if (ns.ran && act) {
        const float2 f = ns.loads ? dw_add(dw_from(node_fext(p, i, q, ns)), dw_neg(s)) : dw_neg(s);
        const float2 an = dw_mul(f, minv);
        vq = dw_add(vq, dw_mul(ns.hdt2, dw_add(aq, an)));
        aq = an;
        changed = true;
    }
    if (ns.run) {
        if (act) {
            uq = dw_add(uq, dw_mul(ns.dtn2, dw_add(vq, dw_mul(ns.hdtn2, aq))));
        } else {
            for (int k = br.x; k < br.x + br.y; k++) {
                const float2 Ud = dw_from(bc_increment(p.bcs[k], ns.dtn, ns.step));
                uq = dw_add(uq, Ud);
                vq = Ud;
                aq = make_float2(0.f, 0.f);
            }
        }
        changed = true;
    }
    if (changed) {
        p.uhl[dof] = uq;
        p.vhl[dof] = vq;
        p.ahl[dof] = aq;
    }
}

// Block-wide min of a float, returned to every thread of the block.
__device__ __forceinline__ float block_min_bcast(float v);

// Reference-order element kernel with the FP32 CFL screen: forces in the
// reference's order for every element, the exact reference-order CFL value only
// for the elements within 2^-8 of the solve's running FP32 minimum (and slivers),
// a set that always holds the exact minimum, so dt is the reference's.  A block
// without any returns at once.
template <bool VISC>
__global__ void __launch_bounds__(kElemBlock) elem_kernel_exact_screened(Problem p, int parity)
{
    if (!p.ctrl[parity].ran) return;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const float gmin = __uint_as_float((unsigned)__ldcg(p.dtmin + 2 + (parity ^ 1))) * (1.0f + 1.0f / 256.0f);
    const float d = e < p.ne ? (float)elem_body_exact<false, true, VISC>(p, e, parity, gmin) : INFINITY;
    if (!__syncthreads_or(!(d > gmin))) return;
    const float bmin = block_min_bcast(d >= 0.0f ? d : INFINITY);
    if (threadIdx.x == 0 && bmin < gmin)
        atomicMin(p.dtmin + 2 + (parity ^ 1), (unsigned long long)__float_as_uint(bmin));
    double v = INFINITY;
    if (e < p.ne && !(d > fminf(gmin, bmin * (1.0f + 1.0f / 256.0f)))) v = cfl_exact_ref(p, e);
    block_min_to(v, p.dtmin + (parity ^ 1));
}

__device__ __forceinline__ float block_min_bcast(float v)
{
    __shared__ float wm[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) wm[w] = v;
    __syncthreads();
    int nw = (blockDim.x + 31) >> 5;
    float r = INFINITY;
    for (int k = 0; k < nw; k++) r = fminf(r, wm[k]);
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------
// Pooled kernels: many independent solves stepped by one persistent grid.
// Each tile is a contiguous element (or node) range of one solve; CTAs stride
// over the tile list, so the grid size is fixed (a multiple of the SM count)
// and the same graph serves any admitted set.  Per-solve control, CFL slot
// and NaN flag are those of the solve's Problem.
// ---------------------------------------------------------------------------
// Where the tiled kernels get their work.  PoolTiles: the pool's tile list and
// descriptors in device memory.  SolveTiles: one solve, whose Problem is a
// kernel argument (the constant bank: no load stands before the first use of
// its pointers) and whose tiles are equal ranges of `size` elements, computed
// instead of loaded.
struct PoolTiles {
    const Problem *descs;
    const Tile *tiles;
    __device__ __forceinline__ Tile tile(int t) const { return tiles[t]; }
    __device__ __forceinline__ const Problem &problem(const Tile &tl) const { return descs[tl.solve]; }
};

struct SolveTiles {
    const Problem &p;
    int size;
    __device__ __forceinline__ Tile tile(int t) const
    {
        const long long b = (long long)t * size, e = b + size;
        return {0, (int)b, (int)(e < p.ne ? e : p.ne)};
    }
    __device__ __forceinline__ const Problem &problem(const Tile &) const { return p; }
};

// Tile assignment over n tiles; sched = {tile count, claim counter, blocks done}.
// When the grid has a block for every tile, block b takes tile b and nothing
// is claimed: the claims of a whole grid serialise on one address, 1.7 us of a
// launch of 608 blocks (0.71 us for the launch alone).  Otherwise dynamic:
// thread 0 claims the block's next tile while the block works on the current
// one; every block makes exactly one claim past the end, and the last block to
// run out puts both counters back to zero for the next launch.  Which block
// runs a tile changes no result.
struct TileQueue {
    int *sched;
    int n;
    bool fixed;
    __device__ __forceinline__ TileQueue(int *sched_, int n_) : sched(sched_), n(n_), fixed(n_ <= (int)gridDim.x) {}
    // the block's first tile, in every thread (s_tile: shared scratch)
    __device__ __forceinline__ int first(int *s_tile)
    {
        if (fixed) return blockIdx.x;
        if (threadIdx.x == 0) *s_tile = atomicAdd(sched + 1, 1);
        __syncthreads();
        return *s_tile;
    }
    // thread 0: claims the next tile (the others: ignored)
    __device__ __forceinline__ int claim() { return fixed || threadIdx.x != 0 ? n : atomicAdd(sched + 1, 1); }
    // the claimed tile, in every thread; a barrier either way
    __device__ __forceinline__ int next(int claimed, int *s_tile)
    {
        __syncthreads();
        if (fixed) return n;
        if (threadIdx.x == 0) *s_tile = claimed;
        __syncthreads();
        return *s_tile;
    }
    __device__ __forceinline__ void finish()
    {
        if (!fixed && threadIdx.x == 0 && atomicAdd(sched + 2, 1) == (int)gridDim.x - 1) {
            atomicExch(sched + 1, 0);
            atomicExch(sched + 2, 0);
        }
    }
};

// Programmatic dependent launch, used for single solves of small grids
// (SolveSched::pdl): the next kernel of the step chain may start
// once every block of this one has called pdl_release, and does its launch and
// the loads of data no step writes (pull_*) while this one runs; pdl_wait
// returns when the kernel before has completed and its writes are visible.  A
// kernel releases only after its own wait, so no more than two are under way and
// what a kernel reads before its wait was complete two kernels earlier.  Without
// the launch attribute both are no-ops.  A kernel is under way while the one
// before still writes the state and the corner forces, so it reads those with
// ordinary loads: __ldg (and pull) are for arrays that no step writes, as the
// read-only path promises nothing about data that changes in a kernel's life.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Loads the line at x into L1 (and drops the value).
template <typename T>
__device__ __forceinline__ void pull(const T *x)
{
    unsigned v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(x));
}

__device__ __forceinline__ void pull_node(const Problem &p, long long i)
{
    if (i >= p.nn) return;
    pull(p.node_ptr + i);
    pull(p.node_bc + i);
    if (p.minv2) pull(p.minv2 + i);
    else pull(p.minv + i);
}

template <int MODE>
__device__ __forceinline__ void pull_element(const Problem &p, long long e)
{
    if (e >= p.ne) return;
    pull(p.conn + e);
    pull(p.slot + e);
    pull(p.Lref32 + e);
    if (MODE == MODE_FP64 && p.fxE) {
        pull(p.fxw + e);
        pull(p.fxD + e);
#pragma unroll
        for (int k = 0; k < 9; k++) pull(p.fxE + k * p.ne + e);
        if (p.fxS)
#pragma unroll
            for (int k = 0; k < 6; k++) pull(p.fxS + k * p.ne + e);
    } else if (MODE == MODE_FP64) {
        pull(p.wJ + e);
#pragma unroll
        for (int k = 0; k < 9; k++) pull(p.G + k * p.ne + e);
    } else {
        pull(p.wJ32 + e);
#pragma unroll
        for (int k = 0; k < 9; k++) pull(p.G32 + k * p.ne + e);
        if (MODE == MODE_DW) {
            pull(p.wJ32lo + e);
#pragma unroll
            for (int k = 0; k < 9; k++) pull(p.G32lo + k * p.ne + e);
        }
    }
}

// The node's corner-force slots [x, y); none without forces to add
__device__ __forceinline__ int2 node_slots(const Problem &p, long long i, bool any)
{
    return any ? make_int2(p.node_ptr[i], p.node_ptr[i + 1]) : make_int2(0, 0);
}

template <int MODE, bool BATCH>
__device__ __forceinline__ void node_quad(const Problem &p, long long i, bool valid, const NodeStep &ns, int2 slots)
{
    if (MODE == MODE_MIXED) node_quad_mixed<BATCH>(p, i, valid, ns, slots);
    else if (MODE == MODE_DW) node_quad_dw<BATCH>(p, i, valid, ns, slots);
    else node_quad_fp64<BATCH>(p, i, valid, ns, slots);
}

// The step decision by one warp for its block: about 60 instructions on the FP64
// pipe, which kept it 69 % busy when every warp took them (mixed node kernel,
// 1.6M tets; 116,000 tets mixed 16.3 -> 14.2 us a step).
template <int MODE>
__device__ __forceinline__ NodeStep block_node_step(const Problem &p, int parity, bool publish)
{
    __shared__ NodeStep s_ns;   // read by all before the caller's next barrier
    if (threadIdx.x < 32) {
        NodeStep ns;
        node_step<MODE>(p, parity, publish && threadIdx.x == 0, ns);
        if (threadIdx.x == 0) s_ns = ns;
    }
    __syncthreads();
    return s_ns;
}

// The pool's node kernel over tiles (node ranges of one solve), four lanes per node.
template <int MODE>
__device__ __forceinline__ void node_tile_loop(const PoolTiles &src, TileQueue q, int parity)
{
    __shared__ int s_tile;
    int t = q.first(&s_tile), cur = -1;
    NodeStep ns;
    while (t < q.n) {
        const int claimed = q.claim();
        const Tile tl = src.tile(t);
        const Problem &p = src.problem(tl);
        if (tl.solve != cur) {   // a solve's first tile (begin 0) is the first of its tiles a block meets
            ns = block_node_step<MODE>(p, parity, tl.begin == 0);
            cur = tl.solve;
        }
        if (ns.ran || ns.run) {
            const int per = blockDim.x >> 2;   // every lane runs the same number of passes
            for (long long b = tl.begin; b < tl.end; b += per) {
                long long i = b + (threadIdx.x >> 2);
                node_quad<MODE, false>(p, i, i < tl.end, ns, node_slots(p, i, i < tl.end && ns.ran));
            }
        }
        t = q.next(claimed, &s_tile);
    }
    q.finish();
}

// CTAs of kStepThreads an SM holds at the least: the register caps of the node
// kernels (6M tets, mixed: 104 us with 48 registers, 109 with 40, 114 with 64;
// FP64: 160 with 48, 163 with 64, 171 with 80)
constexpr int node_ctas(int mode, bool batch) { return batch ? (mode == MODE_MIXED ? 3 : 2) : 5; }

// 64 registers, four CTAs an SM: a step of 16 mixed solves of 162,000 tets 182 us,
// 204 with 48 registers (five CTAs, best for one solve, leave the tile queue a
// longer last wave), 194 with 80; 256 solves 1.97e10, 1.90e10 and 1.93e10
// element-steps/s; FP64 and double-word as with five, 3 to 4 % slower with three.
template <int MODE>
__global__ void __launch_bounds__(kStepThreads, 4) pool_node_kernel(const Problem *__restrict__ descs, const Tile *__restrict__ tiles,
                                 int *__restrict__ sched, int parity)
{
    node_tile_loop<MODE>(PoolTiles{descs, tiles}, TileQueue(sched, sched[0]), parity);
}

// A node's next slots into L2, a line or two a lane
template <int MODE>
__device__ __forceinline__ void prefetch_slots(const Problem &p, int2 slots)
{
    constexpr int bytes = MODE == MODE_MIXED ? 16 : 24;
    const char *f = (MODE == MODE_MIXED ? (const char *)p.fe32 : (const char *)p.fe) + (long long)slots.x * bytes;
    const int n = (slots.y - slots.x) * bytes, o = (threadIdx.x & 3) * 128;
    if (o < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(f + o));
    if (MODE != MODE_MIXED && o + 512 < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(f + o + 512));
}

// One solve: passes of blockDim / 4 nodes, which go to the blocks in turn (a
// node's work hardly differs from the next one's, so claims would only add
// their barriers), with the next pass's slot range loaded a pass ahead and its
// slots prefetched.  Bound by the latency of each pass's loads and, in FP64, the
// ALU pipe.  Node kernel of 6M tets: FP64 174 -> 163 us without claims, 145 with
// the next slots ahead; mixed 121 -> 104 and 104; 1.6M tets double-word 51 -> 46.
// Shared-memory stages of a tile's slots instead: 250, 131 and 54 us, for the
// warps they cost.
// SMALL: blocks of 128 threads, one warp a scheduler, where every warp derives
// the step decision and no barrier is worth it (72 tets 10.4 us a step, 11.2
// with it).
template <int MODE, bool BATCH, bool SMALL = false>
__global__ void __launch_bounds__(SMALL ? 128 : kStepThreads, node_ctas(MODE, BATCH))
    solve_node_kernel(const __grid_constant__ Problem p, int parity)
{
    const long long per = blockDim.x >> 2, stride = per * gridDim.x;
    if (p.nn <= stride) pull_node(p, blockIdx.x * per + (threadIdx.x >> 2));
    pdl_wait();
    pdl_release();
    NodeStep ns;
    if (SMALL) node_step<MODE>(p, parity, blockIdx.x == 0 && threadIdx.x == 0, ns);
    else ns = block_node_step<MODE>(p, parity, blockIdx.x == 0);
    if (!ns.ran && !ns.run) return;
    long long i = blockIdx.x * per + (threadIdx.x >> 2);
    int2 k = node_slots(p, i, i < p.nn && ns.ran);
    for (long long b = blockIdx.x * per; b < p.nn; b += stride, i += stride) {
        const int2 now = k;
        k = node_slots(p, i + stride, i + stride < p.nn && ns.ran);
        node_quad<MODE, BATCH>(p, i, i < p.nn, ns, now);
        if (!BATCH) prefetch_slots<MODE>(p, k);
    }
}

// The fixed-point FP64 kernels' streamed element data of the pass
// of blockDim elements that begins at b, into L2: one or two lines a thread
// instead of a DRAM latency before the next pass's arithmetic (6M tets: element
// kernel 0.497 -> 0.476 ms; 0.473 -> 0.448 with the connectivity one pass ahead).
__device__ __forceinline__ void prefetch_line(const char *r, bool in)
{
    if (in) asm volatile("prefetch.global.L2 [%0];" ::"l"(r));
}

template <int FIXED>
__device__ __forceinline__ void prefetch_pass(const Problem &p, long long b, long long end)
{
    // 16 rows (without fxS 10) of 8-byte entries, blockDim / 16 lines each, then two of 16 and one of
    // 4 bytes; no line that begins past the tile's last element
    const int sh = blockDim.x >= 256 ? 4 : 3, row = threadIdx.x >> sh, t = threadIdx.x;
    const long long left = end - b;   // elements from b on
    const int l = t - (row << sh);
    const char *r = row < 9 ? (const char *)(p.fxE + row * p.ne + b)
                            : (row < 15 ? (const char *)(p.fxS + (row - 9) * p.ne + b) : (const char *)(p.fxw + b));
    prefetch_line(r + l * 128, l * 16 < left && (FIXED == FIXED_CNH || row < 9 || row == 15));
    const int l2 = row < 2 ? t : (row < 4 ? t - (2 << sh) : t - (4 << sh)), per = row < 4 ? 8 : 32;
    r = row < 2 ? (const char *)(p.fxD + b) : (row < 4 ? (const char *)(p.slot + b) : (const char *)(p.Lref32 + b));
    prefetch_line(r + l2 * 128, t < (9 << sh) / 2 && l2 * per < left);
}

// The elements of one tile for the tiled element kernel: each thread's
// elements in turn; returns the thread's FP32 minimum of the CFL screen
// (infinite when the gate let none through).  gmin: (1 + 2^-8) times the
// solve's running minimum as the tile began.  The FP64 and double-word kernels
// list every element whose screen value is not above it (slivers, with -1,
// included) in sval and scand; the mixed one lists none and returns -1 once one
// of its elements was a sliver, so no other register stays live.  The mixed and
// double-word bodies take the element's connectivity loaded one element ahead,
// so their node gathers wait for one memory latency instead of two
// (connectivity, then the nodes).  ACT: element birth is on, and the step's time
// decides which elements are dead.
template <int MODE, bool ACT, bool VISC, int FIXED = FIXED_NONE>
__device__ __forceinline__ float tile_elements(const Problem &p, const Tile &tl, int parity, float gmin, float *sval,
                                               unsigned short *scand, int *ncand, int *nleft)
{
    float v32 = INFINITY;
    const double t = ACT ? p.ctrl[parity].t : 0.0;
    const double idt = VISC ? 1.0 / p.ctrl[parity].dt : 0.0;   // the step's dt (bulk viscosity)
    const float idtf = (float)idt;
    long long e = tl.begin + threadIdx.x;
    int4 cn_next = make_int4(0, 0, 0, 0);
    constexpr bool ahead = MODE == MODE_MIXED || MODE == MODE_DW || FIXED;
    if (ahead) {
        if (e < tl.end) cn_next = p.conn[e];
    }
    for (; e < tl.end; e += blockDim.x) {
        const int4 cn = cn_next;
        if (ahead && e + blockDim.x < tl.end) cn_next = p.conn[e + blockDim.x];
        if constexpr (FIXED != FIXED_NONE) prefetch_pass<FIXED>(p, e - threadIdx.x + blockDim.x, tl.end);
        float d = MODE == MODE_MIXED ? elem_body_mixed<false, ACT, VISC>(p, e, parity, cn, t, idtf, gmin)
                                     : (MODE == MODE_DW ? elem_body_dw<false, ACT, VISC>(p, e, parity, cn, t, idt, gmin)
                                                        : elem_body_fp64<false, ACT, VISC, FIXED>(p, e, parity, t, idt, gmin, cn));
        if (MODE == MODE_MIXED) {
            v32 = d < 0.0f ? -1.0f : fminf(v32, d);   // -1 sticks: fminf(-1, d) = -1 for d >= 0
        } else if (MODE == MODE_FP64 && !VISC && d == kLeftOut) {
            scand[kMaxTileElems - 1 - atomicAdd(nleft, 1)] = (unsigned short)(e - tl.begin);
        } else if (!(d > gmin)) {
            const int k = atomicAdd(ncand, 1);
            sval[k] = d;
            scand[k] = (unsigned short)(e - tl.begin);
            if (d >= 0.0f) v32 = fminf(v32, d);
        }
    }
    return v32;
}

// The nl elements of a tile that fixed point left out, in FP64 by consecutive
// threads: one of them in a warp costs it the FP64 pipe as long as 32 do.  1M
// tets in hexes of 1:1:0.2, compressible neo-Hookean, a third of them left out
// and every warp with some: 346 us a step, 622 with the FP64 form inside their
// warps (407 with all elements in FP64); 1:1:3, jittered, 217, 349 and 276.
// Lists CFL candidates and returns the thread's minimum as tile_elements does.
// Left-out elements lie at the end of scand, last one first; an element is in
// one list at a time, and a pass reads its entries, the lowest that remain,
// before it lists candidates, so these never reach an entry still to be read.
template <bool ACT>
__device__ __forceinline__ float tile_left_out(const Problem &p, const Tile &tl, int parity, float gmin, float *sval,
                                               unsigned short *scand, int *ncand, int nl)
{
    float v32 = INFINITY;
    const double t = ACT ? p.ctrl[parity].t : 0.0;
    for (int at = nl - 1 - (int)threadIdx.x, base = 0; base < nl; base += blockDim.x, at -= blockDim.x) {
        const int i = at >= 0 ? scand[kMaxTileElems - 1 - at] : 0;
        __syncthreads();
        if (at < 0) continue;
        const float d = elem_left_out<false, ACT>(p, tl.begin + i, parity, t, gmin);
        if (!(d > gmin)) {
            const int k = atomicAdd(ncand, 1);
            sval[k] = d;
            scand[k] = (unsigned short)i;
            if (d >= 0.0f) v32 = fminf(v32, d);
        }
    }
    return v32;
}

// The solve's running FP32 minimum of the CFL screen for the step in progress:
// the undeformed minimum at first (publish_step), lowered by the tiles.
__device__ __forceinline__ float running_min(const Problem &p, int parity)
{
    return __uint_as_float((unsigned)__ldcg(p.dtmin + 2 + (parity ^ 1)));
}

constexpr int kMixedPending = 2 * kStepThreads;  // deferred FP64 rechecks a mixed CTA can hold

// The pending entries of a mixed CTA (all posted before the caller's last
// barrier): one warp per entry, four lanes an element of the posting thread's of
// that tile (at most eight), skipping entries above 2^-8 of the solve's running
// screen minimum.
template <typename SRC>
static __device__ __noinline__ void mixed_flush(const SRC src, const int2 *pend, const float *pendv, int np, int parity)
{
    const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    for (int j = threadIdx.x >> 5; j < np; j += nwarp) {
        const int2 pe = pend[j];
        const Tile tl = src.tile(pe.x);
        const Problem &p = src.problem(tl);
        const float mine = pendv[j];
        if (!(mine < 0.0f) && mine > running_min(p, parity) * (1.0f + 1.0f / 256.0f)) continue;
        double v = INFINITY;
        for (long long e0 = tl.begin + pe.y; e0 < tl.end; e0 += 8LL * blockDim.x) {   // the same in every lane
            const long long e = e0 + (long long)(lane >> 2) * blockDim.x;
            v = fmin(v, cfl_quad(p, e < tl.end ? e : e0, true));
        }
#pragma unroll
        for (int o = 16; o > 2; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0 && v >= 0.0 && v < INFINITY)
            atomicMin(p.dtmin + (parity ^ 1), (unsigned long long)__double_as_longlong(v));
    }
}

// The mixed kernel's tile loop.  A thread whose own screen minimum lies within
// 2^-8 of the solve's running minimum as its tile began, or that met a sliver,
// posts (tile, thread, own minimum) to a per-CTA list; a warp that went clearly
// below lowers the running minimum by an integer atomicMin on its bit pattern
// (nothing waited for).  Once the CTA has run out of tiles, every entry whose
// minimum is still within 2^-8 of the running minimum -- by then nearly the
// step's FP32 minimum m -- has that thread's elements of that tile recomputed
// in FP64 by one warp of the CTA.  The running minimum g is never below m, and
// an element x near the exact minimum has d(x) <= m (1 + 2^-8) <= g (1 + 2^-8)
// whenever g is read, so its thread posted (unless it met a sliver, and then it
// posted anyway) and its entry, whose minimum is <= d(x), is rechecked.  A tile
// adds at most one entry per thread, so the list is flushed at a tile boundary
// once it holds more than kMixedPending - blockDim entries, and never
// overflows; the element loop itself calls no FP64 code.
template <bool ACT, bool VISC, typename SRC>
__device__ __forceinline__ void mixed_tile_loop(const SRC &src, TileQueue &q, int parity)
{
    __shared__ int s_tile, s_npend;
    __shared__ int2 s_pend[kMixedPending];      // (tile, thread)
    __shared__ float s_pendv[kMixedPending];    // the thread's minimum, -1 for a sliver
    if (threadIdx.x == 0) s_npend = 0;
    __syncthreads();
    int t = q.first(&s_tile);
    while (t < q.n) {
        const int claimed = q.claim();
        const Tile tl = src.tile(t);
        const Problem &p = src.problem(tl);
        if (p.ctrl[parity].ran) {
            const float g = running_min(p, parity), gmin = g * (1.0f + 1.0f / 256.0f);
            const float mine = tile_elements<MODE_MIXED, ACT, VISC>(p, tl, parity, gmin, nullptr, nullptr, nullptr, nullptr);
            if (!(mine > gmin)) {
                const int k = atomicAdd(&s_npend, 1);   // < kMixedPending: flushed below in time
                s_pend[k] = make_int2(t, (int)threadIdx.x);
                s_pendv[k] = mine;
            }
            float w = mine < 0.0f ? INFINITY : mine;
            if (__any_sync(0xffffffffu, w < g * (1.0f - 1.0f / 1024.0f))) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) w = fminf(w, __shfl_xor_sync(0xffffffffu, w, o));
                if ((threadIdx.x & 31) == 0)
                    atomicMin(p.dtmin + 2 + (parity ^ 1), (unsigned long long)__float_as_uint(w));
            }
        }
        t = q.next(claimed, &s_tile);
        if (s_npend > kMixedPending - (int)blockDim.x) {   // the same value in every thread
            mixed_flush(src, s_pend, s_pendv, s_npend, parity);
            __syncthreads();
            if (threadIdx.x == 0) s_npend = 0;
            __syncthreads();
        }
    }
    mixed_flush(src, s_pend, s_pendv, s_npend, parity);   // posted before the loop's last barrier
}

// Element kernel over tiles.  The solve's running FP32 minimum of the CFL screen
// (a per-step slot that starts from the undeformed minimum, an upper bound of
// every step's, and that tiles lower by an integer atomicMin on its bit
// pattern) decides which elements recompute the exact FP64 value, whose minimum
// goes to the solve's CFL slot: those within 2^-8 of it, and slivers.  The
// screen's error stays far below 2^-9 outside slivers, so that set always holds
// the step's exact minimum.  FP64 and double-word list a tile's candidates in
// shared memory as they come and recompute those that remain at its end by
// consecutive threads, so a few candidates take one warp; a tile without any
// (nearly every tile) closes with one barrier.  The mixed kernel defers its few
// rechecks to the end of the CTA's tiles (mixed_tile_loop).  ACT: the
// instantiation with element birth (single solves whose block has it on), VISC
// the one with artificial bulk viscosity; the plain one carries no trace of
// either.
template <int MODE, bool ACT, bool VISC, int FIXED = FIXED_NONE, typename SRC>
__device__ __forceinline__ void elem_tile_loop(const SRC &src, TileQueue q, int parity)
{
    __shared__ float sval[MODE == MODE_MIXED ? 1 : kMaxTileElems];
    __shared__ unsigned short scand[MODE == MODE_MIXED ? 1 : kMaxTileElems];
    __shared__ int s_tile, s_ncand, s_nleft;
    __shared__ float s_thr;
    if constexpr (MODE == MODE_MIXED) {
        mixed_tile_loop<ACT, VISC>(src, q, parity);
        q.finish();
        return;
    }
    if (threadIdx.x == 0) s_ncand = s_nleft = 0;
    __syncthreads();
    int t = q.first(&s_tile);
    while (t < q.n) {
        const int claimed = q.claim();
        const Tile tl = src.tile(t);
        const Problem &p = src.problem(tl);
        if (p.ctrl[parity].ran) {
            const float gmin = running_min(p, parity) * (1.0f + 1.0f / 256.0f);
            float v32 = tile_elements<MODE, ACT, VISC, FIXED>(p, tl, parity, gmin, sval, scand, &s_ncand, &s_nleft);
            __syncthreads();
            if constexpr (MODE == MODE_FP64 && !VISC) {
                const int nl = s_nleft;
                if (nl > 0) {   // uniform across the block
                    v32 = fminf(v32, tile_left_out<ACT>(p, tl, parity, gmin, sval, scand, &s_ncand, nl));
                    __syncthreads();
                    if (threadIdx.x == 0) s_nleft = 0;
                }
            }
            const int nc = s_ncand;
            if (nc > 0) {   // uniform across the block
                const float bmin = block_min_bcast(v32);
                if (threadIdx.x == 0) {
                    s_ncand = 0;
                    // g: the smallest screen value any tile has reported so far in this
                    // step, this one included, or the undeformed minimum
                    unsigned old = (unsigned)__ldcg(p.dtmin + 2 + (parity ^ 1));
                    if (bmin < __uint_as_float(old))
                        old = (unsigned)atomicMin(p.dtmin + 2 + (parity ^ 1), (unsigned long long)__float_as_uint(bmin));
                    s_thr = fminf(__uint_as_float(old), bmin) * (1.0f + 1.0f / 256.0f);
                }
                __syncthreads();
                const float thr = s_thr;
                double v = INFINITY;
                const int quads = blockDim.x >> 2;
                // One lane a candidate above two passes of four lanes each: those double the
                // instructions on the FP64 pipe and only halve their chain, and a mesh of equal
                // elements lists nearly all of its elements (1M tets of an unjittered cube at
                // rest: 323 us a step, 521 with four lanes throughout).
                if (nc > 2 * quads) {
                    for (int c = threadIdx.x; c < nc; c += blockDim.x)
                        if (!(sval[c] > thr)) v = fmin(v, cfl_lane(p, tl.begin + scand[c], MODE == MODE_DW));
                } else {
                    for (int c0 = 0; c0 < nc; c0 += quads) {
                        const int c = c0 + (threadIdx.x >> 2);
                        const bool mine = c < nc && !(sval[c] > thr);
                        if (!__any_sync(0xffffffffu, mine)) continue;
                        const double d = cfl_quad(p, tl.begin + (mine ? scand[c] : 0), MODE == MODE_DW);
                        if (mine) v = fmin(v, d);
                    }
                }
                block_min_to(v, p.dtmin + (parity ^ 1));
            }
        }
        t = q.next(claimed, &s_tile);
    }
    q.finish();
}

// CTAs of kStepThreads an SM holds: the register caps of the element kernels
constexpr int elem_ctas(int mode) { return mode == MODE_MIXED ? 4 : (mode == MODE_DW ? 3 : 2); }

// (no element birth, no viscosity in a pool)
template <int MODE>
__global__ void __launch_bounds__(kStepThreads, elem_ctas(MODE))
    pool_elem_kernel(const Problem *__restrict__ descs, const Tile *__restrict__ tiles, int *__restrict__ sched, int parity)
{
    elem_tile_loop<MODE, false, false>(PoolTiles{descs, tiles}, TileQueue(sched, sched[0]), parity);
}

// One solve: tiles of `size` elements
template <int MODE, bool ACT = false, bool VISC = false>
__global__ void __launch_bounds__(kStepThreads, elem_ctas(MODE))
    solve_elem_kernel(const __grid_constant__ Problem p, int size, int ntiles, int *__restrict__ sched, int parity)
{
    if (ntiles <= (int)gridDim.x) pull_element<MODE>(p, (long long)blockIdx.x * size + threadIdx.x);
    pdl_wait();
    pdl_release();
    elem_tile_loop<MODE, ACT, VISC>(SolveTiles{p, size}, TileQueue(sched, ntiles), parity);
}

// One solve in FP64 whose every material is compressible neo-Hookean.  128
// registers and two CTAs an SM: three CTAs (80 registers, spills) 0.482 ms
// against 0.497 without the prefetches and 0.509 against 0.448 with them; five
// CTAs of 128 threads (96 registers) 0.469 against 0.452.
static __global__ void __launch_bounds__(kStepThreads, elem_ctas(MODE_FP64))
    solve_elem_cnh_kernel(const __grid_constant__ Problem p, int size, int ntiles, int *__restrict__ sched, int parity)
{
    if (ntiles <= (int)gridDim.x) pull_element<MODE_FP64>(p, (long long)blockIdx.x * size + threadIdx.x);
    pdl_wait();
    pdl_release();
    elem_tile_loop<MODE_FP64, false, false, FIXED_CNH>(SolveTiles{p, size}, TileQueue(sched, ntiles), parity);
}

// One solve in FP64 whose every material is St-Venant-Kirchhoff or linear elastic.
static __global__ void __launch_bounds__(kStepThreads, elem_ctas(MODE_FP64))
    solve_elem_svk_kernel(const __grid_constant__ Problem p, int size, int ntiles, int *__restrict__ sched, int parity)
{
    if (ntiles <= (int)gridDim.x) pull_element<MODE_FP64>(p, (long long)blockIdx.x * size + threadIdx.x);
    pdl_wait();
    pdl_release();
    elem_tile_loop<MODE_FP64, false, false, FIXED_SVK>(SolveTiles{p, size}, TileQueue(sched, ntiles), parity);
}

// ---------------------------------------------------------------------------
// Set-up kernels (reference operation order), built in the exact unit only
// ---------------------------------------------------------------------------
#ifdef MSX_SETUP_KERNELS
// Reference Jacobian of a tet from xyz[i*4 + k] (coordinate i of corner k):
// Jac_ij = 0 + sum_k x_ik natDev_kj in corner order, natDev's entries -1, 0
// and 1 (classLinearTetrahedra.cpp:171-268).  For finite coordinates that sum
// is (0 - x_i0) + x_i(j+1) bit for bit: 0 - x_i0 is never -0, and the products
// with 0 add signed zeros to a partial sum that is never -0, which leaves it
// unchanged.  A non-finite coordinate (x * 0 is NaN) takes the full sum.
__device__ __forceinline__ void ref_jacobian(const double *xyz, double *Jac)
{
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 12; k++) finite &= isfinite(xyz[k]);
    if (finite) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const double y0 = 0.0 - xyz[i * 4];
#pragma unroll
            for (int j = 0; j < 3; j++) Jac[i * 3 + j] = y0 + xyz[i * 4 + j + 1];
        }
    } else {
        const double natDev[12] = {-1.0, -1.0, -1.0, 1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0};
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                double c = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) c += xyz[i * 4 + k] * natDev[k * 3 + j];
                Jac[i * 3 + j] = c;
            }
    }
}

// The plain FP64 mode's fixed-point data of element e
// (Problem::fxE, fxS, fxD, fxw) from its corner coordinates pts[k*3 + i].
__device__ __forceinline__ void write_fixed_arrays(const Problem &p, long long e, const double *pts)
{
    const long long ne = p.ne;
    double E[9];
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int i = 0; i < 3; i++) E[b * 3 + i] = pts[(b + 1) * 3 + i] - pts[i];
    const MatParams &m = mat_of(p, e);
    FixedElem q;
    uint32_t w[2] = {0, 0};
    if (m.law == 1 && fixed_setup(E, m.kq[0], m.ks, q)) {
        fixed_pack(q, w);
#pragma unroll
        for (int k = 0; k < 9; k++) const_cast<long long *>(p.fxE)[k * ne + e] = q.E[k];
#pragma unroll
        for (int k = 0; k < 6; k++) const_cast<int2 *>(p.fxS)[k * ne + e] = make_int2(q.S[k].h, q.S[k].l);
        const_cast<longlong2 *>(p.fxD)[e] = make_longlong2(q.d0, q.rd);
    } else if (m.law >= 2 && fixed_setup_svk(E, 0.5 * m.mu2, m.ks, q)) {
        fixed_pack(q, w);
#pragma unroll
        for (int k = 0; k < 9; k++) const_cast<long long *>(p.fxE)[k * ne + e] = q.E[k];
        const_cast<longlong2 *>(p.fxD)[e] = make_longlong2(limbs_pack(q.S[0]), 0);
    } else if (m.law >= 2) {   // left to the FP64 cofactor form: G as Problem::G holds it
        double xyz[12], Jac[9], iJ[9];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int i = 0; i < 3; i++) xyz[i * 4 + k] = pts[k * 3 + i];
        ref_jacobian(xyz, Jac);
        inv3_ref(Jac, iJ);
#pragma unroll
        for (int k = 0; k < 9; k++) const_cast<long long *>(p.fxE)[k * ne + e] = (long long)double_bits(0.0 + iJ[k]);
        w[0] = 0;
    }
    const_cast<uint2 *>(p.fxw)[e] = make_uint2(w[0], w[1]);
}

// classLinearTetrahedra.cpp:171-268 (Jacobian, inverse, dphi), classGPs.cpp:27
// (wJ = 0.166666666667 |J|), classLinearTetrahedra.cpp:129-140 (charLength).
// Two CTAs an SM: the fixed-point data's 128-bit products would take 133
// registers, one CTA, and msx_create of 6M tets 5.57 ms instead of 5.13.
__global__ void __launch_bounds__(256, 2) setup_elements_kernel(Problem p, const double *X, double *G, double *wJ, double *Lref,
                                      float *G32, float *wJ32, float *Lref32, long long e0, long long e1)
{
    const long long e = e0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;   // elements [e0, e1)
    if (e >= e1) return;
    const long long nn = p.nn, ne = p.ne;
    int4 cn = p.conn[e];
    // an out-of-range node id: the node-list build queued after this kernel
    // rejects the mesh
    if ((unsigned long long)(unsigned)cn.x >= (unsigned long long)nn || (unsigned long long)(unsigned)cn.y >= (unsigned long long)nn ||
        (unsigned long long)(unsigned)cn.z >= (unsigned long long)nn || (unsigned long long)(unsigned)cn.w >= (unsigned long long)nn)
        return;
    int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double xyz[12], pts[12];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int i = 0; i < 3; i++) {
            xyz[i * 4 + k] = X[i * nn + nd[k]];
            pts[k * 3 + i] = X[i * nn + nd[k]];
        }
    double Jac[9], iJ[9];
    ref_jacobian(xyz, Jac);
    double J = det3_ref(Jac);
    inv3_ref(Jac, iJ);
#pragma unroll
    for (int k = 0; k < 9; k++) {
        double g = 0.0 + iJ[k];
        if (G) G[k * ne + e] = g;
        if (G32) G32[k * ne + e] = (float)g;
        if (p.G32lo) const_cast<float *>(p.G32lo)[k * ne + e] = (float)(g - (double)(float)g);
    }
    double w = 0.166666666667 * fabs(J);
    wJ[e] = w;
    if (wJ32) wJ32[e] = (float)w;
    if (p.wJ32lo) const_cast<float *>(p.wJ32lo)[e] = (float)(w - (double)(float)w);
    double v6;   // 6V, signed: the edge determinant of the inscribed-sphere volume
    double L = char_length_ref(pts, &v6);
    Lref[e] = L;
    if (p.fxE) write_fixed_arrays(p, e, pts);
    // A reference sliver (6V below 0.063 |e1||e2||e3|) gets a negative FP32
    // length: the FP32 CFL screens then always recompute it in FP64 (the mixed
    // screen rebuilds the reference edges from G in FP32, which loses accuracy
    // on such a tet).  Lref itself is unchanged.
    {
        double e1[3], e2[3], e3[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            e1[i] = pts[3 + i] - pts[i];
            e2[i] = pts[6 + i] - pts[i];
            e3[i] = pts[9 + i] - pts[i];
        }
        const double l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
        const double l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
        const double l3 = e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2];
        const bool sliver = !(v6 * v6 >= 4e-3 * l1 * l2 * l3);
        Lref32[e] = sliver ? -(float)L : (float)L;
    }
}

// The FP32 element arrays of a precision mode that a handle starts using after
// its set-up (a later solver block in another mode), from the FP64 set-up data
// and X: the same conversions setup_elements_kernel makes, so the same bits.
__global__ void mode_arrays_kernel(Problem p, float *G32, float *wJ32, float *G32lo, float *wJ32lo)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const long long ne = p.ne;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const double g = p.G[k * ne + e];
        if (G32) G32[k * ne + e] = (float)g;
        if (G32lo) G32lo[k * ne + e] = (float)(g - (double)(float)g);
    }
    const double w = p.wJ[e];
    if (wJ32) wJ32[e] = (float)w;
    if (wJ32lo) wJ32lo[e] = (float)(w - (double)(float)w);
}

// Problem::fxE, fxS, fxD and fxw of a handle whose FP64 block starts after its
// set-up: what setup_elements_kernel writes, from X.
__global__ void fixed_arrays_kernel(Problem p)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double pts[12];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int i = 0; i < 3; i++) pts[k * 3 + i] = p.X[i * p.nn + nd[k]];
    write_fixed_arrays(p, e, pts);
}

// Previous-step F diagonal for the bulk viscosity, from displacement u, in the
// reference's order of F (constitutiveManager.cpp:151-164): what the Gauss
// points' previous state holds at the start of a block (the last step's F, or
// I from rest).
__global__ void visc_init_kernel(Problem p, const double *u)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const long long ne = p.ne, nn = p.nn;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double dphi[12];
#pragma unroll
    for (int k = 0; k < 9; k++) dphi[3 + k] = p.G[k * ne + e];
#pragma unroll
    for (int j = 0; j < 3; j++) dphi[j] = (-dphi[3 + j] - dphi[6 + j]) - dphi[9 + j];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        double F = 0.;
        F += 1.;
#pragma unroll
        for (int a = 0; a < 4; a++) F += dphi[a * 3 + i] * u[nd[a] + i * nn];
        if (p.visc_f0) p.visc_f0[i * ne + e] = F;
        if (p.visc_h0) p.visc_h0[i * ne + e] = (float)(F - 1.0);
    }
}

// constitutiveAlgorithms.cpp:191-205 (rho wJ phi_a phi_b summed over b) and
// solverExplicit.cpp:429-459 (element-order sum per node).
__global__ void setup_mass_kernel(Problem p, double *mass, double *minv)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.nn) return;
    const double phi = -1.0 * 0.25 - 1.0 * 0.25 - 1.0 * 0.25 + 1.0;
    double m = 0;
    const int k1 = p.node_ptr[i + 1];
    // the incidences' loads eight at a time, then their sums in element order
    for (int k = p.node_ptr[i]; k < k1; k += 8) {
        double w[8], r[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (k + j < k1) {
                const long long e = p.node_inc[k + j] >> 2;
                w[j] = p.wJ[e];
                r[j] = mat_of(p, e).rho;
            }
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (k + j < k1) {
                // me = 0 + z + z + z + z over the four corners b, z = ((wJ rho) phi) phi:
                // that sum is (3z) + z bit for bit (0 + z = z and z + z = 2z are exact,
                // 2z + z rounds 3z once); a z of -0 gives -0 instead of +0, which adds
                // to m the same way
                const double z = w[j] * r[j] * phi * phi;
                m += __dadd_rn(__dmul_rn(3.0, z), z);
            }
    }
    mass[i] = m;
    minv[i] = 1.0 / m;
}

// boundaryConditions.cpp:1146-1171 BCsGravity: -w rho |J| g phi_a on the z DOF
// of each corner (|J| as classGPs::getJ keeps it), summed per node in element order.
__global__ void setup_gravity_elem_kernel(Problem p, double g, double *grav_e)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const long long nn = p.nn;
    int4 cn = p.conn[e];
    int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double M[9];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) M[i * 3 + j] = p.X[i * nn + nd[j + 1]] - p.X[i * nn + nd[0]];
    const double w = 0.166666666667, phi = -1.0 * 0.25 - 1.0 * 0.25 - 1.0 * 0.25 + 1.0;
    grav_e[e] = -w * mat_of(p, e).rho * fabs(det3_ref(M)) * g * phi;
}

__global__ void setup_gravity_node_kernel(Problem p, const double *grav_e, double *grav_n)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.nn) return;
    double s = 0;
    for (int k = p.node_ptr[i]; k < p.node_ptr[i + 1]; k++) s += grav_e[p.node_inc[k] >> 2];
    grav_n[i] = s;
}

// Contributions of the traction and pressure faces for the step whose control
// slot `parity` the node kernel just wrote, at that step's time and
// displacement, in the reference's operation order (boundaryConditions.cpp:
// 218-275 BCsTractionInst/Ramp, :370-505 BCsPressureRamp/Inst; amounts from
// classNeumannBCs.h:57-181).  Pressure follows the face: n = F^-T n0 with F of
// the bulk tet by classSpatialPoint::getF (classSpatialPoint.cpp:41-66):
// F_ij = 0 + sum_a dphi_aj u_ai (corner order) + delta_ij.
__global__ void face_load_kernel(Problem p, int parity, bool mixed)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= p.nfaces) return;
    const Ctrl c = p.ctrl[parity];
    if (!c.ran) return;
    const double t = c.t;
    const FaceLoad L = p.faces[f];
    const bool ramp = L.kind == MSX_LOAD_TRACTION_RAMP || L.kind == MSX_LOAD_PRESSURE_RAMP;
    const bool pressure = L.kind == MSX_LOAD_PRESSURE_INST || L.kind == MSX_LOAD_PRESSURE_RAMP;
    double amount[3] = {0.0, 0.0, 0.0};
    if (t >= L.t0 && t <= L.tf)
        for (int i = 0; i < (pressure ? 1 : 3); i++) amount[i] = ramp ? L.value[i] / (L.tf - L.t0) * (t - L.t0) : L.value[i];
    double *out = p.fcon + (long long)L.con * 3;
    if (!pressure) {
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) out[a * 3 + i] = L.wabsJ * L.phi[a] * amount[i];
        return;
    }
    const long long nn = p.nn, ne = p.ne, e = L.tet;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double dphi[12];
    for (int a = 1; a < 4; a++)
        for (int j = 0; j < 3; j++) dphi[a * 3 + j] = p.G[((a - 1) * 3 + j) * ne + e];
    for (int j = 0; j < 3; j++) dphi[j] = ((-dphi[3 + j]) - dphi[6 + j]) - dphi[9 + j];
    double F[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int a = 0; a < 4; a++) {
        double disp[3];
        for (int i = 0; i < 3; i++) {
            const long long dof = nd[a] + i * nn;
            disp[i] = mixed ? (double)p.uhl[dof].x + (double)p.uhl[dof].y : p.u[dof];
        }
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) F[i * 3 + j] += dphi[a * 3 + j] * disp[i];
    }
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) F[i * 3 + j] += (i == j ? 1.0 : 0.0);
    double Fi[9], n[3];
    const double Jac = det3_ref(F);
    inv3_ref(F, Fi);
    for (int i = 0; i < 3; i++) {
        n[i] = 0;
        for (int j = 0; j < 3; j++) n[i] += Fi[j * 3 + i] * L.n0[j];
    }
    if (L.kind == MSX_LOAD_PRESSURE_RAMP) {
        // the bulk tet's shape function of its first node at natural coordinates 0 is 1
        for (int i = 0; i < 3; i++) out[i] = L.wabsJ * 1.0 * Jac * amount[0] * n[i];
    } else {
        for (int a = 0; a < 3; a++)
            for (int i = 0; i < 3; i++) out[a * 3 + i] = L.wabsJ * L.phi[a] * Jac * amount[0] * n[i];
    }
}

// Node data extraction (dataExtraction.cpp:778-840): the displacement, the
// external force of the last step at its time t, or the internal force summed
// from zero in element order (computeInternalForce, solverExplicit.cpp:363-379)
// from the corner forces the last element kernel left: element order in the
// reference-order mode, the node's CSR slots (also element order) otherwise.
__global__ void node_values_kernel(Problem p, int mode, int field, int comp, const int *nodes, long long n, double t,
                                   double *out)
{
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const long long i = nodes[j], dof = i + comp * p.nn;
    double v = 0.0;
    if (field == MSX_FIELD_DISPLACEMENT) {
        v = p.u[dof];
    } else if (field == MSX_FIELD_EXTERNAL_FORCE) {
        if (p.ext_ptr) v = ext_force_dof(p, dof, t);
    } else {
        for (int k = p.node_ptr[i]; k < p.node_ptr[i + 1]; k++) {
            if (mode == MODE_EXACT) v += p.fe[(long long)p.node_inc[k] * 3 + comp];
            else if (mode == MODE_MIXED) v += (double)p.fe32[(long long)k * 4 + comp];
            else if (mode == MODE_DW) {
                const float2 w = reinterpret_cast<const float2 *>(p.fe)[(long long)k * 3 + comp];
                v += (double)w.x + (double)w.y;
            } else v += p.fe[(long long)k * 3 + comp];
        }
    }
    out[j] = v;
}

// solvers.cpp:276-287 (uK == nullptr) and :296-320: element min into dtmin[slot]
__global__ void __launch_bounds__(kElemBlock) initial_cfl_kernel(Problem p, const double *uK, int slot)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double v = INFINITY;
    if (e < p.ne) {
        const MatParams &m = mat_of(p, e);
        if (!uK) {
            v = p.Lref[e] / m.c;
        } else {
            int4 cn = p.conn[e];
            int nd[4] = {cn.x, cn.y, cn.z, cn.w};
            double x[12];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    x[a * 3 + k] = p.X[k * p.nn + nd[a]];
                    x[a * 3 + k] += uK[p.nn * k + nd[a]];
                }
            double dist = char_length_ref(x);
            double Lr = p.Lref[e];
            v = ((dist < Lr) ? dist : Lr) / m.c;
        }
    }
    block_min_to(v, p.dtmin + slot);
}

// Output fields of one element from the current u, in the reference's order:
// Cauchy (NH: the law's sigma, hyperElasticNeoHookean.cpp:113-124; other laws
// P F^T / J, maths.cpp:1250-1254), Green-Lagrange E (maths.cpp:1227-1243) and
// von Mises (maths.cpp:1261-1271).
__global__ void element_fields_kernel(Problem p, double t, double *cauchy, double *gl, double *vms)
{
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    if (elem_dead(p, e, t)) {   // never updated: the Gauss point's initial, zero state
#pragma unroll
        for (int k = 0; k < 9; k++) {
            if (cauchy) cauchy[e * 9 + k] = 0.0;
            if (gl) gl[e * 9 + k] = 0.0;
        }
        if (vms) vms[e] = 0.0;
        return;
    }
    const long long ne = p.ne, nn = p.nn;
    int4 cn = p.conn[e];
    int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    double dphi[12];
#pragma unroll
    for (int k = 0; k < 9; k++) dphi[3 + k] = p.G[k * ne + e];
#pragma unroll
    for (int j = 0; j < 3; j++) dphi[j] = (-dphi[3 + j] - dphi[6 + j]) - dphi[9 + j];
    double F[9], P[9], S[9], E[9];
#pragma unroll
    for (int i = 0; i < 9; i++) F[i] = 0.;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        F[i * 3 + i] += 1.;
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int j = 0; j < 3; j++) F[i * 3 + j] += dphi[a * 3 + j] * p.u[nd[a] + i * nn];
    }
    const MatParams &m = mat_of(p, e);
    if (m.law == 0) {
        double B[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                double c = 0;
#pragma unroll
                for (int k = 0; k < 3; k++) c += F[i * 3 + k] * F[j * 3 + k];
                B[i * 3 + j] = c;
            }
        double J = det3_ref(F);
        double trB = 0;
#pragma unroll
        for (int i = 0; i < 3; i++) trB += B[i * 3 + i];
        double fact1 = pow(J, 5.0 / 3.0);
        double fact2 = m.mu / fact1;
#pragma unroll
        for (int i = 0; i < 9; i++) S[i] = 0 + fact2 * B[i];
        double fact3 = -(m.mu / 3.0) * trB / fact1 + m.K1 * (J - 1.0);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) S[i * 3 + j] += fact3 * (i == j ? 1.0 : 0.0);
    } else {
        stress_ref(m, F, P);
        double detJinv = 1. / det3_ref(F);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                double c = 0;
#pragma unroll
                for (int k = 0; k < 3; k++) c += P[i * 3 + k] * F[j * 3 + k];
                S[i * 3 + j] = c;
            }
#pragma unroll
        for (int i = 0; i < 9; i++) S[i] = S[i] * detJinv;
    }
    // the compressible neo-Hookean law never updates its Green-Lagrange strain
    // (hyperElasticNeoHookean.cpp:221-289), so the reference reports zero; the
    // linear-elastic law stores its small strain there (linearElastic.cpp:71-76)
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double c = 0;
#pragma unroll
            for (int k = 0; k < 3; k++) c += F[k * 3 + i] * F[k * 3 + j];
            E[i * 3 + j] = m.law == 1 ? 0.0
                         : m.law == 3 ? 0.5 * (F[i * 3 + j] + F[j * 3 + i] - 2. * (i == j ? 1. : 0.))
                                      : 0.5 * (c - (i == j ? 1.0 : 0.0));
        }
    if (cauchy)
#pragma unroll
        for (int k = 0; k < 9; k++) cauchy[e * 9 + k] = S[k];
    if (gl)
#pragma unroll
        for (int k = 0; k < 9; k++) gl[e * 9 + k] = E[k];
    if (vms)
        vms[e] = sqrt(0.5 * ((S[0] - S[4]) * (S[0] - S[4]) + (S[4] - S[8]) * (S[4] - S[8]) +
                             (S[8] - S[0]) * (S[8] - S[0]) + 6 * (S[1] * S[1] + S[2] * S[2] + S[5] * S[5])));
}

// One Gauss point's element-extraction value (msx_element_quantity) at the
// current u, v, in the reference's operation order: getValueAtGP
// (dataExtraction.cpp:508-563; Cauchy = P F^T / det F, classStates.cpp:309-316),
// the laws' defoEnergy (hyperElasticNeoHookean.cpp:291-304,
// hyperElasticStVenantKirchhoff.cpp:251-274; the Neo-Hookean law keeps the
// zero default, constitutiveModels.h:91-94), kineticEnergy's density at the
// centroid, where every shape function is 0.25 (dataExtraction.cpp:626-688),
// and volume's wJ det F (:690-748).  The internal variables read zero: no law
// here has more than one (getValueAtGP wants more than k for INVAR k).
__device__ double element_quantity_ref(const Problem &p, int q, long long e, double t)
{
    if (elem_dead(p, e, t)) return 0.0;   // dataExtraction.cpp:510
    if (q >= MSX_ELEM_INVAR1 && q <= MSX_ELEM_INVAR6) return 0.0;
    const long long ne = p.ne, nn = p.nn;
    const int4 cn = p.conn[e];
    const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
    const MatParams &m = mat_of(p, e);
    if (q == MSX_ELEM_KIN_ENERGY) {
        double vel[3] = {0., 0., 0.}, val = 0;
        for (int a = 0; a < 4; a++)
            for (int j = 0; j < 3; j++) vel[j] += 0.25 * p.v[nd[a] + j * nn];
        for (int j = 0; j < 3; j++) val += 0.5 * m.rho * vel[j] * vel[j];
        return val;
    }
    if (q == MSX_ELEM_DEFO_ENERGY && m.law == 0) return 0.0;
    double dphi[12];
    for (int k = 0; k < 9; k++) dphi[3 + k] = p.G[k * ne + e];
    for (int j = 0; j < 3; j++) dphi[j] = (-dphi[3 + j] - dphi[6 + j]) - dphi[9 + j];
    double F[9];
    for (int i = 0; i < 9; i++) F[i] = 0.;
    for (int i = 0; i < 3; i++) {
        F[i * 3 + i] += 1.;
        for (int a = 0; a < 4; a++)
            for (int j = 0; j < 3; j++) F[i * 3 + j] += dphi[a * 3 + j] * p.u[nd[a] + i * nn];
    }
    if (q >= MSX_ELEM_FXX && q <= MSX_ELEM_FZZ) return F[q - MSX_ELEM_FXX];
    if (q == MSX_ELEM_VOLUME) return p.wJ[e] * det3_ref(F);
    if (q == MSX_ELEM_DEFO_ENERGY && m.law == 3) {
        // linearElastic.cpp:88-101: 0.5 (P:F - P:I), contractions summed from 0
        double P[9], a = 0, b = 0;
        stress_ref(m, F, P);
        for (int i = 0; i < 9; i++) a += P[i] * F[i];
        for (int i = 0; i < 9; i++) b += P[i] * ((i % 4) == 0 ? 1. : 0.);
        return 0.5 * (a - b);
    }
    if (q == MSX_ELEM_DEFO_ENERGY) {
        double C[9];
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) {
                double c = 0;
                for (int k = 0; k < 3; k++) c += F[k * 3 + i] * F[k * 3 + j];
                C[i * 3 + j] = c;
            }
        if (m.law == 1) {
            const double J = det3_ref(F);
            double tr = 0;
            for (int i = 0; i < 3; i++) tr += C[i * 3 + i];
            return 0.5 * m.lambda * log(J) * log(J) - m.mu * log(J) + 0.5 * m.mu * tr;
        }
        double E[9], S[9], trE = 0, w = 0;
        for (int i = 0; i < 9; i++) E[i] = 0.5 * (C[i] - ((i % 4) == 0 ? 1.0 : 0.0));
        for (int i = 0; i < 3; i++) trE += E[i * 3 + i];
        for (int i = 0; i < 9; i++) S[i] = E[i] * m.mu2;
        for (int i = 0; i < 3; i++) S[i * 3 + i] += m.lam_stvk * trE;
        for (int i = 0; i < 9; i++) w += S[i] * E[i];
        return 0.5 * w;
    }
    double P[9];
    stress_ref(m, F, P);
    if (q >= MSX_ELEM_PXX && q <= MSX_ELEM_PZZ) return P[q - MSX_ELEM_PXX];
    // SVM, KVM
    const double detF = det3_ref(F), detJinv = 1. / detF;
    double S[9];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double c = 0;
            for (int k = 0; k < 3; k++) c += P[i * 3 + k] * F[j * 3 + k];
            S[i * 3 + j] = c;
        }
    for (int i = 0; i < 9; i++) S[i] = S[i] * detJinv;
    const double svm = sqrt(0.5 * ((S[0] - S[4]) * (S[0] - S[4]) + (S[4] - S[8]) * (S[4] - S[8]) +
                                   (S[8] - S[0]) * (S[8] - S[0]) + 6 * (S[1] * S[1] + S[2] * S[2] + S[5] * S[5])));
    return q == MSX_ELEM_KVM ? svm * detF : svm;
}

__global__ void element_values_kernel(Problem p, int q, const int *elems, long long n, double t, double *out)
{
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) out[j] = element_quantity_ref(p, q, elems ? elems[j] : j, t);
}

// The element-extraction reduction in two fixed-shape passes, so the result
// does not depend on the GPU or the run: kReduceBlocks blocks each take a
// grid-stride share in index order and fold it in a shared-memory tree into
// part[2b] (the weighted sum, or the extreme) and part[2b+1] (the sum of dV);
// one block then folds the partials the same way.
// Blocks of 64 threads: on meshes of less than kReduceBlocks x kReduceThreads
// elements the FP64 work of an element spreads evenly over the SMs' pipes (48,000
// elements: 750 blocks of two warps against 188 of eight, 152 SMs).
constexpr int kReduceBlocks = 2048, kReduceThreads = 64, kFinishThreads = 256;

__device__ __forceinline__ void fold_pair(int op, double &s, double &w, double s2, double w2)
{
    if (op == MSX_OP_MAX) s = s2 > s ? s2 : s;
    else if (op == MSX_OP_MIN) s = s2 < s ? s2 : s;
    else s += s2;
    w += w2;
}

template <int THREADS>
__device__ __forceinline__ void block_fold(int op, double &s, double &w)
{
    __shared__ double ss[THREADS], ws[THREADS];
    ss[threadIdx.x] = s;
    ws[threadIdx.x] = w;
    __syncthreads();
    for (int h = THREADS / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            double a = ss[threadIdx.x], b = ws[threadIdx.x];
            fold_pair(op, a, b, ss[threadIdx.x + h], ws[threadIdx.x + h]);
            ss[threadIdx.x] = a;
            ws[threadIdx.x] = b;
        }
        __syncthreads();
    }
    s = ss[0];
    w = ws[0];
}

__device__ __forceinline__ double reduce_identity(int op)
{
    return op == MSX_OP_MAX ? -INFINITY : (op == MSX_OP_MIN ? INFINITY : 0.0);
}

__global__ void __launch_bounds__(kReduceThreads) element_reduce_kernel(Problem p, int q, int op, const int *elems,
                                                                        long long n, double t, double *part)
{
    double s = reduce_identity(op), w = 0.0;
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
        if (q == MSX_ELEM_EXTERNAL_ENERGY) {
            s += p.u[j] * (p.ext_ptr ? ext_force_dof(p, j, t) : 0.0);
            continue;
        }
        const long long e = elems ? elems[j] : j;
        // the energies and the volume skip dead Gauss points altogether (:577-578, 644-645, 706-707)
        if ((q == MSX_ELEM_DEFO_ENERGY || q == MSX_ELEM_KIN_ENERGY || q == MSX_ELEM_VOLUME) && elem_dead(p, e, t))
            continue;
        const double v = element_quantity_ref(p, q, e, t), dV = p.wJ[e];
        fold_pair(op, s, w, q == MSX_ELEM_VOLUME || op == MSX_OP_MAX || op == MSX_OP_MIN ? v : v * dV, dV);
    }
    block_fold<kReduceThreads>(op, s, w);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = s;
        part[2 * blockIdx.x + 1] = w;
    }
}

__global__ void __launch_bounds__(kFinishThreads) element_reduce_finish_kernel(int q, int op, const double *part,
                                                                               double *out)
{
    double s = reduce_identity(op), w = 0.0;
    for (int b = threadIdx.x; b < kReduceBlocks; b += blockDim.x) fold_pair(op, s, w, part[2 * b], part[2 * b + 1]);
    block_fold<kFinishThreads>(op, s, w);
    if (threadIdx.x == 0) *out = op == MSX_OP_MEAN ? s / w : s;
}

#endif  // MSX_SETUP_KERNELS

// f_int gather for the internal-force hook: fint[node + c*nn] in element order,
// a thread a node and component, its terms loaded eight at a time before they
// are added (one after another they cost a memory latency each; 39,304 nodes in
// FP64: 10 us)
template <int MODE>
__global__ void gather_kernel(Problem p, double *fint)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / 3;
    const int c = (int)(t - 3 * i);
    if (i >= p.nn) return;
    double s = 0;
    const int k1 = p.node_ptr[i + 1];
    for (int k0 = p.node_ptr[i]; k0 < k1; k0 += 8) {
        double f[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            f[j] = 0.0;
            if (k0 + j >= k1) continue;
            // reference-order corner forces are in element order, the others in CSR slots
            const long long inc = MODE == MODE_EXACT ? p.node_inc[k0 + j] : k0 + j;
            if (MODE == MODE_MIXED) {
                f[j] = (double)p.fe32[inc * 4 + c];
            } else if (MODE == MODE_DW) {
                const float2 w = reinterpret_cast<const float2 *>(p.fe)[inc * 3 + c];
                f[j] = (double)w.x + (double)w.y;
            } else {
                f[j] = p.fe[inc * 3 + c];
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (k0 + j < k1) s += f[j];
    }
    fint[i + c * p.nn] = s;
}

inline unsigned grid_for(long long n, int block) { return (unsigned)((n + block - 1) / block); }

}  // namespace msx
