// msx_fast.cu -- FP64 (contracted, simplified algebra), double-word and
// mixed-precision kernels.  The tiled step kernels of single solves (msx_run)
// and of the pool are the same loops, instantiated here only, so a pooled solve
// gives the bits of the solve run alone.
#include "msx_device.cuh"

namespace msx {

void launch_internal_force_fp64(const Problem &p, double *fint, cudaStream_t s)
{
    elem_force_kernel_fp64<<<grid_for(p.ne, kElemBlock), kElemBlock, 0, s>>>(p, 0);
    gather_kernel<MODE_FP64><<<grid_for(3 * p.nn, 256), 256, 0, s>>>(p, fint);
}

void launch_internal_force_mixed(const Problem &p, double *fint, cudaStream_t s)
{
    elem_force_kernel_mixed<<<grid_for(p.ne, kElemBlock), kElemBlock, 0, s>>>(p, 0);
    gather_kernel<MODE_MIXED><<<grid_for(3 * p.nn, 256), 256, 0, s>>>(p, fint);
}

void launch_internal_force_dw(const Problem &p, double *fint, cudaStream_t s)
{
    elem_force_kernel_dw<<<grid_for(p.ne, kElemBlock), kElemBlock, 0, s>>>(p, 0);
    gather_kernel<MODE_DW><<<grid_for(3 * p.nn, 256), 256, 0, s>>>(p, fint);
}

void launch_tiled_node(const Problem *descs, const Tile *ntiles, int *counts, int mode, int parity, int grid,
                       int threads, cudaStream_t s)
{
    if (mode == MODE_MIXED)
        pool_node_kernel<MODE_MIXED><<<grid, threads, 0, s>>>(descs, ntiles, counts + 3, parity);
    else if (mode == MODE_DW)
        pool_node_kernel<MODE_DW><<<grid, threads, 0, s>>>(descs, ntiles, counts + 3, parity);
    else
        pool_node_kernel<MODE_FP64><<<grid, threads, 0, s>>>(descs, ntiles, counts + 3, parity);
}

void launch_tiled_elem(const Problem *descs, const Tile *etiles, int *counts, int mode, int parity, int grid,
                       int threads, cudaStream_t s)
{
    if (mode == MODE_MIXED)
        pool_elem_kernel<MODE_MIXED><<<grid, threads, 0, s>>>(descs, etiles, counts, parity);
    else if (mode == MODE_DW)
        pool_elem_kernel<MODE_DW><<<grid, threads, 0, s>>>(descs, etiles, counts, parity);
    else
        pool_elem_kernel<MODE_FP64><<<grid, threads, 0, s>>>(descs, etiles, counts, parity);
}

// A step kernel of one solve on n CTAs or the most that are resident, with
// programmatic dependent launch for small grids (SolveSched::pdl).
template <typename... ARGS>
static void launch_solve(void (*f)(const Problem, ARGS...), const Problem &p, const SolveSched &q, int n, int most,
                         cudaStream_t s, ARGS... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(n < most ? n : most);
    c.blockDim = dim3(q.threads);
    c.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    Problem P = p;
    P.dependent = c.numAttrs = n <= q.pdl ? 1 : 0;
    cudaLaunchKernelEx(&c, f, P, args...);
}

typedef void (*solve_node_fn)(const Problem, int);
typedef void (*solve_elem_fn)(const Problem, int, int, int *, int);

template <int MODE>
static solve_node_fn solve_node_variant(const SolveSched &q)
{
    if (!q.node_batch) return solve_node_kernel<MODE, false>;
    return q.threads == 128 ? solve_node_kernel<MODE, true, true> : solve_node_kernel<MODE, true>;
}

static solve_node_fn solve_node(int mode, const SolveSched &q)
{
    return mode == MODE_MIXED ? solve_node_variant<MODE_MIXED>(q)
                              : (mode == MODE_DW ? solve_node_variant<MODE_DW>(q) : solve_node_variant<MODE_FP64>(q));
}

// element birth and bulk viscosity are separate instantiations (never both: the host refuses that)
template <int MODE>
static solve_elem_fn solve_elem_variant(const Problem &p, const SolveSched &q)
{
    if (p.act_t) return solve_elem_kernel<MODE, true>;
    if (MODE == MODE_FP64 && q.fixed) return q.fixed == FIXED_CNH ? solve_elem_cnh_kernel : solve_elem_svk_kernel;
    return p.visc ? solve_elem_kernel<MODE, false, true> : solve_elem_kernel<MODE>;
}

static solve_elem_fn solve_elem(const Problem &p, int mode, const SolveSched &q)
{
    return mode == MODE_MIXED ? solve_elem_variant<MODE_MIXED>(p, q)
                              : (mode == MODE_DW ? solve_elem_variant<MODE_DW>(p, q) : solve_elem_variant<MODE_FP64>(p, q));
}

void launch_solve_node(const Problem &p, const SolveSched &q, int mode, int parity, cudaStream_t s)
{
    const int per = q.threads / 4;
    launch_solve(solve_node(mode, q), p, q, (int)((p.nn + per - 1) / per), q.node_grid, s, parity);
}

void launch_solve_elem(const Problem &p, const SolveSched &q, int *counts, int mode, int parity, cudaStream_t s)
{
    const int n = (int)((p.ne + q.elem_tile - 1) / q.elem_tile);
    launch_solve(solve_elem(p, mode, q), p, q, n, q.elem_grid, s, (int)q.elem_tile, (int)n, counts, parity);
}

// a32: the mixed mode, whose acceleration is one FP32 per DOF (mixed_a32)
__global__ void state_split_kernel(Problem p, bool a32)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * p.nn) return;
    p.uhl[i] = df_from(p.u[i]);
    p.vhl[i] = df_from(p.v[i]);
    if (a32) mixed_a32(p)[i] = (float)p.a[i];
    else p.ahl[i] = df_from(p.a[i]);
}

__global__ void state_merge_kernel(Problem p, bool a32)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * p.nn) return;
    float2 u = p.uhl[i], v = p.vhl[i];
    p.u[i] = (double)u.x + (double)u.y;
    p.v[i] = (double)v.x + (double)v.y;
    if (a32) {
        p.a[i] = (double)mixed_a32(p)[i];
    } else {
        const float2 a = p.ahl[i];
        p.a[i] = (double)a.x + (double)a.y;
    }
}

__global__ void u4_from_u_kernel(const double *u, double *u4, long long nn)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    reinterpret_cast<double2 *>(u4)[2 * i] = make_double2(u[i], u[nn + i]);
    reinterpret_cast<double2 *>(u4)[2 * i + 1] = make_double2(u[2 * nn + i], 0.0);
}

void launch_u4_from_u(const double *u, double *u4, long long nn, cudaStream_t s)
{
    u4_from_u_kernel<<<grid_for(nn, 256), 256, 0, s>>>(u, u4, nn);
}

__global__ void minv_split_kernel(const double *minv, float2 *minv2, long long nn)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nn) minv2[i] = df_from(minv[i]);
}

void launch_state_split(const Problem &p, bool mixed, cudaStream_t s)
{
    state_split_kernel<<<grid_for(3 * p.nn, 256), 256, 0, s>>>(p, mixed);
}

void launch_state_merge(const Problem &p, bool mixed, cudaStream_t s)
{
    state_merge_kernel<<<grid_for(3 * p.nn, 256), 256, 0, s>>>(p, mixed);
}

void launch_minv_split(const double *minv, float2 *minv2, long long nn, cudaStream_t s)
{
    minv_split_kernel<<<grid_for(nn, 256), 256, 0, s>>>(minv, minv2, nn);
}

__global__ void node_bc_scatter_kernel(int *node_bc, const int2 *nodes, long long n)
{
    long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) node_bc[nodes[k].x] = nodes[k].y;
}

void launch_node_bc_scatter(int *node_bc, long long nn, const int2 *nodes, long long n, cudaStream_t s)
{
    cudaMemsetAsync(node_bc, 0xFF, sizeof(int) * nn, s);   // -1: no entry
    if (n > 0) node_bc_scatter_kernel<<<grid_for(n, 256), 256, 0, s>>>(node_bc, nodes, n);
}

__global__ void abs_range_kernel(const double *x, long long n, unsigned long long *mm)
{
    unsigned long long lo = ~0ULL, hi = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(x[i]));
        if (b != 0) {
            lo = b < lo ? b : lo;
            hi = b > hi ? b : hi;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(mm, lo);
        atomicMax(mm + 1, hi);
    }
}

__global__ void abs_range_init_kernel(unsigned long long *mm)
{
    mm[0] = ~0ULL;
    mm[1] = 0;
}

void launch_abs_range(const double *x, long long n, unsigned long long *mm, cudaStream_t s)
{
    abs_range_init_kernel<<<1, 1, 0, s>>>(mm);
    abs_range_kernel<<<256, 256, 0, s>>>(x, n, mm);
}

static int ctas_per_sm(const void *kernel, int threads)
{
    int a = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, kernel, threads, 0);
    return a > 0 ? a : 1;
}

int solve_node_ctas(int mode, const SolveSched &q) { return ctas_per_sm((const void *)solve_node(mode, q), q.threads); }

int solve_elem_ctas(const Problem &p, int mode, const SolveSched &q)
{
    return ctas_per_sm((const void *)solve_elem(p, mode, q), q.threads);
}

int pool_ctas_per_sm(int mode, int threads, bool node)
{
    const void *f[3][2] = {{(const void *)pool_elem_kernel<MODE_FP64>, (const void *)pool_node_kernel<MODE_FP64>},
                           {(const void *)pool_elem_kernel<MODE_MIXED>, (const void *)pool_node_kernel<MODE_MIXED>},
                           {(const void *)pool_elem_kernel<MODE_DW>, (const void *)pool_node_kernel<MODE_DW>}};
    return ctas_per_sm(f[mode == MODE_MIXED ? 1 : (mode == MODE_DW ? 2 : 0)][node], threads);
}

}  // namespace msx
