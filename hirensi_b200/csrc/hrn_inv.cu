// hrn_inv.cu -- device side of the model update of the inversion loop
// (S4/Program_Main.F90:411-896, S4/LBFGS_Coupled.F90, S4/Control_Problem_Operators.F90):
// FP64 vector algebra with deterministic reductions, the TV regularization and
// lumped gradient mass element kernels, and the coupled L-BFGS two-loop
// recursion.  All vectors are nodal (length nj) FP64 device arrays; the driver
// keeps its control flow on the host and reads back scalars only.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "hrn_internal.h"
#include "hrn_pdl.cuh"

namespace hrn {

constexpr int kRedBlocks = 296;   // 2 x 148 SMs
constexpr int kRedThreads = 256;

// Sum (or maximum) of N values over a block of a whole number of warps, in a fixed
// order; the result is thread 0's.
template <int N, bool MAX>
__device__ __forceinline__ void block_reduce(double (&v)[N])
{
    __shared__ double sh[N][32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const double o = __shfl_down_sync(0xffffffffu, v[k], off);
            v[k] = MAX ? fmax(v[k], o) : v[k] + o;
        }
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < N; ++k) sh[k][warp] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < N; ++k)
            for (int w = 1; w < nw; ++w) v[k] = MAX ? fmax(v[k], sh[k][w]) : v[k] + sh[k][w];
    __syncthreads();
}

// True in the block that finishes last, which then sees every block's partials; the
// count returns to zero for the next launch.
__device__ __forceinline__ bool last_block(unsigned *count)
{
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
        if (last) *count = 0;
        __threadfence();
    }
    __syncthreads();
    return last;
}

// out[0] (host memory) = dot, 2-norm or inf-norm, in one launch: block partials in a
// fixed order, summed in a fixed order by the block that finishes last.  A vector of
// 10^5 entries takes a few us of the device, so the call is bound by its launch and the
// synchronisation that hands the scalar over: no second launch (one thread over the
// partials) and no copy to pageable memory.  Eight such calls, TV and the direction on
// 46575 nodes with memory 5: 1226 us with both, 222 us in this form.
template <int KIND>
__global__ void __launch_bounds__(kRedThreads) k_reduce(int n, const double *__restrict__ x, const double *__restrict__ y,
                                                        double *part, unsigned *count, double *out)
{
    double acc[1] = {0.0};
    for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads) {
        if constexpr (KIND == 0) acc[0] += x[i] * y[i];             // dot
        else if constexpr (KIND == 1) acc[0] += x[i] * x[i];        // squared 2-norm
        else acc[0] = fmax(acc[0], fabs(x[i]));                     // inf-norm
    }
    block_reduce<1, KIND == 2>(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc[0];
    if (!last_block(count)) return;
    acc[0] = 0.0;
    for (int b = threadIdx.x; b < int(gridDim.x); b += kRedThreads) {
        const double p = __ldcg(part + b);
        acc[0] = KIND == 2 ? fmax(acc[0], p) : acc[0] + p;
    }
    block_reduce<1, KIND == 2>(acc);
    if (threadIdx.x == 0) out[0] = KIND == 1 ? sqrt(acc[0]) : acc[0];
}

// z = a x + b y  (y may be null: z = a x)
__global__ void k_axpby(int n, double a, const double *__restrict__ x, double b, const double *__restrict__ y, double *__restrict__ z)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        z[i] = y ? a * x[i] + b * y[i] : a * x[i];
}

__global__ void k_mul(int n, const double *__restrict__ x, const double *__restrict__ y, double *__restrict__ z)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) z[i] = x[i] * y[i];
}

__global__ void k_clip(int n, double lo, double hi, double *__restrict__ x)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = x[i];
        x[i] = v < lo ? lo : (v > hi ? hi : v);
    }
}

__global__ void k_gather(int n, const int32_t *__restrict__ map, const double *__restrict__ x, double *__restrict__ y)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = x[map[i]];
}

// ----------------------------------------------------------------------------
// element kernels over the regular domain (GLL points, one thread per point)

// local node of grid point x + 3 y + 9 z, and the derivative matrix of the 3-point GLL rule
__device__ const int v_node_at[27] = {3, 11, 0, 10, 20, 8, 2, 9, 1, 15, 24, 12, 23, 26, 21, 14, 22, 13, 7, 19, 4, 18, 25, 16, 6, 17, 5};
__constant__ double v_D[3][3] = {{-1.5, 2.0, -0.5}, {-0.5, 0.0, 0.5}, {0.5, -2.0, 1.5}};

// TV regularization (ELEMENT_TV_TN_Reg_3D, S4/Element_Matrices_3D.F90:1899-2074, unweighted):
// per point, ER = sum_k dN_I/dx_k dN_J/dx_k, vh = ER e, den = sqrt(e.vh + 0.01),
// E_Reg += vh / den * w detJ, cost += (e.vh) / den * w detJ.  With the GLL rule
// vh_I = sum_k dN_I/dx_k g_k and e.vh = |g|^2 where g = grad e at the point, and
// only the 7 nodes on the lines through the point receive a contribution.
// One thread per point, 8 elements to a block: the points exchange nodal values and
// fluxes through shared memory, so that an element sends one atomic per node and field
// (27 x 2) where a scatter from the points sent 18 per point (27 x 18); the block that
// finishes last sums the cost, and the tables are initialised with the module.
constexpr int kTvElems = 8, kTvThreads = 224;   // 216 points, whole warps

__global__ void __launch_bounds__(kTvThreads) k_tv(int nel_rd, const int32_t *__restrict__ rd_elems, const int32_t *__restrict__ inod,
                                                   const double *__restrict__ geom, const double *__restrict__ lam,
                                                   const double *__restrict__ mu, double *__restrict__ reg_l,
                                                   double *__restrict__ reg_m, double *cost_part, unsigned *count, double *cost)
{
    __shared__ double val[2][kTvElems * 27], flux[2][3][kTvElems * 27];
    const int le = threadIdx.x / 27, q = threadIdx.x % 27, e = blockIdx.x * kTvElems + le;
    const bool on = threadIdx.x < kTvElems * 27 && e < nel_rd;
    const int qi[3] = {q % 3, (q / 3) % 3, q / 9};
    const int stride[3] = {1, 3, 9};
    const int at = threadIdx.x;
    int node = 0;
    if (on) {
        node = inod[size_t(rd_elems[e]) * 27 + v_node_at[q]];
        val[0][at] = mu[node];
        val[1][at] = lam[node];
    }
    __syncthreads();
    double cost2[2] = {0.0, 0.0};   // lambda, mu
    if (on) {
        const double *gp = geom + (size_t(e) * 27 + q) * 10;
        double g[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) g[k] = gp[k];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            double dxi[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double *v = val[f] + at - qi[m] * stride[m];   // the line through the point
                dxi[m] = 0.0;
#pragma unroll
                for (int u = 0; u < 3; ++u) dxi[m] += v_D[qi[m]][u] * v[u * stride[m]];
            }
            double gr[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) gr[k] = dxi[0] * g[0 * 3 + k] + dxi[1] * g[1 * 3 + k] + dxi[2] * g[2 * 3 + k];
            const double num = gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2];
            const double den = sqrt(num + 0.01);
            const double w = g[9] / den;
            // vh_I = sum_k DFX(I,k) gr_k with DFX(I,k) = sum_m DFXI(I,m) DJI(m,k)
#pragma unroll
            for (int m = 0; m < 3; ++m) flux[f][m][at] = (g[m * 3 + 0] * gr[0] + g[m * 3 + 1] * gr[1] + g[m * 3 + 2] * gr[2]) * w;
            cost2[1 - f] = num / den * g[9];
        }
    }
    __syncthreads();
    if (on) {
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            double s = 0.0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double *v = flux[f][m] + at - qi[m] * stride[m];
#pragma unroll
                for (int u = 0; u < 3; ++u) s += v_D[u][qi[m]] * v[u * stride[m]];
            }
            atomicAdd((f == 0 ? reg_m : reg_l) + node, s);
        }
    }
    block_reduce<2, false>(cost2);
    if (threadIdx.x == 0) {
        cost_part[2 * blockIdx.x] = cost2[0];
        cost_part[2 * blockIdx.x + 1] = cost2[1];
    }
    if (!last_block(count)) return;
    cost2[0] = cost2[1] = 0.0;
    for (int b = threadIdx.x; b < int(gridDim.x); b += kTvThreads) {
        cost2[0] += __ldcg(cost_part + 2 * b);
        cost2[1] += __ldcg(cost_part + 2 * b + 1);
    }
    block_reduce<2, false>(cost2);
    if (threadIdx.x == 0) {
        cost[0] = cost2[0];
        cost[1] = cost2[1];
    }
}

// Lumped gradient mass (ELEMENT_R_Mg_3D diagonal): Mg(node) += w detJ at the node's point.
__global__ void k_gradient_mass(int nel_rd, const int32_t *__restrict__ rd_elems, const int32_t *__restrict__ inod,
                                const double *__restrict__ geom, double *__restrict__ mg)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nel_rd * 27) return;
    const int e = t / 27, q = t % 27;
    atomicAdd(mg + inod[size_t(rd_elems[e]) * 27 + v_node_at[q]], geom[size_t(t) * 10 + 9]);
}

// ----------------------------------------------------------------------------
// host helpers

static int grid_for(int n) { return std::min(std::max((n + 255) / 256, 1), 148 * 8); }

// Reduction workspace: partials, then the count of finished blocks (zero between launches).
static int red_space(hrn_ctx *c)
{
    HRN_CUDA(c, c->h_red.alloc(4 * sizeof(double)));
    if (!c->d_red.p) {
        HRN_CUDA(c, c->d_red.alloc((kRedBlocks + 1) * 8));
        // zeroed now, not on a stream that may be under capture
        cudaError_t e = cudaMemset(c->d_red.p, 0, c->d_red.bytes);
        if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
        if (e != cudaSuccess) {
            c->d_red.release();
            return cuda_error(c, e, "zeroing the reduction workspace");
        }
    }
    return 0;
}

int vec_reduce(hrn_ctx *c, int kind, int n, const double *x, const double *y, double *out)
{
    if (int rc = red_space(c)) return rc;
    double *part = c->d_red.as<double>(), *res = c->h_red.as<double>();
    unsigned *count = reinterpret_cast<unsigned *>(part + kRedBlocks);
    const int nb = std::min(std::max((n + kRedThreads - 1) / kRedThreads, 1), kRedBlocks);
    if (kind == 0) k_reduce<0><<<nb, kRedThreads, 0, c->stream>>>(n, x, y, part, count, res);
    else if (kind == 1) k_reduce<1><<<nb, kRedThreads, 0, c->stream>>>(n, x, y, part, count, res);
    else k_reduce<2><<<nb, kRedThreads, 0, c->stream>>>(n, x, y, part, count, res);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));
    *out = *static_cast<volatile double *>(res);
    return 0;
}

int vec_axpby(hrn_ctx *c, int n, double a, const double *x, double b, const double *y, double *z)
{
    k_axpby<<<grid_for(n), 256, 0, c->stream>>>(n, a, x, b, y, z);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    return 0;
}

int regularization_tv(hrn_ctx *c, const double *lam, const double *mu, double *reg_l, double *reg_m, double *cost_l, double *cost_m)
{
    if (int rc = red_space(c)) return rc;
    HRN_CUDA(c, cudaMemsetAsync(reg_l, 0, size_t(c->nj) * 8, c->stream));
    HRN_CUDA(c, cudaMemsetAsync(reg_m, 0, size_t(c->nj) * 8, c->stream));
    const int nb = std::max((c->nel_rd + kTvElems - 1) / kTvElems, 1);
    HRN_CUDA(c, c->d_tv_part.alloc(size_t(2) * nb * 8));   // kept, so that repeated calls allocate nothing
    double *res = c->h_red.as<double>();
    k_tv<<<nb, kTvThreads, 0, c->stream>>>(c->nel_rd, c->d_rd_elems.as<int32_t>(), c->d_inod.as<int32_t>(),
                                           c->d_rd_geom.as<double>(), lam, mu, reg_l, reg_m, c->d_tv_part.as<double>(),
                                           reinterpret_cast<unsigned *>(c->d_red.as<double>() + kRedBlocks), res);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));
    *cost_l = static_cast<volatile double *>(res)[0];
    *cost_m = static_cast<volatile double *>(res)[1];
    return 0;
}

int gradient_mass(hrn_ctx *c, double *mg)
{
    HRN_CUDA(c, cudaMemsetAsync(mg, 0, size_t(c->nj) * 8, c->stream));
    const int th = 256;
    if (c->nel_rd > 0)
        k_gradient_mass<<<(c->nel_rd * 27 + th - 1) / th, th, 0, c->stream>>>(c->nel_rd, c->d_rd_elems.as<int32_t>(),
                                                                               c->d_inod.as<int32_t>(), c->d_rd_geom.as<double>(), mg);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    return 0;
}

// ----------------------------------------------------------------------------
// coupled L-BFGS direction as a chain of launches

// Every launch updates q by one pair and leaves the block partials of the next pair's
// products (lambda and mu together); the next launch sums them again in every block, in
// one fixed order, so the recursion's scalars never leave the device.  Vectors of 10^5
// entries lie in L2 and a launch is bound by latency; 2 M + 1 launches, each started while
// the one before drains, take the place of 4 M + 6 reductions with a host synchronisation
// each (26 of the 34 in a model update with memory 5, 1226 us before and 222 us now).
constexpr int kDirThreads = 256, kDirBlocks = 592, kDirSums = 6;

struct DirArgs {
    int n;
    const double *q_l, *q_m;      // in
    double *out_l, *out_m;        // q after this pair
    const double *u_l, *u_m;      // vectors that the update adds
    const double *v_l, *v_m;      // vectors of the next products
    const double *part_in;
    double *part_out;             // null at the last pair
    double *rho, *alpha, *h0;     // rho and alpha of this pair, H0 of the call
    double *rho_out;              // host memory
};

// y = g - g_pre, s = m - m_pre; stores the pair (s restricted) and leaves y.s, y.y and
// the first products g.S of the new pair
__global__ void __launch_bounds__(kDirThreads) k_dir_pair(int n, const double *__restrict__ g_l, const double *__restrict__ g_m,
                                                          const double *__restrict__ g_l_pre, const double *__restrict__ g_m_pre,
                                                          const double *__restrict__ lam, const double *__restrict__ mu,
                                                          const double *__restrict__ lam_pre, const double *__restrict__ mu_pre,
                                                          const double *__restrict__ rs, double *__restrict__ Y_l,
                                                          double *__restrict__ Y_m, double *__restrict__ S_l,
                                                          double *__restrict__ S_m, double *__restrict__ part)
{
    dep_trigger();
    double v[kDirSums] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int i = blockIdx.x * kDirThreads + threadIdx.x; i < n; i += gridDim.x * kDirThreads) {
        const double a = g_l[i], b = g_m[i], r = rs[i];
        const double yl = a - g_l_pre[i], ym = b - g_m_pre[i], sl = lam[i] - lam_pre[i], sm = mu[i] - mu_pre[i];
        const double rl = sl * r, rm = sm * r;
        Y_l[i] = yl; Y_m[i] = ym; S_l[i] = rl; S_m[i] = rm;
        v[0] += a * rl; v[1] += b * rm;
        v[2] += yl * sl; v[3] += ym * sm;
        v[4] += yl * yl; v[5] += ym * ym;
    }
    block_reduce<kDirSums, false>(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < kDirSums; ++k) part[size_t(k) * gridDim.x + blockIdx.x] = v[k];
}

// One pair of the recursion.  LOOP 1: q -= alpha Y, alpha = rho q.S; LOOP 2: q += (alpha -
// rho q.Y) S.  FIRST: the new pair of loop 1 (rho and H0 from the sums); TAIL: the last
// pair of its loop (loop 1 then scales by H0, loop 2 negates).
template <int LOOP, bool FIRST, bool TAIL>
__global__ void __launch_bounds__(kDirThreads) k_dir_step(DirArgs A)
{
    dep_trigger();
    dep_wait();
    constexpr int N = FIRST ? kDirSums : 2;
    __shared__ double sc[2];
    double v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = 0.0;
    for (int b = threadIdx.x; b < int(gridDim.x); b += kDirThreads)
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] += __ldcg(A.part_in + size_t(k) * gridDim.x + b);
    block_reduce<N, false>(v);
    if (threadIdx.x == 0) {
        double rho, h0 = 0.0;
        if constexpr (FIRST) {
            rho = 1.0 / (v[2] + v[3]);
            h0 = (v[2] + v[3]) / (v[4] + v[5]);
            if (blockIdx.x == 0) { A.rho[0] = rho; A.h0[0] = h0; A.rho_out[0] = rho; }
        } else {
            rho = __ldcg(A.rho);
            if constexpr (LOOP == 1 && TAIL) h0 = __ldcg(A.h0);
        }
        const double d = rho * v[0] + rho * v[1];
        if constexpr (LOOP == 1) {
            if (blockIdx.x == 0) A.alpha[0] = d;
            sc[0] = -d;
            sc[1] = h0;
        } else {
            sc[0] = __ldcg(A.alpha) - d;
            sc[1] = -1.0;
        }
    }
    __syncthreads();
    const double w = sc[0], f = sc[1];
    double p[2] = {0.0, 0.0};
    for (int i = blockIdx.x * kDirThreads + threadIdx.x; i < A.n; i += gridDim.x * kDirThreads) {
        double a = __ldcg(A.q_l + i) + w * __ldcg(A.u_l + i), b = __ldcg(A.q_m + i) + w * __ldcg(A.u_m + i);
        if constexpr (TAIL) { a *= f; b *= f; }
        A.out_l[i] = a;
        A.out_m[i] = b;
        if constexpr (LOOP == 1 || !TAIL) { p[0] += a * __ldcg(A.v_l + i); p[1] += b * __ldcg(A.v_m + i); }
    }
    if constexpr (LOOP == 1 || !TAIL) {
        block_reduce<2, false>(p);
        if (threadIdx.x == 0) {
            A.part_out[blockIdx.x] = p[0];
            A.part_out[gridDim.x + blockIdx.x] = p[1];
        }
    }
}

}  // namespace hrn

using namespace hrn;

namespace hrn {
// Source illumination of every stored node: the sum over steps, shots and the three
// displacement components of u^2 in the forward history [nstep+1][nstore][S].
template <typename T>
__global__ void k_illumination(int nnode, int nstore, int nstep, int S, const T *__restrict__ hist, double *__restrict__ out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nnode) return;
    double acc = 0.0;
    for (int n = 0; n <= nstep; ++n) {
        const T *h = hist + (size_t(n) * nstore + 3 * size_t(k)) * S;
        for (int i = 0; i < 3 * S; ++i) {
            const double v = double(h[i]);
            acc = fma(v, v, acc);
        }
    }
    out[k] = acc;
}

}  // namespace hrn

extern "C" {

int hrn_vec_dot(hrn_ctx *c, int32_t n, const double *x, const double *y, double *out)
{
    if (!c || !x || !y || !out || n < 0) return HRN_EARG;
    return vec_reduce(c, 0, n, x, y, out);
}

int hrn_vec_norm(hrn_ctx *c, int32_t n, const double *x, int32_t kind, double *out)
{
    if (!c || !x || !out || n < 0 || (kind != 2 && kind != 0)) return c ? set_error(c, HRN_EARG, "norm kind must be 2 or 0 (infinity)") : HRN_EARG;
    return vec_reduce(c, kind == 2 ? 1 : 2, n, x, nullptr, out);
}

int hrn_vec_axpby(hrn_ctx *c, int32_t n, double a, const double *x, double b, const double *y, double *z)
{
    if (!c || !x || !z || n < 0) return HRN_EARG;
    return vec_axpby(c, n, a, x, b, y, z);
}

int hrn_vec_mul(hrn_ctx *c, int32_t n, const double *x, const double *y, double *z)
{
    if (!c || !x || !y || !z || n < 0) return HRN_EARG;
    k_mul<<<grid_for(n), 256, 0, c->stream>>>(n, x, y, z);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    return HRN_OK;
}

int hrn_vec_clip(hrn_ctx *c, int32_t n, double lo, double hi, double *x)
{
    if (!c || !x || n < 0) return HRN_EARG;
    k_clip<<<grid_for(n), 256, 0, c->stream>>>(n, lo, hi, x);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    return HRN_OK;
}

int hrn_vec_gather(hrn_ctx *c, int32_t n, const int32_t *map, const double *x, double *y)
{
    if (!c || !map || !x || !y || n < 0) return HRN_EARG;
    k_gather<<<grid_for(n), 256, 0, c->stream>>>(n, map, x, y);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    return HRN_OK;
}

int hrn_regularization_tv(hrn_ctx *c, const double *d_lambda, const double *d_mu, double *d_reg_lambda, double *d_reg_mu,
                          double *cost_lambda, double *cost_mu)
{
    if (!c || !d_lambda || !d_mu || !d_reg_lambda || !d_reg_mu || !cost_lambda || !cost_mu) return HRN_EARG;
    if (!c->have_mesh) return set_error(c, HRN_ESTATE, "no mesh: call hrn_set_mesh first");
    return regularization_tv(c, d_lambda, d_mu, d_reg_lambda, d_reg_mu, cost_lambda, cost_mu);
}

int hrn_illumination(hrn_ctx *c, double *d_out)
{
    if (!c || !d_out) return HRN_EARG;
    if (!c->have_forward) return set_error(c, HRN_ESTATE, "no forward history: call hrn_forward first");
    if (c->ckpt > 0) return set_error(c, HRN_ESTATE, "illumination needs the whole forward history (checkpointing is on)");
    if (c->nstore % 3 != 0) return set_error(c, HRN_EARG, "history rows must come in x, y, z triples");
    cudaSetDevice(c->device);
    const int nnode = c->nstore / 3, th = 128;
    if (c->precision == HRN_FP64)
        k_illumination<double><<<(nnode + th - 1) / th, th, 0, c->stream>>>(nnode, c->nstore, c->nstep, c->nshot,
                                                                          c->d_hist.as<double>(), d_out);
    else
        k_illumination<float><<<(nnode + th - 1) / th, th, 0, c->stream>>>(nnode, c->nstore, c->nstep, c->nshot,
                                                                         c->d_hist.as<float>(), d_out);
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    return HRN_OK;
}

int hrn_pseudo_hessian(hrn_ctx *c, double *d_h_lambda, double *d_h_mu)
{
    if (!c || !d_h_lambda || !d_h_mu) return HRN_EARG;
    if (!c->have_forward) return set_error(c, HRN_ESTATE, "no forward history: call hrn_forward first");
    if (c->ckpt > 0) return set_error(c, HRN_ESTATE, "the pseudo-Hessian needs the whole forward history (checkpointing is on)");
    if (!c->have_mesh) return set_error(c, HRN_ESTATE, "no mesh: call hrn_set_mesh first");
    cudaSetDevice(c->device);
    return run_pseudo_hessian(c, d_h_lambda, d_h_mu);
}

int hrn_gradient_mass(hrn_ctx *c, double *d_mg)
{
    if (!c || !d_mg) return HRN_EARG;
    if (!c->have_mesh) return set_error(c, HRN_ESTATE, "no mesh: call hrn_set_mesh first");
    return gradient_mass(c, d_mg);
}

// Coupled L-BFGS memory (S4/LBFGS_Coupled.F90; M_LBFGS in S4/Adjustments.F90:180).
int hrn_lbfgs_setup(hrn_ctx *c, int32_t m, const double *d_restriction)
{
    if (!c || m < 1 || !d_restriction) return HRN_EARG;
    if (!c->have_mesh) return set_error(c, HRN_ESTATE, "no mesh: call hrn_set_mesh first");
    const size_t nj = size_t(c->nj), bytes = ((4 * size_t(m) + 2) * nj + 2 * size_t(m) + 1 + 2 * kDirSums * kDirBlocks) * 8;
    HRN_CUDA(c, c->d_lbfgs.alloc(bytes));
    HRN_CUDA(c, cudaMemsetAsync(c->d_lbfgs.p, 0, bytes, c->stream));
    HRN_CUDA(c, c->d_restrict.alloc(nj * 8));
    HRN_CUDA(c, cudaMemcpyAsync(c->d_restrict.p, d_restriction, nj * 8, cudaMemcpyDeviceToDevice, c->stream));
    c->lbfgs_m = m;
    return HRN_OK;
}

// Search direction p = -H g of the coupled L-BFGS two-loop recursion
// (S4/LBFGS_Coupled.F90:4-218); every vector is a device array [nj].
int hrn_lbfgs_direction(hrn_ctx *c, int32_t iter, int32_t iter_begin, const double *g_l, const double *g_m,
                        const double *g_l_pre, const double *g_m_pre, const double *lam, const double *mu,
                        const double *lam_pre, const double *mu_pre, double *p_l, double *p_m, double *rho_out)
{
    if (!c || !g_l || !g_m || !p_l || !p_m) return HRN_EARG;
    if (c->lbfgs_m < 1) return set_error(c, HRN_ESTATE, "call hrn_lbfgs_setup first");
    if (iter < iter_begin) return set_error(c, HRN_EARG, "iter lies before iter_begin");   // no such pair
    const int n = c->nj, M = c->lbfgs_m;
    if (iter == iter_begin) {   // p = -g
        if (int rc = vec_axpby(c, n, -1.0, g_l, 0.0, nullptr, p_l)) return rc;
        if (int rc = vec_axpby(c, n, -1.0, g_m, 0.0, nullptr, p_m)) return rc;
        if (rho_out) *rho_out = 0.0;
        return HRN_OK;
    }
    if (!g_l_pre || !g_m_pre || !lam || !mu || !lam_pre || !mu_pre) return HRN_EARG;
    const int k = iter - iter_begin;
    double *base = c->d_lbfgs.as<double>();
    auto Ys_l = [&](int i) { return base + (size_t(0) * M + i) * n; };
    auto Ys_m = [&](int i) { return base + (size_t(1) * M + i) * n; };
    auto Ss_l = [&](int i) { return base + (size_t(2) * M + i) * n; };
    auto Ss_m = [&](int i) { return base + (size_t(3) * M + i) * n; };
    double *q_l = base + 4 * size_t(M) * n, *q_m = q_l + n, *rho = q_m + n, *alpha = rho + M, *h0 = alpha + M;
    double *part[2] = {h0 + 1, h0 + 1 + kDirSums * kDirBlocks};
    if (int rc = red_space(c)) return rc;
    std::vector<int> seq;
    int n_use;
    if (k > 0 && k <= M) {
        n_use = k;
        for (int i = k; i >= 1; --i) seq.push_back(i);
    } else {
        n_use = M;
        const int end = k % M;
        for (int i = end; i >= 1; --i) seq.push_back(i);
        int j = 0;
        while (int(seq.size()) < M) seq.push_back(M - j++);
    }
    const int n_store = (k % M) != 0 ? (k % M) : M;
    const int nb = std::min(std::max((n + kDirThreads - 1) / kDirThreads, 1), kDirBlocks), st = n_store - 1;
    k_dir_pair<<<nb, kDirThreads, 0, c->stream>>>(n, g_l, g_m, g_l_pre, g_m_pre, lam, mu, lam_pre, mu_pre, c->d_restrict.as<double>(),
                                                  Ys_l(st), Ys_m(st), Ss_l(st), Ss_m(st), part[0]);
    int at = 0;
    auto start = [&](auto kern, int i, DirArgs A) {
        A.n = n;
        A.part_in = part[at];
        A.part_out = part[at ^ 1];
        A.rho = rho + i;
        A.alpha = alpha + i;
        A.h0 = h0;
        A.rho_out = c->h_red.as<double>();
        chain_start(kern, nb, kDirThreads, 0, c->stream, true, A);
        at ^= 1;
    };
    for (int iv = 0; iv < n_use; ++iv) {   // loop 1; seq starts with the pair just stored
        const int i = seq[iv] - 1;
        const bool first = iv == 0, tail = iv == n_use - 1;
        DirArgs A = {};
        A.q_l = first ? g_l : q_l; A.q_m = first ? g_m : q_m;
        A.out_l = q_l; A.out_m = q_m;
        A.u_l = Ys_l(i); A.u_m = Ys_m(i);
        A.v_l = tail ? Ys_l(i) : Ss_l(seq[iv + 1] - 1);   // loop 2 begins with the pair that ends loop 1
        A.v_m = tail ? Ys_m(i) : Ss_m(seq[iv + 1] - 1);
        if (first && tail) start(k_dir_step<1, true, true>, i, A);
        else if (first) start(k_dir_step<1, true, false>, i, A);
        else if (tail) start(k_dir_step<1, false, true>, i, A);
        else start(k_dir_step<1, false, false>, i, A);
    }
    for (int iv = n_use - 1; iv >= 0; --iv) {   // loop 2
        const int i = seq[iv] - 1;
        DirArgs A = {};
        A.q_l = q_l; A.q_m = q_m;
        A.out_l = iv == 0 ? p_l : q_l; A.out_m = iv == 0 ? p_m : q_m;
        A.u_l = Ss_l(i); A.u_m = Ss_m(i);
        if (iv > 0) {
            A.v_l = Ys_l(seq[iv - 1] - 1);
            A.v_m = Ys_m(seq[iv - 1] - 1);
            start(k_dir_step<2, false, false>, i, A);
        } else start(k_dir_step<2, false, true>, i, A);
    }
    c->launches += 1 + 2 * n_use;
    HRN_CUDA(c, cudaGetLastError());
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));   // the inputs are free when the call returns
    if (rho_out) *rho_out = *c->h_red.as<volatile double>();
    return HRN_OK;
}

}  // extern "C"
