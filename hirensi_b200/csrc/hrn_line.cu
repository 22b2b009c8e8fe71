// hrn_line.cu -- tables of the line-operator stage (hrn_line.cuh): the nodal
// derivative operators D_x, D_y, D_z of the PML and their transposes, the PML
// coefficients of every node, and the regular-domain element tables.  All of
// them depend on the mesh alone, so they are built once per mesh.
#include <cuda_runtime.h>
#include <stdint.h>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>

#include "hrn_internal.h"

namespace hrn {

constexpr int kLineNb = 32;        // most nodes that share a grid line through one node (13 on structured meshes)
constexpr int kLineBuildThreads = 32;
// Entries below this share of their node's largest one are rounding residue of opposite
// contributions (the one-sided derivatives at a node between two equal elements).
constexpr double kLineDrop = 16 * 2.2204460492503131e-16;
// PML weights that differ by less along a line are the same value with rounding.
constexpr double kWeightTol = 1e-13;

__device__ __forceinline__ double gll_d(int a, int b)   // l_b'(xi_a)
{
    return a == 0 ? (b == 0 ? -1.5 : (b == 1 ? 2.0 : -0.5))
                  : (a == 1 ? (b == 0 ? -0.5 : (b == 1 ? 0.0 : 0.5)) : (b == 0 ? 0.5 : (b == 1 ? -2.0 : 1.5)));
}

// Entries of row r of D_k (TR = 0: PML node J, columns the nodes on its lines) or of
// D_k^T (TR = 1: displacement node I, columns the PML nodes J whose lines pass it), at
// most w a direction (TR = 0) or a row (TR = 1).  idx == null: the most a direction or a
// row has, into *most; else write them, entry u of a direction at
// idx[(k w + u) nrow + r], of a row at idx[u nrow + r], divided by fj = F j0 of node J.
template <typename T, int TR>
__global__ void __launch_bounds__(kLineBuildThreads)
k_line_entries(int nrow, const int32_t *__restrict__ nodes, const int32_t *__restrict__ nptr, const uint32_t *__restrict__ nslot,
               int nel_pml, const int32_t *__restrict__ el_node, const double *__restrict__ geom,
               const int32_t *__restrict__ target, int ntarget, const double *__restrict__ pmlw, const double *__restrict__ fj, int w,
               int *most, int32_t *__restrict__ idx, T *__restrict__ cf, int *__restrict__ bad)
{
    __shared__ int32_t s_nb[kLineNb][kLineBuildThreads];
    __shared__ double s_cf[3][kLineNb][kLineBuildThreads];
    const int r = blockIdx.x * kLineBuildThreads + threadIdx.x, th = threadIdx.x;
    if (r >= nrow) return;
    const int node = nodes[r];
    int n = 0;
    for (int s = nptr[node]; s < nptr[node + 1]; ++s) {
        const uint32_t sl = nslot[s] & 0x7fffffffu;
        const int p = int(sl / 27), q = int(sl % 27);
        if (p >= nel_pml) continue;   // regular-domain elements follow the PML's
        const int qm[3] = {q % 3, (q / 3) % 3, q / 9};
        const int str[3] = {1, 3, 9};
        for (int m = 0; m < 3; ++m)
            for (int t = 0; t < 3; ++t) {
                const int o = q + (t - qm[m]) * str[m];
                const int nb = el_node[size_t(p) * 27 + o];
                // the derivative at point J = q (TR 0) or J = o (TR 1) of the node at the other
                const double *g = geom + (size_t(p) * 27 + (TR ? o : q)) * 10;
                const double d = g[9] * (TR ? gll_d(t, qm[m]) : gll_d(qm[m], t));
                int k = 0;
                while (k < n && s_nb[k][th] != nb) ++k;
                if (k == n) {
                    if (n == kLineNb) { atomicExch(bad, 1); return; }
                    s_nb[n][th] = nb;
                    for (int x = 0; x < 3; ++x) s_cf[x][n][th] = 0.0;
                    ++n;
                }
                for (int x = 0; x < 3; ++x) s_cf[x][k][th] += d * g[3 * m + x];
            }
    }
    double top = 0.0;
    for (int k = 0; k < n; ++k)
        for (int x = 0; x < 3; ++x) top = fmax(top, fabs(s_cf[x][k][th]));
    int at = 0;
    auto raise = [&]() {   // most threads find their count there
        if (at > *static_cast<volatile int *>(most)) atomicMax(most, at);
    };
    for (int x = 0; x < 3; ++x) {
        if (!TR) at = 0;
        for (int k = 0; k < n; ++k) {
            const int nb = s_nb[k][th], to = target[nb];
            if (to < 0 || !(fabs(s_cf[x][k][th]) > kLineDrop * top)) continue;
            if (idx) {
                const size_t o = (size_t(TR ? 0 : x) * w + at) * nrow + r;
                idx[o] = TR ? 3 * ntarget * x + to : to;
                cf[o] = T(s_cf[x][k][th] / fj[TR ? to : r]);
                // the weights of direction x have to be the same at both ends of the entry
                for (int t = 0; t < 3; ++t) {
                    const double wn = pmlw[size_t(node) * 12 + 3 * t + x], wb = pmlw[size_t(nb) * 12 + 3 * t + x];
                    if (!(fabs(wn - wb) <= kWeightTol * fabs(wn))) atomicExch(bad, 2);
                }
            }
            ++at;
        }
        if (!idx && !TR) raise();
    }
    if (!idx && TR) raise();
}

// Coefficient planes of the PML nodes' stress rows (disp = 0) or of the displacement
// nodes (disp = 1), summed over a node's PML elements; eq: first equation of its rows.
template <typename T>
__global__ void k_line_coef(int n, int disp, const int32_t *__restrict__ ids, const int32_t *__restrict__ eqs,
                            const int32_t *__restrict__ nptr, const uint32_t *__restrict__ nslot, int nel_pml,
                            const double *__restrict__ geom, const double *__restrict__ rho, const double *__restrict__ pmlw,
                            const double *__restrict__ im, double j0, T *__restrict__ out)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int node = ids[r];
    double F = 0.0;
    for (int s = nptr[node]; s < nptr[node + 1]; ++s) {
        const uint32_t sl = nslot[s] & 0x7fffffffu;
        const int p = int(sl / 27);
        if (p >= nel_pml) continue;
        const double f0 = geom[size_t(sl) * 10 + 9];
        F += disp ? rho[p] * f0 : f0;
    }
    const double *w = pmlw + size_t(node) * 12;
    auto put = [&](int i, double v) { out[size_t(i) * n + r] = T(v); };
    const int eq = eqs[r];
    const double fj = disp ? 1.0 : F * j0;
    for (int k = 0; k < 9; ++k) put(k, fj * w[k]);
    for (int t = 0; t < 3; ++t) put(9 + t, -im[eq] * F * w[9 + t]);
    put(12, disp ? 0.0 : -im[eq] * fj);
    put(13, disp ? 0.0 : -im[eq + 3] * fj);
    put(14, (w[6] != 0.0 || w[7] != 0.0 || w[8] != 0.0 || F * w[11] != 0.0) ? 1.0 : 0.0);
}

__global__ void k_line_uim(int n, const int4 *__restrict__ unode, const double *__restrict__ im, double *__restrict__ out)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) out[r] = -im[unode[r].x];
}

// F j0 of the PML nodes: the sum of w detJ over a node's PML elements times j0.
__global__ void k_line_fj(int n, const int32_t *__restrict__ ids, const int32_t *__restrict__ nptr, const uint32_t *__restrict__ nslot,
                          int nel_pml, const double *__restrict__ geom, double j0, double *__restrict__ out)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double F = 0.0;
    for (int s = nptr[ids[r]]; s < nptr[ids[r] + 1]; ++s) {
        const uint32_t sl = nslot[s] & 0x7fffffffu;
        if (int(sl / 27) < nel_pml) F += geom[size_t(sl) * 10 + 9];
    }
    out[r] = F * j0;
}

// State rows of a list of equations (out may be null), and whether one is a stress row.
__global__ void k_line_rows(int n, int first_stress, const int32_t *__restrict__ row, const int32_t *__restrict__ eq,
                            int32_t *__restrict__ out, int *__restrict__ stress)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = row[eq[i]];
    if (out) out[i] = r;
    if (r >= first_stress) atomicExch(stress, 1);
}

__global__ void k_line_rgeo(int64_t n, int box, const double *__restrict__ geom, double *__restrict__ out)
{
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= n) return;
    if (box) {
        const double *c = geom + (size_t(t / 4) * 27 + 13) * 10;   // the centre point, weight 64/27
        const int k = int(t % 4);
        out[t] = k == 0 ? c[4] / c[0] : (k == 1 ? c[8] / c[0] : (k == 2 ? c[9] / (64.0 / 27.0) * c[0] * c[0] : 0.0));
    } else {
        out[t] = geom[t];
    }
}

// Entry planes of D (TR = 0) or D^T (TR = 1): *w entries a direction or a row.
template <typename T, int TR>
static int build_entries(hrn_ctx *c, int nrow, const DevBuf &nodes, const DevBuf &target, const DevBuf &fj, int *w, DevBuf &idx, DevBuf &cf, DevBuf &bad)
{
    *w = 0;
    if (nrow == 0) return 0;
    const size_t nc = size_t(nrow) * (TR ? 1 : 3);
    int *most = bad.as<int>() + 1;
    HRN_CUDA(c, cudaMemsetAsync(most, 0, 4, c->stream));
    const int nb = (nrow + kLineBuildThreads - 1) / kLineBuildThreads;
    auto launch = [&](int32_t *out) {
        k_line_entries<T, TR><<<nb, kLineBuildThreads, 0, c->stream>>>(
            nrow, nodes.as<int32_t>(), c->d_nslot_ptr.as<int32_t>(), c->d_nslot.as<uint32_t>(), c->nel_pml_e,
            c->d_el_node.as<int32_t>(), c->d_el_geom.as<double>(), target.as<int32_t>(), c->line_npn, c->d_pmlw.as<double>(), fj.as<double>(), *w,
            most, out, cf.as<T>(), bad.as<int>());
        ++c->launches;
        return cudaGetLastError();
    };
    HRN_CUDA(c, launch(nullptr));
    HRN_CUDA(c, cudaMemcpyAsync(w, most, 4, cudaMemcpyDeviceToHost, c->stream));
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));
    *w = std::max(*w, 1);
    const size_t n = nc * size_t(*w);
    HRN_CUDA(c, idx.alloc(n * 4));
    HRN_CUDA(c, cf.alloc(n * sizeof(T)));
    HRN_CUDA(c, cudaMemsetAsync(idx.p, 0xff, n * 4, c->stream));   // -1: no entry
    HRN_CUDA(c, cudaMemsetAsync(cf.p, 0, n * sizeof(T), c->stream));
    HRN_CUDA(c, launch(idx.as<int32_t>()));
    return 0;
}

// What the numbering of the nodes says, and the place of every node among those that the
// tables list: flag [3][nj + 1] is 1 where a node has a record of P, a free displacement in
// the PML, one outside of it.
constexpr int kLineDispRow = 1, kLineStressRow = 2, kLineStressOut = 4, kLineStressFixed = 8;

__global__ void k_line_nodes(int nj, const int32_t *__restrict__ id, const int32_t *__restrict__ nptr, const uint32_t *__restrict__ nslot,
                             int nel_pml, int32_t *__restrict__ flag, int32_t *__restrict__ nrd, int *__restrict__ info)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j > nj) return;
    int32_t in_pml = 0, rd = 0, u = 0, why = 0;
    if (j < nj) {
        for (int s = nptr[j]; s < nptr[j + 1]; ++s) {
            if (int((nslot[s] & 0x7fffffffu) / 27) < nel_pml) in_pml = 1;
            else ++rd;
        }
        const int32_t *e = id + size_t(j) * 9;
        for (int d = 1; d < 3; ++d)
            if (e[d] != (e[0] < 0 ? -1 : e[0] + d)) why |= kLineDispRow;
        for (int d = 1; d < 6; ++d)
            if (e[3 + d] != (e[3] < 0 ? -1 : e[3] + d)) why |= kLineStressRow;
        if (!in_pml && e[3] >= 0) why |= kLineStressOut;
        if (in_pml && e[3] < 0) why |= kLineStressFixed;
        u = e[0] >= 0;
        nrd[j] = rd;
        if (why) atomicOr(info, why);
        if (u) atomicMax(info + 1, rd);
    }
    const size_t n = size_t(nj) + 1;   // the last entry is 0: its sum is the total
    flag[j] = in_pml;
    flag[n + j] = u && in_pml;
    flag[2 * n + j] = u && !in_pml;
}

// The lists, from the sums `at` of those flags (at[..][j + 1] > at[..][j] where it is 1).
// Rows of the state: displacements [3][nun], those of the PML first, then stresses [6][npn].
__global__ void k_line_lists(int nj, int npn, int nup, int nun, const int32_t *__restrict__ id, const int32_t *__restrict__ at,
                             const int32_t *__restrict__ nrd, int2 *__restrict__ pnode, int4 *__restrict__ unode,
                             int32_t *__restrict__ pn_id, int32_t *__restrict__ pn_eq, int32_t *__restrict__ un_id,
                             int32_t *__restrict__ un_eq, int32_t *__restrict__ pidx, int32_t *__restrict__ zidx,
                             int32_t *__restrict__ unidx, int32_t *__restrict__ row)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nj) return;
    const size_t n = size_t(nj) + 1;
    const int32_t u0 = id[size_t(j) * 9], s0 = id[size_t(j) * 9 + 3];
    const int32_t p = at[j + 1] > at[j] ? at[j] : -1;
    const bool up = at[n + j + 1] > at[n + j], ur = at[2 * n + j + 1] > at[2 * n + j];
    const int32_t u = up ? at[n + j] : (ur ? nup + at[2 * n + j] : -1);
    pidx[j] = p;
    zidx[j] = u0 < 0 ? -1 : p;   // records of Z: PML nodes whose displacements are free
    unidx[j] = u;
    if (p >= 0) {
        pnode[p] = make_int2(j, s0);
        pn_id[p] = j;
        pn_eq[p] = s0;
        for (int d = 0; d < 6; ++d) row[s0 + d] = 3 * nun + d * npn + p;
    }
    if (u >= 0) {
        unode[u] = make_int4(u0, p, nrd[j], 0);
        un_id[u] = j;
        un_eq[u] = u0;
        for (int d = 0; d < 3; ++d) row[u0 + d] = d * nun + u;
    }
}

// Regular-domain contributions of every displacement node, in ascending element order.
__global__ void k_line_ridx(int nun, int nrd, int nel_pml, const int32_t *__restrict__ un_id, const int32_t *__restrict__ nptr,
                            const uint32_t *__restrict__ nslot, int32_t *__restrict__ ridx)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nun) return;
    int k = 0;
    for (int s = nptr[un_id[u]]; s < nptr[un_id[u] + 1]; ++s) {
        const uint32_t sl = nslot[s] & 0x7fffffffu;
        const int p = int(sl / 27), q = int(sl % 27);
        if (p >= nel_pml) ridx[size_t(k++) * nun + u] = 3 * nrd * q + (p - nel_pml);
    }
}

// Nodes of the regular-domain elements' points, by element and by point.
__global__ void k_line_points(int nrd, const int32_t *__restrict__ el_node, const int32_t *__restrict__ unidx, int2 *__restrict__ rpt,
                              int32_t *__restrict__ runode)
{
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= int64_t(nrd) * 27) return;
    const int e = int(t / 27), q = int(t % 27), node = el_node[t], u = unidx[node];
    rpt[t] = make_int2(node, u);
    runode[size_t(q) * nrd + e] = u;
}

// The tables are made on the device, from the element and node lists of elem_prepare: host
// loops over the nodes and element points took 190 ms of the first solve on a mesh of 7.4
// million equations, more than the timing of the element variants that they spare (first
// forward of one FP32 shot, matrix-free, ten steps: 206 ms with those, 340 with the loops, 175
// here; 309 thousand equations 8.3, 11.1 and 9.2).
template <typename T>
static int line_tables(hrn_ctx *c)
{
    const int nj = c->nj, nrd = c->nel_rd_e;
    c->line_ok = -1;
    auto no = [&](const char *why) { c->line_why = why; return 0; };
    if (c->neq >= (1 << 29)) return no("more than 2^29 equations");   // 32-bit offsets into [neq][8 shots]
    DevBuf d_flag, d_nrd, d_info, d_pn, d_pe, d_un, d_ue, d_zi, d_pi, d_ui, d_fj, bad;
    const size_t n1 = size_t(nj) + 1;
    HRN_CUDA(c, d_flag.alloc(3 * n1 * 4));
    HRN_CUDA(c, d_nrd.alloc(size_t(nj) * 4));
    HRN_CUDA(c, d_info.alloc(8));
    HRN_CUDA(c, cudaMemsetAsync(d_info.p, 0, 8, c->stream));
    int32_t *flag = d_flag.as<int32_t>();
    k_line_nodes<<<(nj + 256) / 256, 256, 0, c->stream>>>(nj, c->d_id.as<int32_t>(), c->d_nslot_ptr.as<int32_t>(),
                                                          c->d_nslot.as<uint32_t>(), c->nel_pml_e, flag, d_nrd.as<int32_t>(), d_info.as<int>());
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    int info[2], total[3];
    DevBuf d_tmp;   // of the scans, which throw nothing
    size_t tmp = 0;
    HRN_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tmp, flag, flag, int(n1), c->stream));
    HRN_CUDA(c, d_tmp.alloc(std::max<size_t>(tmp, 16)));
    for (int k = 0; k < 3; ++k) {
        HRN_CUDA(c, cub::DeviceScan::ExclusiveSum(d_tmp.p, tmp, flag + k * n1, flag + k * n1, int(n1), c->stream));
        HRN_CUDA(c, cudaMemcpyAsync(&total[k], flag + k * n1 + nj, 4, cudaMemcpyDeviceToHost, c->stream));
    }
    HRN_CUDA(c, cudaMemcpyAsync(info, d_info.p, 8, cudaMemcpyDeviceToHost, c->stream));
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));
    if (info[0] & kLineDispRow) return no("a node's displacement equations are not numbered in a row");
    if (info[0] & kLineStressRow) return no("a node's stress equations are not numbered in a row");
    if (info[0] & kLineStressOut) return no("a stress unknown lies outside the PML");
    if (info[0] & kLineStressFixed) return no("the stresses of a PML node are constrained");
    const int npn = total[0], nup = total[1], nun = total[1] + total[2], most = info[1];
    if (int64_t(3) * nun + int64_t(6) * npn != c->neq) return no("an equation belongs to no node or to several");
    if (most > kLineNb) return no("more than 32 elements share a node");
    if (nun == 0) return no("no displacement is free");
    c->line_npn = npn;
    c->line_nup = nup;
    c->line_nun = nun;
    auto room = [&](DevBuf &b, size_t bytes) { return b.alloc(std::max<size_t>(bytes, 16)); };
    HRN_CUDA(c, room(c->d_line_pnode, size_t(npn) * 8));
    HRN_CUDA(c, room(c->d_line_unode, size_t(nun) * 16));
    HRN_CUDA(c, room(c->d_line_row, size_t(c->neq) * 4));
    HRN_CUDA(c, room(d_pn, size_t(npn) * 4));
    HRN_CUDA(c, room(d_pe, size_t(npn) * 4));
    HRN_CUDA(c, room(d_un, size_t(nun) * 4));
    HRN_CUDA(c, room(d_ue, size_t(nun) * 4));
    HRN_CUDA(c, room(d_zi, size_t(nj) * 4));
    HRN_CUDA(c, room(d_pi, size_t(nj) * 4));
    HRN_CUDA(c, room(d_ui, size_t(nj) * 4));
    k_line_lists<<<(nj + 255) / 256, 256, 0, c->stream>>>(
        nj, npn, nup, nun, c->d_id.as<int32_t>(), flag, d_nrd.as<int32_t>(), c->d_line_pnode.as<int2>(), c->d_line_unode.as<int4>(),
        d_pn.as<int32_t>(), d_pe.as<int32_t>(), d_un.as<int32_t>(), d_ue.as<int32_t>(), d_pi.as<int32_t>(), d_zi.as<int32_t>(),
        d_ui.as<int32_t>(), c->d_line_row.as<int32_t>());
    ++c->launches;
    HRN_CUDA(c, room(c->d_line_ridx, size_t(most) * nun * 4));
    HRN_CUDA(c, cudaMemsetAsync(c->d_line_ridx.p, 0xff, c->d_line_ridx.bytes, c->stream));   // -1: no entry
    k_line_ridx<<<(nun + 255) / 256, 256, 0, c->stream>>>(nun, nrd, c->nel_pml_e, d_un.as<int32_t>(), c->d_nslot_ptr.as<int32_t>(),
                                                          c->d_nslot.as<uint32_t>(), c->d_line_ridx.as<int32_t>());
    ++c->launches;
    HRN_CUDA(c, room(c->d_line_rpt, size_t(nrd) * 27 * 8));
    HRN_CUDA(c, room(c->d_line_runode, size_t(nrd) * 27 * 4));
    if (nrd > 0) {
        k_line_points<<<unsigned((int64_t(nrd) * 27 + 255) / 256), 256, 0, c->stream>>>(
            nrd, c->d_el_node.as<int32_t>() + size_t(c->nel_pml_e) * 27, d_ui.as<int32_t>(), c->d_line_rpt.as<int2>(), c->d_line_runode.as<int32_t>());
        ++c->launches;
    }
    HRN_CUDA(c, cudaGetLastError());
    HRN_CUDA(c, bad.alloc(8));
    HRN_CUDA(c, cudaMemsetAsync(bad.p, 0, 8, c->stream));
    double j0 = 1.0;   // an inverse length of the PML's elements
    if (npn > 0) {
        double g[9];
        HRN_CUDA(c, cudaMemcpyAsync(g, c->d_el_geom.p, sizeof(g), cudaMemcpyDeviceToHost, c->stream));
        HRN_CUDA(c, cudaStreamSynchronize(c->stream));
        for (double v : g)
            if (v != 0.0) { j0 = std::fabs(v); break; }
        HRN_CUDA(c, d_fj.alloc(size_t(npn) * 8));
        k_line_fj<<<(npn + 127) / 128, 128, 0, c->stream>>>(npn, d_pn.as<int32_t>(), c->d_nslot_ptr.as<int32_t>(), c->d_nslot.as<uint32_t>(),
                                                            c->nel_pml_e, c->d_el_geom.as<double>(), j0, d_fj.as<double>());
        ++c->launches;
        HRN_CUDA(c, cudaGetLastError());
    }
    if (int rc = build_entries<T, 0>(c, npn, d_pn, d_zi, d_fj, &c->line_wd, c->d_line_didx, c->d_line_dcf, bad)) return rc;
    if (int rc = build_entries<T, 1>(c, c->line_nup, d_un, d_pi, d_fj, &c->line_wt, c->d_line_tidx, c->d_line_tcf, bad)) return rc;
    auto coef = [&](int n, int disp, const DevBuf &ids, const DevBuf &eqs, DevBuf &out) -> int {
        HRN_CUDA(c, out.alloc(size_t(std::max(n, 1)) * kLineCoef * sizeof(T)));
        if (n == 0) return 0;
        k_line_coef<T><<<(n + 127) / 128, 128, 0, c->stream>>>(
            n, disp, ids.as<int32_t>(), eqs.as<int32_t>(), c->d_nslot_ptr.as<int32_t>(), c->d_nslot.as<uint32_t>(), c->nel_pml_e,
            c->d_el_geom.as<double>(), c->d_el_rho.as<double>(), c->d_pmlw.as<double>(), c->d_im.as<double>(), j0, out.as<T>());
        ++c->launches;
        HRN_CUDA(c, cudaGetLastError());
        return 0;
    };
    if (int rc = coef(npn, 0, d_pn, d_pe, c->d_line_pcoef)) return rc;
    if (int rc = coef(c->line_nup, 1, d_un, d_ue, c->d_line_ucoef)) return rc;
    HRN_CUDA(c, c->d_line_uim.alloc(size_t(nun) * 8));
    k_line_uim<<<(nun + 255) / 256, 256, 0, c->stream>>>(nun, c->d_line_unode.as<int4>(), c->d_im.as<double>(), c->d_line_uim.as<double>());
    ++c->launches;
    HRN_CUDA(c, cudaGetLastError());
    const double *rg = c->d_el_geom.as<double>() + size_t(c->nel_pml_e) * 270;
    int unfit = 0;
    HRN_CUDA(c, cudaMemcpyAsync(&unfit, bad.p, 4, cudaMemcpyDeviceToHost, c->stream));
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));
    if (unfit == 1) return no("more than 32 nodes lie on the grid lines through one");
    if (unfit) return no("the PML's weights across a grid line vary along it (its elements are not aligned with the axes)");
    const int box = c->rd_box ? 1 : 0;
    const int64_t ng = int64_t(c->nel_rd_e) * (box ? 4 : 270);
    HRN_CUDA(c, c->d_line_rgeo.alloc(std::max<size_t>(size_t(ng), 1) * 8));
    if (ng > 0) {
        k_line_rgeo<<<unsigned((ng + 255) / 256), 256, 0, c->stream>>>(ng, box, rg, c->d_line_rgeo.as<double>());
        ++c->launches;
        HRN_CUDA(c, cudaGetLastError());
    }
    HRN_CUDA(c, cudaStreamSynchronize(c->stream));
    c->line_ok = 1;
    return 0;
}

// Tables of the current mesh; c->line_ok says whether the mesh suits the line operator.
static int line_prepare(hrn_ctx *c)
{
    if (int rc = elem_prepare(c)) return rc;
    if (c->have_line) return 0;
    const int rc = c->precision == HRN_FP64 ? line_tables<double>(c) : line_tables<float>(c);
    if (rc) return rc;
    c->have_line = true;
    return 0;
}

// Whether the regular-domain elements take the kernel that keeps an element in one
// thread's registers: FP32 (in FP64 an element does not fit) boxes, and enough of them to
// hide its longer chain and the extra launch.  Elements x shots, us a stage with the
// thread-per-point blocks / with the register kernel: 8 thousand 17.2 / 23.1, 16 thousand
// 29.5 / 34.4, 28 thousand 40.0 / 41.4, 61 thousand 151 / 125, 256 thousand 253 / 197.
constexpr int64_t kLineRegElements = 50000;
bool line_reg_elements(const hrn_ctx *c)
{
    return c->precision == HRN_FP32 && c->rd_box && int64_t(c->nel_rd_e) * c->nshot >= kLineRegElements;
}

// Tables and buffers for the current shots; *ok = 0 when the mesh needs another variant.
int line_ready(hrn_ctx *c, int *ok)
{
    *ok = 0;
    if (!c->op_from_mesh) return 0;
    if (int rc = line_prepare(c)) return rc;
    if (c->line_ok != 1) return 0;
    const size_t rec = size_t(c->nshot) * c->elem_bytes();
    const size_t sets = c->ckpt > 0 ? 2 : 1;   // the recomputed forward segments interleave with the adjoint steps
    HRN_CUDA(c, c->d_line_P.alloc(std::max<size_t>(sets * 3 * 9 * c->line_npn * rec, 16)));
    if (line_reg_elements(c)) HRN_CUDA(c, c->d_line_rmat.alloc(size_t(c->nel_rd_e) * 54 * c->elem_bytes()));
    HRN_CUDA(c, c->d_line_rslot.alloc(std::max<size_t>(size_t(c->nel_rd_e) * 81 * rec, 16)));
    if (c->line_epoch != c->epoch) {
        // sources, receivers or history rows on stress equations (none in an ordinary
        // set-up), and the state rows of the history and the receivers
        DevBuf flags;   // sources and receivers, history
        HRN_CUDA(c, flags.alloc(8));
        HRN_CUDA(c, cudaMemsetAsync(flags.p, 0, 8, c->stream));
        auto rows = [&](int n, const DevBuf &eq, DevBuf *out, int which) -> int {
            if (out) HRN_CUDA(c, out->alloc(std::max<size_t>(size_t(n) * 4, 16)));
            if (n == 0) return 0;
            k_line_rows<<<(n + 255) / 256, 256, 0, c->stream>>>(n, 3 * c->line_nun, c->d_line_row.as<int32_t>(), eq.as<int32_t>(),
                                                                out ? out->as<int32_t>() : nullptr, flags.as<int>() + which);
            ++c->launches;
            HRN_CUDA(c, cudaGetLastError());
            return 0;
        };
        if (int rc = rows(c->nslot_f, c->d_fslot_eq, nullptr, 0)) return rc;
        if (int rc = rows(c->nrec3, c->d_eqdis, &c->d_line_rec_row, 0)) return rc;
        if (int rc = rows(c->nstore, c->d_store_eq, &c->d_line_store_row, 1)) return rc;
        int h[2];
        HRN_CUDA(c, cudaMemcpyAsync(h, flags.p, 8, cudaMemcpyDeviceToHost, c->stream));
        HRN_CUDA(c, cudaStreamSynchronize(c->stream));
        c->line_stress_src = h[0];
        c->line_stress_hist = h[1];
        c->line_epoch = c->epoch;
    }
    *ok = 1;
    return 0;
}

int line_stage(hrn_ctx *c, const void *args, int stage, int adj, int variant, int first, bool pdl)
{
    const int sv = 1 << (variant - 96);
    return c->precision == HRN_FP64 ? line_stage_f64(c, args, stage, adj, sv, first, pdl) : line_stage_f32(c, args, stage, adj, sv, first, pdl);
}

}  // namespace hrn
