// hrn_line.cuh -- kernels of the line-operator RK4 stage (variants 96-98): the
// PML operator as three assembled nodal derivatives, the regular domain element
// by element.  Included by one source file per precision.
//
// In the PML the stresses are nodal unknowns, and with the 3-point GLL rule the
// EA blocks of node J only see the displacement gradient at J
// (S4/Element_Matrices_3D.F90:618-882).  The PML weights and the material enter
// there as values of node J, so they factor out of the sum over J's elements:
//     stress rows of J:        sum_t w_k^t(J) (D_k u_t)(J),   (D_k u)(J) = sum_I D_k(J,I) u(I)
//     displacement rows of I:  -sum_k sum_J D_k(J,I) P_k(J),  P_k(J) = sum_t w_k^t(J) (C s_t)_k(J)
// with D_k(J,I) = sum over the PML elements of J of w detJ dN_I/dx_k at J.  D_k
// depends on the mesh alone and holds 2-5 entries per node and direction on
// aligned meshes (the points of one grid line), against about 166 stored entries
// of C, K and G per node.  The weight w_k depends on the coordinates across x_k
// only, which are the same all along the line, so it can be applied at either end:
//     Z_k(I) = sum_t w_k^t(I) u_t(I),   sum_t w_k^t(J) (D_k u_t)(J) = (D_k Z_k)(J).
// Meshes where it is not constant along the lines take another variant.  The
// adjoint exchanges the roles: P takes the weighted stresses without C, and C
// acts on the weighted gradients.
//
// A stage is two launches:
//   k_line_a: every PML node's six stress rows (D Z, EN diagonal, row update) and
//             the P of its next stage inputs; and, in blocks of their own, the
//             regular-domain elements' contributions to their nodes;
//   k_line_b: every node's displacement rows: D^T P, the regular-domain element
//             contributions in ascending element order, the EM diagonal, the row
//             update, and Z (in the PML) or K's input (at regular-domain nodes) of
//             the next stage.
// Rows rebuild their own stage inputs from x and the earlier kb.  All sums run in a
// fixed order.
//
// Layout: state, kb, P and Z are stored by component, [component][node][S], so that one
// thread takes a node's shots through all of its rows and consecutive threads read
// consecutive nodes -- of the node itself and of each of its line neighbours.  The row of
// an equation: line_row[eq]; displacements first ([3][nun]), then stresses ([6][npn]).
// In equation order (nine rows of a node in a run) the same work needed three threads a
// node to read whole lines, an exchange through shared memory, and four times the
// instructions: 20 us a stage for one FP64 shot on the inversion mesh, of which 3 us
// was waiting for memory.
//
// Why this form: the stored operator is bound by the traffic of its row records
// (18.5 gathers of S values per row through L1 and shared memory) and streams 12
// bytes per entry besides; here a node gathers about 21 records of three rows for
// all of its nine rows, and streams as many small entries.  Microseconds a stage
// (forward), best other variant -> here:
//     16 x 16 x 8 + PML 3, FP64, 4 shots   68.6 -> 29.9      FP32, 4 shots   37.0 -> 17.0
//     the same, FP64, 1 shot               30.7 -> 13.1
//     11 x 7 x 5 + PML 2, FP64, 3 shots    19.0 -> 12.3
//     40 x 40 x 20 + PML 3, FP32, 8 shots   372 -> 197
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>
#include <utility>

#include "hrn_internal.h"
#include "hrn_pdl.cuh"
#include "hrn_stage.cuh"

namespace hrn {

// D is stored relative to F(J) j0, F(J) = sum of w detJ over the node's PML elements and j0
// one inverse length of the mesh: small rationals on uniform elements, exact in FP32 too.
// The factors that remain are products formed in FP64 and rounded once, so that no
// rounding of a geometric constant repeats at every node (in FP32 such a constant shifts
// the wave speeds everywhere by the same 1e-8 to 1e-7).
// Planes of a PML node's coefficients:
//   0-8    w_x, w_y, w_z of C, K, G: times F j0 for the stresses (P), as they are for the
//          displacements (Z)
//   9-11   -M^-1 EN (or EM) b, c, d
//   12, 13 -M^-1 F j0 of the normal and the shear rows
//   14     1 if a factor of G is not 0
constexpr int kCoefDiag = 9, kCoefY = 12, kCoefYShear = 13, kCoefG = 14;

template <typename T>
struct LineArgs {
    int npn, nup, nun, nrd;              // PML nodes; displacement nodes in the PML, all; regular-domain elements
    int wd, wt;                          // entries per direction of D, per node of D^T
    const int2 *__restrict__ pnode;      // [npn] node, first stress equation
    const int32_t *__restrict__ didx;    // [3 wd][npn] PML node of the entry, -1 past the last
    const T *__restrict__ dcf;
    const T *__restrict__ pcoef;         // [kLineCoef][npn]
    const int4 *__restrict__ unode;      // [nun] first equation, PML node (-1), regular-domain elements, 0
    const int32_t *__restrict__ tidx;    // [wt][nup] 3 npn * direction + PML node, -1 past the last
    const T *__restrict__ tcf;
    const int32_t *__restrict__ ridx;    // [..][nun] 3 nrd * point + element of the node's elements, ascending
    const T *__restrict__ ucoef;         // [kLineCoef][nup]
    const double *__restrict__ uim;      // [nun] -M^-1
    const int2 *__restrict__ rpt;        // [nrd * 27] node, displacement node (-1: constrained)
    const double *__restrict__ rgeo;     // boxes: [nrd][4] DJI_y / DJI_x, DJI_z / DJI_x, detJ DJI_x^2, 0; else
                                         // [nrd * 27][10] DJI and w*detJ
    const double *__restrict__ lam, *__restrict__ mu;
    const int32_t *__restrict__ runode;  // [27][nrd] displacement node of the element's point (-1: constrained)
    T *rlam, *rmu;                       // [27][nrd] lambda, mu times w detJ DJI_x^2 of the point
    // written by the launches of a loop
    T *x1, *x2, *x3, *k1, *k2, *k3;      // [3][nun][S], then [6][npn][S]
    T *kt;                               // [3][nun][S] K's input at the regular-domain nodes
    T *rslot;                            // [27][3][nrd][S] regular-domain element contributions
    T *P, *Pn, *Z;                       // [3 directions][3 components][npn][S]: P of this and the next stage, Z
    T *hist;                             // [nstore][S] of this step, or null (stage 1)
    const int32_t *__restrict__ slot, *__restrict__ store_pos;   // by equation
    const T *__restrict__ srcv;          // [4][nslot][S]
    int nslot;
    int stress_src, stress_hist;         // a source / a history position lies on a stress row
    T c, D, d6;
};

template <typename T>
__device__ __forceinline__ void gll_drow(int a, T &d0, T &d1, T &d2)
{
    d0 = a == 0 ? T(-1.5) : (a == 1 ? T(-0.5) : T(0.5));
    d1 = a == 0 ? T(2.0) : (a == 1 ? T(0.0) : T(-2.0));
    d2 = a == 0 ? T(-0.5) : (a == 1 ? T(0.5) : T(1.5));
}
template <typename T>
__device__ __forceinline__ void gll_dcol(int b, T &d0, T &d1, T &d2)
{
    d0 = b == 0 ? T(-1.5) : (b == 1 ? T(2.0) : T(-0.5));
    d1 = b == 0 ? T(-0.5) : (b == 1 ? T(0.0) : T(0.5));
    d2 = b == 0 ? T(0.5) : (b == 1 ? T(-2.0) : T(1.5));
}

// Values that earlier launches of the loop wrote (state, kb, Z, P, slots).  Not the
// read-only path: a launch may start before the one that writes them has ended.
template <typename T, int N>
__device__ __forceinline__ void ldw(const T *p, T (&o)[N])
{
    static_assert(N == 1 || N == 2 || N == 4, "1, 2 or 4 shots per thread");
    if constexpr (sizeof(T) == 8) {
        if constexpr (N == 4)
            asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3]) : "l"(p));
        else if constexpr (N == 2)
            asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(o[0]), "=d"(o[1]) : "l"(p));
        else
            asm volatile("ld.global.f64 %0, [%1];" : "=d"(o[0]) : "l"(p));
    } else {
        if constexpr (N == 4)
            asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "l"(p));
        else if constexpr (N == 2)
            asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(o[0]), "=f"(o[1]) : "l"(p));
        else
            asm volatile("ld.global.f32 %0, [%1];" : "=f"(o[0]) : "l"(p));
    }
}

// The same where `in` holds, zeros elsewhere: a predicated load, so that a run of them
// has no branches between.
template <typename T, int N>
__device__ __forceinline__ void ldw_if(bool in, const T *p, T (&o)[N])
{
    const uint32_t f = in;
    if constexpr (sizeof(T) == 8) {
        if constexpr (N == 2)
            asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.f64 %0, 0d0000000000000000;\n mov.f64 %1, 0d0000000000000000;\n"
                         " @p ld.global.v2.f64 {%0,%1}, [%2];\n}" : "=&d"(o[0]), "=&d"(o[1]) : "l"(p), "r"(f));
        else
            asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.f64 %0, 0d0000000000000000;\n @p ld.global.f64 %0, [%1];\n}"
                         : "=&d"(o[0]) : "l"(p), "r"(f));
    } else {
        if constexpr (N == 4)
            asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n"
                         " mov.f32 %2, 0f00000000;\n mov.f32 %3, 0f00000000;\n @p ld.global.v4.f32 {%0,%1,%2,%3}, [%4];\n}"
                         : "=&f"(o[0]), "=&f"(o[1]), "=&f"(o[2]), "=&f"(o[3]) : "l"(p), "r"(f));
        else if constexpr (N == 2)
            asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n"
                         " @p ld.global.v2.f32 {%0,%1}, [%2];\n}" : "=&f"(o[0]), "=&f"(o[1]) : "l"(p), "r"(f));
        else
            asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.f32 %0, 0f00000000;\n @p ld.global.f32 %0, [%1];\n}"
                         : "=&f"(o[0]) : "l"(p), "r"(f));
    }
}

// The earlier values of one row that a stage needs, and what follows from them.
template <typename T, int SV, int stage>
struct RowIn {
    T x1[SV], x2[SV], x3[SV], k1[SV], k2[SV], k3[SV];
    // lean: only km and x2 are wanted (stages 1-3)
    __device__ __forceinline__ void load(const LineArgs<T> &L, uint32_t o, bool want_x1, bool lean = false)
    {
        ldw<T, SV>(L.x2 + o, x2);
        ldw<T, SV>(L.x3 + o, x3);
        ldw_if<T, SV>(want_x1 || stage == 4, L.x1 + o, x1);
        if (stage == 3) ldw_if<T, SV>(!lean, L.k1 + o, k1);
        else if (stage >= 2) ldw<T, SV>(L.k1 + o, k1);
        if (stage >= 3) ldw<T, SV>(L.k2 + o, k2);
        if (stage == 4) ldw<T, SV>(L.k3 + o, k3);
    }
    // the row's stage inputs, with the fused multiply-adds of the other stage kernels
    __device__ __forceinline__ void inputs(const LineArgs<T> &a, T (&m)[SV], T (&t)[SV], T (&h)[SV]) const
    {
#pragma unroll
        for (int v = 0; v < SV; ++v) {
            if (stage == 1) {
                m[v] = x3[v]; t[v] = x2[v]; h[v] = x1[v];
            } else if (stage == 2) {
                m[v] = fmaT(a.c, k1[v], x3[v]); t[v] = fmaT(a.c, x3[v], x2[v]); h[v] = fmaT(a.c, x2[v], x1[v]);
            } else if (stage == 3) {
                m[v] = fmaT(a.c, k2[v], x3[v]);
                t[v] = fmaT(a.c, fmaT(a.c, k1[v], x3[v]), x2[v]);
                h[v] = fmaT(a.c, fmaT(a.c, x3[v], x2[v]), x1[v]);
            } else {
                m[v] = fmaT(a.D, k3[v], x3[v]);
                t[v] = fmaT(a.D, fmaT(a.c, k2[v], x3[v]), x2[v]);
                h[v] = fmaT(a.D, fmaT(a.c, fmaT(a.c, k1[v], x3[v]), x2[v]), x1[v]);
            }
        }
    }
    // kb of the row into its array, or (stage 4) the new state in place; the next stage's inputs
    __device__ __forceinline__ void finish(const LineArgs<T> &a, uint32_t o, const T (&kb)[SV], const T (&m)[SV], const T (&t)[SV],
                                           T (&nm)[SV], T (&nt)[SV], T (&nh)[SV]) const
    {
        if (stage < 4) {
            stv<T, SV>((stage == 1 ? a.k1 : (stage == 2 ? a.k2 : a.k3)) + o, kb);
            const T cc = stage == 3 ? a.D : a.c;
#pragma unroll
            for (int v = 0; v < SV; ++v) {
                nm[v] = fmaT(cc, kb[v], x3[v]);
                nt[v] = fmaT(cc, m[v], x2[v]);
                nh[v] = fmaT(cc, t[v], x1[v]);
            }
        } else {
#pragma unroll
            for (int v = 0; v < SV; ++v) {
                const T km2 = fmaT(a.c, k1[v], x3[v]);
                const T km3 = fmaT(a.c, k2[v], x3[v]);
                const T km4 = fmaT(a.D, k3[v], x3[v]);
                const T kt2 = fmaT(a.c, x3[v], x2[v]);
                const T kt3 = fmaT(a.c, km2, x2[v]);
                const T kt4 = fmaT(a.D, km3, x2[v]);
                const T ht = ((x2[v] + T(2) * kt2) + T(2) * kt3) + kt4;
                const T hm = ((x3[v] + T(2) * km2) + T(2) * km3) + km4;
                const T hb = ((k1[v] + T(2) * k2[v]) + T(2) * k3[v]) + kb[v];
                nh[v] = fmaT(a.d6, ht, x1[v]);
                nt[v] = fmaT(a.d6, hm, x2[v]);
                nm[v] = fmaT(a.d6, hb, x3[v]);
            }
            stv<T, SV>(a.x1 + o, nh);
            stv<T, SV>(a.x2 + o, nt);
            stv<T, SV>(a.x3 + o, nm);
        }
    }
};

template <typename T, int S, int SV, int stage>
__device__ __forceinline__ void add_source(const LineArgs<T> &L, int eq, int s0, T (&kb)[SV])
{
    const int sl = __ldg(L.slot + eq);
    if (sl >= 0) {
        const T *sv = L.srcv + (size_t(stage - 1) * L.nslot + sl) * S + s0;
#pragma unroll
        for (int v = 0; v < SV; ++v) kb[v] = __ldg(sv + v) + kb[v];
    }
}
template <typename T, int S, int SV>
__device__ __forceinline__ void add_history(const LineArgs<T> &L, int eq, int s0, const T (&x2)[SV])
{
    const int pos = __ldg(L.store_pos + eq);
    if (pos >= 0) stv<T, SV>(L.hist + size_t(pos) * S + s0, x2);
}

// Threads of a block: one per node and SV shots, or 27 per regular-domain element and SV
// shots.  Blocks of three to seven warps: with 224 to 256 threads for every shot count fewer
// blocks share an SM and their phases run in step (270 against 250 us, 40 x 40 x 20, FP32).
template <int S, int SV>
constexpr int line_threads()
{
    constexpr int TP = S / SV;
    return TP == 3 ? 96 : TP == 5 ? 160 : (TP == 6 || TP == 7) ? 192 : TP == 8 ? 224 : 128;
}
template <int S, int SV>
constexpr int line_elems() { return line_threads<S, SV>() / (27 * (S / SV)); }
template <int S, int SV>
constexpr int line_nodes() { return line_threads<S, SV>() / (S / SV); }
// Resident blocks the register limits leave: k_line_a needs up to 168 registers a thread
// with 16 bytes of shots and 96 with 8; k_line_b does better with 128 in the first case.
template <typename T, int S, int SV, int B>
constexpr int line_blocks() { return (SV * sizeof(T) > 8 ? (B ? 512 : 384) : 640) / line_threads<S, SV>(); }
template <typename T, int S, int SV, int BOX>
constexpr size_t line_smem() { return size_t(line_elems<S, SV>()) * 27 * (3 + (BOX ? 6 : 9)) * S * sizeof(T); }

// Contributions of a block's regular-domain elements to their nodes: thread (element, point, shots).
template <typename T, int S, int SV, int BOX>
__device__ __forceinline__ void line_rd_elements(const LineArgs<T> &L, const T *ut, int block, T *smem)
{
    constexpr int TP = S / SV, NF = BOX ? 6 : 9, EPB = line_elems<S, SV>();
    const int tid = threadIdx.x;
    const int tp = tid % TP, q = (tid / TP) % 27, el = tid / (27 * TP);
    const int e = block * EPB + el;
    const bool active = el < EPB && e < L.nrd;
    const int s0 = tp * SV;
    // [component][point][S]: the threads of a warp read runs of points, without bank conflicts
    T *U = smem + size_t(el < EPB ? el : 0) * 27 * 3 * S;
    T *F = smem + size_t(EPB) * 27 * 3 * S + size_t(el < EPB ? el : 0) * 27 * NF * S;
    T own[3][SV];
    T lam = T(0), mu = T(0);
    T geo[BOX ? 3 : 9];
    if (active) {
        const int2 pt = __ldg(L.rpt + size_t(e) * 27 + q);
        const double *gp = L.rgeo + (BOX ? size_t(e) * 4 : (size_t(e) * 27 + q) * 10);
        double f;   // w detJ of the point (times DJI_x^2)
        if constexpr (BOX != 0) {
            geo[0] = T(1);
            geo[1] = T(__ldg(gp));
            geo[2] = T(__ldg(gp + 1));
            const double third = 1.0 / 3.0, mid = 4.0 / 3.0;   // GLL weights
            f = __ldg(gp + 2) * (q % 3 == 1 ? mid : third) * (q / 3 % 3 == 1 ? mid : third) * (q / 9 == 1 ? mid : third);
        } else {
#pragma unroll
            for (int k = 0; k < 9; ++k) geo[k] = T(__ldg(gp + k));
            f = __ldg(gp + 9);
        }
        lam = T(f * __ldg(L.lam + pt.x));
        mu = T(f * __ldg(L.mu + pt.x));
        dep_wait();
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (pt.y >= 0) {
                ldw<T, SV>(ut + (size_t(c) * L.nun + pt.y) * S + s0, own[c]);
            } else {
#pragma unroll
                for (int i = 0; i < SV; ++i) own[c][i] = T(0);
            }
            stv<T, SV>(U + (c * 27 + q) * S + s0, own[c]);
        }
    }
    __syncthreads();
    const int qm[3] = {q % 3, (q / 3) % 3, q / 9};
    const int base[3] = {q - qm[0], q - 3 * qm[1], q - 9 * qm[2]};
    constexpr int kStride[3] = {1, 3, 9};
    constexpr int kAt[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};   // xx, yy, zz, xy, xz, yz
    T flux[NF][SV];
    auto lds = [](const T *p, T (&o)[SV]) {
        if constexpr (SV * sizeof(T) == 16 && sizeof(T) == 4) {
            const float4 v = *reinterpret_cast<const float4 *>(p);
            o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
        } else if constexpr (SV * sizeof(T) == 16 && sizeof(T) == 8) {
            const double2 v = *reinterpret_cast<const double2 *>(p);
            o[0] = v.x; o[1] = v.y;
        } else if constexpr (SV * sizeof(T) == 8 && sizeof(T) == 4) {
            const float2 v = *reinterpret_cast<const float2 *>(p);
            o[0] = v.x; o[1] = v.y;
        } else {
#pragma unroll
            for (int i = 0; i < SV; ++i) o[i] = p[i];
        }
    };
    if (active) {
        T gr[3][3][SV];   // d u_c / d xi_m
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            T d0, d1, d2;
            gll_drow<T>(qm[m], d0, d1, d2);
            // the other two points of the line, and their factors
            const int i0 = qm[m] == 0 ? 1 : 0, i1 = qm[m] == 2 ? 1 : 2;
            const T f0 = i0 == 0 ? d0 : d1, f1 = i1 == 2 ? d2 : d1, fo = qm[m] == 0 ? d0 : (qm[m] == 1 ? d1 : d2);
            const T *p0 = U + (base[m] + i0 * kStride[m]) * S + s0, *p1 = U + (base[m] + i1 * kStride[m]) * S + s0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                T a0[SV], a1[SV];
                lds(p0 + c * 27 * S, a0);
                lds(p1 + c * 27 * S, a1);
#pragma unroll
                for (int v = 0; v < SV; ++v) {
                    gr[c][m][v] = fmaT(f1, a1[v], fmaT(f0, a0[v], fo * own[c][v]));
                    if constexpr (BOX != 0) { if (m > 0) gr[c][m][v] *= geo[m]; }
                }
            }
        }
        if constexpr (BOX == 0) {   // physical gradient: sum over xi directions
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int v = 0; v < SV; ++v) {
                    const T x = gr[c][0][v], y = gr[c][1][v], z = gr[c][2][v];
#pragma unroll
                    for (int k = 0; k < 3; ++k) gr[c][k][v] = fmaT(z, geo[6 + k], fmaT(y, geo[3 + k], x * geo[k]));
                }
        }
        const T m2 = T(2) * mu;
        T sig[6][SV];   // stresses times w*detJ
#pragma unroll
        for (int v = 0; v < SV; ++v) {
            const T tr = lam * (gr[0][0][v] + gr[1][1][v] + gr[2][2][v]);
            sig[0][v] = fmaT(m2, gr[0][0][v], tr);
            sig[1][v] = fmaT(m2, gr[1][1][v], tr);
            sig[2][v] = fmaT(m2, gr[2][2][v], tr);
            sig[3][v] = mu * (gr[0][1][v] + gr[1][0][v]);
            sig[4][v] = mu * (gr[0][2][v] + gr[2][0][v]);
            sig[5][v] = mu * (gr[1][2][v] + gr[2][1][v]);
        }
        T *fp = F + q * S + s0;
        if constexpr (BOX != 0) {
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                stv<T, SV>(fp + d * 27 * S, sig[d]);
#pragma unroll
                for (int v = 0; v < SV; ++v) flux[d][v] = sig[d][v];
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int m = 0; m < 3; ++m) {
#pragma unroll
                    for (int v = 0; v < SV; ++v)
                        flux[c * 3 + m][v] = fmaT(geo[3 * m + 2], sig[kAt[c][2]][v], fmaT(geo[3 * m + 1], sig[kAt[c][1]][v], geo[3 * m] * sig[kAt[c][0]][v]));
                    stv<T, SV>(fp + (c * 3 + m) * 27 * S, flux[c * 3 + m]);
                }
        }
    }
    __syncthreads();
    if (!active) return;
    T y[3][SV];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int v = 0; v < SV; ++v) y[c][v] = T(0);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        T d0, d1, d2;
        gll_dcol<T>(qm[m], d0, d1, d2);
        if constexpr (BOX != 0) { if (m > 0) { d0 *= geo[m]; d1 *= geo[m]; d2 *= geo[m]; } }
        const int i0 = qm[m] == 0 ? 1 : 0, i1 = qm[m] == 2 ? 1 : 2;
        const T f0 = i0 == 0 ? d0 : d1, f1 = i1 == 2 ? d2 : d1, fo = qm[m] == 0 ? d0 : (qm[m] == 1 ? d1 : d2);
        const T *p0 = F + (base[m] + i0 * kStride[m]) * S + s0, *p1 = F + (base[m] + i1 * kStride[m]) * S + s0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int f = BOX ? kAt[c][m] : c * 3 + m;
            T a0[SV], a1[SV];
            lds(p0 + f * 27 * S, a0);
            lds(p1 + f * 27 * S, a1);
#pragma unroll
            for (int v = 0; v < SV; ++v) y[c][v] += fmaT(f1, a1[v], fmaT(f0, a0[v], fo * flux[f][v]));
        }
    }
    T *o = L.rslot + (size_t(q) * 3 * L.nrd + e) * S + s0;
#pragma unroll
    for (int c = 0; c < 3; ++c) stv<T, SV>(o + size_t(c) * L.nrd * S, y[c]);
}

// The same for large grids in FP32, with one thread per (box element, shot): the 81
// displacements and the 81 sums of an element live in its thread's registers (254 of
// them).  With a thread per point the kernel is bound by shared memory (39 reads and 9
// writes a point and shot); here nothing passes through it: 88 -> 45 us a stage for 32000
// elements and 8 shots, 113 MB.
template <typename T, int S>
__global__ void __launch_bounds__(64, 4) k_line_r(const LineArgs<T> L, const T *ut)
{
    dep_trigger();
    const int64_t tid = blockIdx.x * int64_t(64) + threadIdx.x;
    const int64_t e64 = tid / S;
    if (e64 >= L.nrd) return;
    const int e = int(e64), s = int(tid % S);
    const size_t nrd = size_t(L.nrd);
    const T r[3] = {T(1), T(__ldg(L.rgeo + size_t(e) * 4)), T(__ldg(L.rgeo + size_t(e) * 4 + 1))};
    T u[3][27], y[3][27];
    int id[27];
#pragma unroll
    for (int q = 0; q < 27; ++q) id[q] = __ldg(L.runode + q * nrd + e);
    dep_wait();
#pragma unroll
    for (int q = 0; q < 27; ++q)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            T v[1];
            ldw_if<T, 1>(id[q] >= 0, ut + (size_t(c) * L.nun + uint32_t(id[q])) * S + s, v);
            u[c][q] = v[0];
            y[c][q] = T(0);
        }
    constexpr int str[3] = {1, 3, 9};
    constexpr T D[3][3] = {{T(-1.5), T(2), T(-0.5)}, {T(-0.5), T(0), T(0.5)}, {T(0.5), T(-2), T(1.5)}};
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int qm[3] = {q % 3, (q / 3) % 3, q / 9};
        T g[3][3];   // d u_c / d x_m
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int b = q - qm[m] * str[m];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                T v = D[qm[m]][0] * u[c][b];
                if (qm[m] != 1) v = fmaT(D[qm[m]][1], u[c][b + str[m]], v);
                v = fmaT(D[qm[m]][2], u[c][b + 2 * str[m]], v);
                g[c][m] = m > 0 ? v * r[m] : v;
            }
        }
        const T lam = L.rlam[q * nrd + e], mu = L.rmu[q * nrd + e], m2 = T(2) * mu;
        const T tr = lam * (g[0][0] + g[1][1] + g[2][2]);
        T f[3][3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f[c][c] = fmaT(m2, g[c][c], tr);
#pragma unroll
            for (int m = c + 1; m < 3; ++m) f[c][m] = f[m][c] = mu * (g[c][m] + g[m][c]);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int b = q - qm[m] * str[m];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T v = m > 0 ? f[c][m] * r[m] : f[c][m];
                y[c][b] = fmaT(D[qm[m]][0], v, y[c][b]);
                if (qm[m] != 1) y[c][b + str[m]] = fmaT(D[qm[m]][1], v, y[c][b + str[m]]);
                y[c][b + 2 * str[m]] = fmaT(D[qm[m]][2], v, y[c][b + 2 * str[m]]);
            }
        }
    }
    T *o = L.rslot + size_t(e) * S + s;
#pragma unroll
    for (int q = 0; q < 27; ++q)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[size_t(3 * q + c) * nrd * S] = y[c][q];
}
// Its material: lambda, mu of the points times w detJ DJI_x^2, formed in FP64.
template <typename T>
__global__ void __launch_bounds__(256) k_line_material(const LineArgs<T> L)
{
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= int64_t(27) * L.nrd) return;
    const int q = int(t / L.nrd), e = int(t % L.nrd);
    const double third = 1.0 / 3.0, mid = 4.0 / 3.0;   // GLL weights
    const double f = __ldg(L.rgeo + size_t(e) * 4 + 2) * (q % 3 == 1 ? mid : third) * (q / 3 % 3 == 1 ? mid : third) * (q / 9 == 1 ? mid : third);
    const int node = __ldg(L.rpt + size_t(e) * 27 + q).x;
    L.rlam[t] = T(f * __ldg(L.lam + node));
    L.rmu[t] = T(f * __ldg(L.mu + node));
}

// Stress rows of one PML node and the P of its next inputs.
template <typename T, int S, int SV, int stage, int ADJ>
__device__ __forceinline__ void line_stress_rows(const LineArgs<T> &L, int block)
{
    constexpr int TP = S / SV, N = 4;   // entries of a direction in flight
    const int pn = block * line_nodes<S, SV>() + int(threadIdx.x) / TP, s0 = int(threadIdx.x % TP) * SV;
    if (int(threadIdx.x) / TP >= line_nodes<S, SV>() || pn >= L.npn) return;
    const uint32_t np = uint32_t(L.npn), plane = np * S;
    const int2 nd = __ldg(L.pnode + pn);
    auto coef = [&](int i) { return __ldg(L.pcoef + size_t(i) * np + pn); };
    int id[3][N];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int u = 0; u < N; ++u) id[k][u] = u < L.wd ? __ldg(L.didx + size_t(k * L.wd + u) * np + pn) : -1;
    const bool use_g = coef(kCoefG) != T(0);
    const T lam = T(__ldg(L.lam + nd.x)), mu2 = T(2.0 * __ldg(L.mu + nd.x));
    dep_wait();
    T g[3][3][SV];   // [direction][component]
    {
        T q[2][N][3][SV];
        auto get = [&](int k, T (&o)[N][3][SV]) {
#pragma unroll
            for (int u = 0; u < N; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    ldw_if<T, SV>(id[k][u] >= 0, L.Z + (size_t(3 * k + c) * plane + uint32_t(id[k][u]) * S + s0), o[u][c]);
        };
        auto sum = [&](int k, const T (&o)[N][3][SV]) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int v = 0; v < SV; ++v) g[k][c][v] = T(0);
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const T cf = u < L.wd ? __ldg(L.dcf + size_t(k * L.wd + u) * np + pn) : T(0);
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int v = 0; v < SV; ++v) g[k][c][v] = fmaT(cf, o[u][c][v], g[k][c][v]);
            }
            for (int u = N; u < L.wd; ++u) {   // lines with more points
                const int j = __ldg(L.didx + size_t(k * L.wd + u) * np + pn);
                if (j < 0) break;
                const T cf = __ldg(L.dcf + size_t(k * L.wd + u) * np + pn);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    T z[SV];
                    ldw<T, SV>(L.Z + (size_t(3 * k + c) * plane + uint32_t(j) * S + s0), z);
#pragma unroll
                    for (int v = 0; v < SV; ++v) g[k][c][v] = fmaT(cf, z[v], g[k][c][v]);
                }
            }
        };
        get(0, q[0]);
        get(1, q[1]);
        sum(0, q[0]);
        get(2, q[0]);
        sum(1, q[1]);
        sum(2, q[0]);
    }
    const uint32_t o0 = 3 * uint32_t(L.nun) * S + uint32_t(pn) * S + s0;   // row of component xx
    // adjoint: C and G enter with a minus sign (their transposes are negated)
    const T sg = ADJ ? T(-1) : T(1);
    const T n0 = sg * coef(kCoefDiag), n1 = coef(kCoefDiag + 1), n2 = use_g ? sg * coef(kCoefDiag + 2) : T(0);
    T w[9];
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = i < 3 ? sg * coef(i) : coef(i);
#pragma unroll
    for (int i = 6; i < 9; ++i) w[i] = use_g ? sg * coef(i) : T(0);
    T *P = L.Pn + uint32_t(pn) * S + s0;
    T pk[3][SV];   // P_k(k)
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int v = 0; v < SV; ++v) pk[k][v] = T(0);
    T tr[SV];
#pragma unroll
    for (int v = 0; v < SV; ++v) tr[v] = lam * (g[0][0][v] + g[1][1][v] + g[2][2][v]);
#pragma unroll
    for (int half = 0; half < 2; ++half) {   // normal rows, then shear rows: three rows' operands in flight
        const T cy = coef(half ? kCoefYShear : kCoefY);
        RowIn<T, SV, stage> x[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) x[i].load(L, o0 + uint32_t(3 * half + i) * plane, use_g);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int d = 3 * half + i;
            const int ci = half ? (i == 2 ? 1 : 0) : i, cj = half ? (i == 0 ? 1 : 2) : i;   // the component's axes
            T y[SV], m[SV], t[SV], h[SV], kb[SV], nm[SV], nt[SV], nh[SV];
#pragma unroll
            for (int v = 0; v < SV; ++v) {
                if (half) {
                    y[v] = g[cj][ci][v] + g[ci][cj][v];
                    if (ADJ) y[v] *= -mu2;
                } else {
                    y[v] = ADJ ? -fmaT(mu2, g[i][i][v], tr[v]) : g[i][i][v];
                }
            }
            x[i].inputs(L, m, t, h);
#pragma unroll
            for (int v = 0; v < SV; ++v) kb[v] = fmaT(n2, h[v], fmaT(n1, t[v], fmaT(n0, m[v], cy * y[v])));
            if (L.stress_src) add_source<T, S, SV, stage>(L, nd.y + d, s0, kb);
            if (stage == 1 && L.stress_hist && L.hist) add_history<T, S, SV>(L, nd.y + d, s0, x[i].x2);
            x[i].finish(L, o0 + uint32_t(d) * plane, kb, m, t, nm, nt, nh);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const bool shear = half && (k == ci || k == cj);
                if (!shear && (half || (ADJ && k != i))) continue;
                T z[SV];
#pragma unroll
                for (int v = 0; v < SV; ++v) z[v] = fmaT(w[6 + k], nh[v], fmaT(w[3 + k], nt[v], w[k] * nm[v]));
                if (half) {
                    // direction k, the other axis as component
#pragma unroll
                    for (int v = 0; v < SV; ++v)
                        if (!ADJ) z[v] *= -mu2;
                    stv<T, SV>(P + size_t(3 * k + (k == ci ? cj : ci)) * plane, z);
                } else {
#pragma unroll
                    for (int v = 0; v < SV; ++v) pk[k][v] = ADJ ? z[v] : fmaT(k == i ? -(lam + mu2) : -lam, z[v], pk[k][v]);
                }
            }
        }
        if (!half) {
#pragma unroll
            for (int k = 0; k < 3; ++k) stv<T, SV>(P + size_t(4 * k) * plane, pk[k]);
        }
    }
}

template <typename T, int S, int SV, int stage, int ADJ, int BOX>
__global__ void __launch_bounds__(line_threads<S, SV>(), line_blocks<T, S, SV, 0>()) k_line_a(const LineArgs<T> L, int nb_stress)
{
    extern __shared__ __align__(16) unsigned char line_sm[];
    dep_trigger();
    if (int(blockIdx.x) < nb_stress)
        line_stress_rows<T, S, SV, stage, ADJ>(L, int(blockIdx.x));
    else
        line_rd_elements<T, S, SV, BOX>(L, stage == 1 ? L.x2 : L.kt, int(blockIdx.x) - nb_stress, reinterpret_cast<T *>(line_sm));
}

// P and Z of the state, for the first stage of a run of steps: one thread per PML node,
// direction and shot.
template <typename T, int S, int ADJ>
__global__ void __launch_bounds__(256) k_line_p0(const LineArgs<T> L)
{
    const int64_t tid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    const int64_t j = tid / S;
    const int s = int(tid % S);
    if (j >= int64_t(3) * L.npn) return;
    const int k = int(j / L.npn), pn = int(j % L.npn);
    const uint32_t np = uint32_t(L.npn), plane = np * S;
    const int2 nd = __ldg(L.pnode + pn);
    const T sg = ADJ ? T(-1) : T(1);
    const T w0 = sg * __ldg(L.pcoef + size_t(k) * np + pn), w1 = __ldg(L.pcoef + size_t(3 + k) * np + pn),
            w2 = sg * __ldg(L.pcoef + size_t(6 + k) * np + pn);
    const T lam = T(__ldg(L.lam + nd.x)), mu2 = T(2.0 * __ldg(L.mu + nd.x));
    T q[6];
    const uint32_t o0 = 3 * uint32_t(L.nun) * S + uint32_t(pn) * S + s;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const uint32_t o = o0 + uint32_t(d) * plane;
        q[d] = fmaT(w2, L.x1[o], fmaT(w1, L.x2[o], w0 * L.x3[o]));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const T n = k == 0 ? q[0] : (k == 1 ? q[1] : q[2]);
        const T sh = k + c == 1 ? q[3] : (k + c == 2 ? q[4] : q[5]);
        const T v = ADJ ? (c == k ? n : sh) : (c == k ? -fmaT(mu2, n, lam * (q[0] + q[1] + q[2])) : -mu2 * sh);
        L.Pn[size_t(3 * k + c) * plane + uint32_t(pn) * S + s] = v;
    }
}
// Z of one displacement node of the PML and direction.
template <typename T, int S, int ADJ>
__global__ void __launch_bounds__(256) k_line_z0(const LineArgs<T> L)
{
    const int64_t tid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    const int64_t j = tid / S;
    const int s = int(tid % S);
    if (j >= int64_t(3) * L.nup) return;
    const int k = int(j / L.nup), un = int(j % L.nup), pn = __ldg(L.unode + un).y;
    const T sg = ADJ ? T(-1) : T(1);
    const T w0 = sg * __ldg(L.ucoef + size_t(k) * L.nup + un), w1 = __ldg(L.ucoef + size_t(3 + k) * L.nup + un),
            w2 = sg * __ldg(L.ucoef + size_t(6 + k) * L.nup + un);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const size_t o = (size_t(c) * L.nun + un) * S + s;
        L.Z[(size_t(3 * k + c) * L.npn + pn) * S + s] = fmaT(w2, L.x1[o], fmaT(w1, L.x2[o], w0 * L.x3[o]));
    }
}

// Displacement rows of one node; nodes of the PML first.
template <typename T, int S, int SV, int stage, int ADJ>
__global__ void __launch_bounds__(line_threads<S, SV>(), line_blocks<T, S, SV, 1>()) k_line_b(const LineArgs<T> L)
{
    constexpr int TP = S / SV, N = 4;   // records in flight
    dep_trigger();
    const int un = int(blockIdx.x) * line_nodes<S, SV>() + int(threadIdx.x) / TP, s0 = int(threadIdx.x % TP) * SV;
    if (int(threadIdx.x) / TP >= line_nodes<S, SV>() || un >= L.nun) return;
    const int4 nd = __ldg(L.unode + un);
    const bool pml = un < L.nup;
    const uint32_t plane = uint32_t(L.npn) * S, rplane = uint32_t(L.nrd) * S, uplane = uint32_t(L.nun) * S;
    auto coef = [&](int i) { return __ldg(L.ucoef + size_t(i) * L.nup + un); };
    const double im = __ldg(L.uim + un);   // applied in FP64: it repeats over the regular domain
    const bool use_g = pml && coef(kCoefG) != T(0);
    int id[8];
    if (pml) {
#pragma unroll
        for (int u = 0; u < 8; ++u) id[u] = u < L.wt ? __ldg(L.tidx + size_t(u) * L.nup + un) : -1;
    } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) id[u] = u < nd.z ? __ldg(L.ridx + size_t(u) * L.nun + un) : -1;
    }
    dep_wait();
    T acc[3][SV];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int v = 0; v < SV; ++v) acc[c][v] = T(0);
    // records of N entries in flight: P with the factors of D^T, element contributions with 1
    auto some = [&](const T *base, uint32_t pl, const int *ix, const T *cf, size_t stride) {
        T q[N][3][SV];
#pragma unroll
        for (int u = 0; u < N; ++u)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                ldw_if<T, SV>(ix[u] >= 0, base + (size_t(c) * pl + size_t(uint32_t(ix[u])) * S + s0), q[u][c]);
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const T f = cf && ix[u] >= 0 ? __ldg(cf + u * stride) : T(1);
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int v = 0; v < SV; ++v) acc[c][v] = fmaT(f, q[u][c][v], acc[c][v]);
        }
    };
    int ne = nd.z, e = 0;   // element contributions, and how many of them are already in id[]
    if (pml) {
        some(L.P, plane, id, L.tcf + un, L.nup);
        some(L.P, plane, id + N, L.tcf + size_t(N) * L.nup + un, L.nup);
        for (int u0 = 8; u0 < L.wt; u0 += N) {
            int ix[N];
#pragma unroll
            for (int u = 0; u < N; ++u) ix[u] = u0 + u < L.wt ? __ldg(L.tidx + size_t(u0 + u) * L.nup + un) : -1;
            if (ix[0] < 0) break;
            some(L.P, plane, ix, L.tcf + size_t(u0) * L.nup + un, L.nup);
        }
    } else {
        some(L.rslot, rplane, id, nullptr, 0);
        if (ne > N) some(L.rslot, rplane, id + N, nullptr, 0);
        e = 8;
    }
    for (; e < ne; e += N) {
        int ix[N];
#pragma unroll
        for (int u = 0; u < N; ++u) ix[u] = e + u < ne ? __ldg(L.ridx + size_t(e + u) * L.nun + un) : -1;
        some(L.rslot, rplane, ix, nullptr, 0);
    }
    RowIn<T, SV, stage> x[3];
    const uint32_t o0 = uint32_t(un) * S + s0;
#pragma unroll
    for (int c = 0; c < 3; ++c) x[c].load(L, o0 + uint32_t(c) * uplane, use_g, !pml);
    const T sg = ADJ ? T(-1) : T(1);
    T w[9], d0 = T(0), d1 = T(0), d2 = T(0);
    if (pml) {
        d0 = sg * coef(kCoefDiag);
        d1 = coef(kCoefDiag + 1);
#pragma unroll
        for (int i = 0; i < 6; ++i) w[i] = i < 3 ? sg * coef(i) : coef(i);
    }
    if (use_g) d2 = sg * coef(kCoefDiag + 2);
#pragma unroll
    for (int i = 6; i < 9; ++i) w[i] = use_g ? sg * coef(i) : T(0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint32_t o = o0 + uint32_t(c) * uplane;
        T m[SV], t[SV], h[SV], kb[SV], nm[SV], nt[SV], nh[SV];
        x[c].inputs(L, m, t, h);   // outside the PML only m is meaningful, and only m is used
#pragma unroll
        for (int v = 0; v < SV; ++v) kb[v] = T(im * double(acc[c][v]));
        if (pml) {
#pragma unroll
            for (int v = 0; v < SV; ++v) kb[v] = fmaT(d2, h[v], fmaT(d1, t[v], fmaT(d0, m[v], kb[v])));
        }
        add_source<T, S, SV, stage>(L, nd.x + c, s0, kb);
        if (stage == 1 && L.hist) add_history<T, S, SV>(L, nd.x + c, s0, x[c].x2);
        x[c].finish(L, o, kb, m, t, nm, nt, nh);
        if (stage < 4 && ne > 0) stv<T, SV>(L.kt + o, nt);
        if (pml) {
            T *Z = L.Z + (size_t(c) * plane + uint32_t(nd.y) * S + s0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                T z[SV];
#pragma unroll
                for (int v = 0; v < SV; ++v) z[v] = fmaT(w[6 + k], nh[v], fmaT(w[3 + k], nt[v], w[k] * nm[v]));
                stv<T, SV>(Z + size_t(3 * k) * plane, z);
            }
        }
    }
}

// ----------------------------------------------------------------------------
// launches

template <typename T, int S, int SV, int STAGE, int ADJ>
static void line_launch(hrn_ctx *c, LineArgs<T> &L, int first, bool pdl)
{
    constexpr int NT = line_threads<S, SV>(), NPB = line_nodes<S, SV>(), EPB = line_elems<S, SV>();
    const size_t psz = size_t(L.npn) * 9 * S;   // P of the two parities, then Z
    T *buf = L.P;
    L.Z = buf + 2 * psz;
    if constexpr (STAGE == 1) {
        if (first && L.npn > 0) {
            L.Pn = buf;
            const int64_t np = int64_t(3) * L.npn * S, nz = int64_t(3) * L.nup * S;
            k_line_p0<T, S, ADJ><<<unsigned((np + 255) / 256), 256, 0, c->stream>>>(L);
            ++c->launches;
            if (nz > 0) {
                k_line_z0<T, S, ADJ><<<unsigned((nz + 255) / 256), 256, 0, c->stream>>>(L);
                ++c->launches;
            }
        }
    }
    L.P = buf + ((STAGE - 1) & 1) * psz;
    L.Pn = buf + (STAGE & 1) * psz;
    const int nb_s = (L.npn + NPB - 1) / NPB;
    int nb_r = (L.nrd + EPB - 1) / EPB;
    if constexpr (sizeof(T) == 4) {
        if (line_reg_elements(c)) {
            if (STAGE == 1 && first) {
                k_line_material<T><<<unsigned((int64_t(27) * L.nrd + 255) / 256), 256, 0, c->stream>>>(L);
                ++c->launches;
            }
            chain_start(k_line_r<T, S>, int((int64_t(L.nrd) * S + 63) / 64), 64, 0, c->stream, pdl, L, static_cast<const T *>(STAGE == 1 ? L.x2 : L.kt));
            ++c->launches;
            pdl = true;
            nb_r = 0;
        }
    }
    if (nb_s + nb_r > 0) {
        static_assert(line_smem<T, S, SV, 0>() <= 48 * 1024, "k_line_a exceeds the default shared memory of a CTA");
        if (c->rd_box)
            chain_start(k_line_a<T, S, SV, STAGE, ADJ, 1>, nb_s + nb_r, NT, line_smem<T, S, SV, 1>(), c->stream, pdl, L, nb_s);
        else
            chain_start(k_line_a<T, S, SV, STAGE, ADJ, 0>, nb_s + nb_r, NT, line_smem<T, S, SV, 0>(), c->stream, pdl, L, nb_s);
        ++c->launches;
    }
    const int nb_u = (L.nun + NPB - 1) / NPB;
    if (nb_u > 0) chain_start(k_line_b<T, S, SV, STAGE, ADJ>, nb_u, NT, 0, c->stream, nb_s + nb_r > 0 || pdl, L);
    // the caller counts one launch per stage
}

template <typename T>
static LineArgs<T> line_args(hrn_ctx *c, const StageArgs<T> &a, int set)
{
    LineArgs<T> L{};
    L.npn = c->line_npn;
    L.nup = c->line_nup;
    L.nun = c->line_nun;
    L.nrd = c->nel_rd_e;
    L.wd = c->line_wd;
    L.wt = c->line_wt;
    L.pnode = c->d_line_pnode.as<int2>();
    L.didx = c->d_line_didx.as<int32_t>();
    L.dcf = c->d_line_dcf.as<T>();
    L.pcoef = c->d_line_pcoef.as<T>();
    L.unode = c->d_line_unode.as<int4>();
    L.tidx = c->d_line_tidx.as<int32_t>();
    L.tcf = c->d_line_tcf.as<T>();
    L.ridx = c->d_line_ridx.as<int32_t>();
    L.ucoef = c->d_line_ucoef.as<T>();
    L.uim = c->d_line_uim.as<double>();
    L.rpt = c->d_line_rpt.as<int2>();
    L.rgeo = c->d_line_rgeo.as<double>();
    L.runode = c->d_line_runode.as<int32_t>();
    L.rlam = c->d_line_rmat.as<T>();
    L.rmu = L.rlam + size_t(27) * c->nel_rd_e;
    L.lam = c->d_lam.as<double>();
    L.mu = c->d_mu.as<double>();
    L.x1 = const_cast<T *>(a.x1);
    L.x2 = const_cast<T *>(a.x2);
    L.x3 = const_cast<T *>(a.x3);
    L.k1 = const_cast<T *>(a.kb1);
    L.k2 = const_cast<T *>(a.kb2);
    L.k3 = const_cast<T *>(a.kb3);
    L.kt = a.out_t;
    L.rslot = c->d_line_rslot.as<T>();
    L.P = c->d_line_P.as<T>() + (c->ckpt > 0 ? set : 0) * (size_t(3) * 9 * c->line_npn * c->nshot);
    L.hist = a.hist;
    L.slot = a.slot;
    L.store_pos = a.store_pos;
    L.srcv = a.srcv;
    L.nslot = a.nslot;
    L.stress_src = c->line_stress_src;
    L.stress_hist = c->line_stress_hist;
    L.c = a.c;
    L.D = a.D;
    L.d6 = a.d6;
    return L;
}

template <typename T, int S>
static int line_stage_t(hrn_ctx *c, const StageArgs<T> &a, int stage, int adj, int sv, int first, bool pdl)
{
    LineArgs<T> L = line_args<T>(c, a, adj);
    auto go = [&](auto svc) {
        constexpr int SV = decltype(svc)::value;
        auto st = [&](auto stc) {
            constexpr int ST = decltype(stc)::value;
            if (adj) line_launch<T, S, SV, ST, 1>(c, L, first, pdl);
            else line_launch<T, S, SV, ST, 0>(c, L, first, pdl);
        };
        switch (stage) {
        case 1: st(std::integral_constant<int, 1>{}); break;
        case 2: st(std::integral_constant<int, 2>{}); break;
        case 3: st(std::integral_constant<int, 3>{}); break;
        default: st(std::integral_constant<int, 4>{}); break;
        }
    };
    if constexpr (S % 4 == 0 && sizeof(T) == 4) {
        if (sv >= 4) { go(std::integral_constant<int, 4>{}); return 0; }
    }
    if constexpr (S % 2 == 0) {
        if (sv >= 2) { go(std::integral_constant<int, 2>{}); return 0; }
    }
    go(std::integral_constant<int, 1>{});
    return 0;
}

template <typename T>
static int line_stage_any(hrn_ctx *c, const void *args, int stage, int adj, int sv, int first, bool pdl)
{
    const StageArgs<T> &a = *static_cast<const StageArgs<T> *>(args);
    switch (c->nshot) {
    case 1: return line_stage_t<T, 1>(c, a, stage, adj, sv, first, pdl);
    case 2: return line_stage_t<T, 2>(c, a, stage, adj, sv, first, pdl);
    case 3: return line_stage_t<T, 3>(c, a, stage, adj, sv, first, pdl);
    case 4: return line_stage_t<T, 4>(c, a, stage, adj, sv, first, pdl);
    case 5: return line_stage_t<T, 5>(c, a, stage, adj, sv, first, pdl);
    case 6: return line_stage_t<T, 6>(c, a, stage, adj, sv, first, pdl);
    case 7: return line_stage_t<T, 7>(c, a, stage, adj, sv, first, pdl);
    default: return line_stage_t<T, 8>(c, a, stage, adj, sv, first, pdl);
    }
}

}  // namespace hrn
