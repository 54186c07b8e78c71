// Control-net reduced Gauss-Newton kernels (src/control_net.hpp:486-1106,
// src/control_solve.hpp:533-820).
//
// A net drives one block of the store: X = M C + b with M the tensor product
// of per-axis clamped B-spline bases (banded: node i of axis k reads controls
// off_k[i] .. off_k[i] + k_supp - 1 with weights wt_k[i, :]).  Several nets
// (one per mesh of a batch) are stacked: net-node, lattice and free-control
// spaces are concatenations indexed through per-net offsets.
//
// Per-node work runs over a net's block nodes and reads the block's canonical
// cell stencil directly (cells of the block around the node, 2^D corner
// samples each, the node's role in each), so no membership tables are stored
// and each sample's metric work is fused with the node gather:
//   grad  y_n = sum_p wt_p J_b(n,p)^T dmu/dT(T_p)
//   hvp   y_n = sum_p wt_p J_b(n,p)^T H(T_p) dT_p,  dT_p assembled from corr
//   hess  h_n = sum_p wt_p J_b^T H(T_p) J_b          (Jacobi preconditioner)
// J_b(n,p) is rank one, e_i v^T: v = -W^T s for the corner, s_k W[k,:] for
// the axis-k neighbour.
#pragma once

#include "kernels3d.cuh"

#include <cooperative_groups.h>

namespace egg_b200
{

struct CtlNet {
    int32_t block;
    int32_t k_supp;
    int32_t node_shape[3];
    int32_t ctrl_shape[3];
    int32_t ctrl_stride[3];
    int32_t pad;
    int64_t node_off;  // store slot of the block's first node
    int64_t cell_off;  // first canonical energy-stencil cell of the block
    int64_t n_off;     // first net node (b and node-space buffers)
    int64_t c_off;     // first lattice control
    int64_t f_off;     // first free control
    int64_t n_nodes, n_ctrl, n_free;
    int64_t ax_off[3];   // into the concatenated per-axis off / wt tables (nodes)
    int64_t sup_base[3]; // into the concatenated support CSR offsets (controls + 1)
};

struct CtlTables {
    int32_t n_nets;
    const CtlNet* nets;
    const int64_t* node_pfx;  // [n_nets + 1] net-node prefix
    const int64_t* ctrl_pfx;  // [n_nets + 1] lattice prefix
    const int64_t* free_pfx;  // [n_nets + 1] free-control prefix
    const int32_t* off;       // per-axis first support control per node
    const double* wt;         // per-axis basis weights [node * k_supp]
    const int32_t* sup_off;   // per-axis support CSR offsets (relative to sup entries of the net axis)
    const int32_t* sup_node;  // support nodes
    const double* sup_w;      // support weights
    const int32_t* free_idx;  // [free] lattice index within the net
    const int32_t* free_midx; // [free * D] multi-index
    const int32_t* free_of;   // [lattice] stacked free index or -1
};

// Per-net PCG state (device resident; thread 0 of the per-net reduction CTA
// updates it, kernels skip nets whose `done` is set).
struct PcgState {
    double b_norm2, stop2, r_norm2, rz, alpha, beta, lam, pad;
    int32_t it, its, done, max_iter, active, pad2;
};

__device__ __forceinline__ int net_of(const int64_t* pfx, int n, int64_t i)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pfx[mid] <= i) {
            lo = mid;
        } else {
            hi = mid - 1;
        }
    }
    return lo;
}

template <int D> __device__ __forceinline__ void unravel_node(const CtlNet& n, int64_t f, int L[3])
{
    L[2] = 0;
    if (D == 3) {
        L[2] = int(f % n.node_shape[2]);
        f /= n.node_shape[2];
    }
    L[1] = int(f % n.node_shape[1]);
    L[0] = int(f / n.node_shape[1]);
}

// X (store) = M C + b, or a net-node field out = M C (b == null, node_space).
template <int D>
__global__ void ctl_eval_kernel(CtlTables T, int64_t total_nodes, const double* __restrict__ C,
                                const double* __restrict__ b, double* __restrict__ out, bool node_space,
                                const PcgState* __restrict__ st)
{
    for (int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; g < total_nodes;
         g += int64_t(gridDim.x) * blockDim.x) {
        const int ni = net_of(T.node_pfx, T.n_nets, g);
        if (st && st[ni].done) { continue; }
        const CtlNet n = T.nets[ni];
        const int64_t f = g - n.n_off;
        int L[3];
        unravel_node<D>(n, f, L);
        const int ks = n.k_supp;
        double acc[D];
#pragma unroll
        for (int c = 0; c < D; ++c) { acc[c] = 0.0; }
        const int32_t* off0 = T.off + n.ax_off[0];
        const int32_t* off1 = T.off + n.ax_off[1];
        const double* wt0 = T.wt + n.ax_off[0] * ks;
        const double* wt1 = T.wt + n.ax_off[1] * ks;
        const double* Cn = C + n.c_off * D;
        if (D == 2) {
            for (int t0 = 0; t0 < ks; ++t0) {
                const double w0 = wt0[L[0] * ks + t0];
                const int64_t r0 = int64_t(off0[L[0]] + t0) * n.ctrl_stride[0];
                for (int t1 = 0; t1 < ks; ++t1) {
                    const double w = 1.0 * w0 * wt1[L[1] * ks + t1];
                    const int64_t ci = r0 + int64_t(off1[L[1]] + t1) * n.ctrl_stride[1];
#pragma unroll
                    for (int c = 0; c < D; ++c) { acc[c] += w * Cn[ci * D + c]; }
                }
            }
        } else {
            const int32_t* off2 = T.off + n.ax_off[2];
            const double* wt2 = T.wt + n.ax_off[2] * ks;
            for (int t0 = 0; t0 < ks; ++t0) {
                const double w0 = wt0[L[0] * ks + t0];
                const int64_t r0 = int64_t(off0[L[0]] + t0) * n.ctrl_stride[0];
                for (int t1 = 0; t1 < ks; ++t1) {
                    const double w01 = 1.0 * w0 * wt1[L[1] * ks + t1];
                    const int64_t r1 = r0 + int64_t(off1[L[1]] + t1) * n.ctrl_stride[1];
                    for (int t2 = 0; t2 < ks; ++t2) {
                        const double w = w01 * wt2[L[2] * ks + t2];
                        const int64_t ci = r1 + int64_t(off2[L[2]] + t2) * n.ctrl_stride[2];
#pragma unroll
                        for (int c = 0; c < D; ++c) { acc[c] += w * Cn[ci * D + c]; }
                    }
                }
            }
        }
        if (node_space) {
#pragma unroll
            for (int c = 0; c < D; ++c) { out[g * D + c] = acc[c]; }
        } else {
            const int64_t slot = n.node_off + f;
#pragma unroll
            for (int c = 0; c < D; ++c) { out[slot * D + c] = acc[c] + (b ? b[g * D + c] : 0.0); }
        }
    }
}

// C_dir[lattice] = v[free] on free controls, 0 elsewhere.
template <int D>
__global__ void ctl_scatter_kernel(CtlTables T, int64_t total_ctrl, const double* __restrict__ v,
                                   double* __restrict__ Cdir)
{
    for (int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; g < total_ctrl;
         g += int64_t(gridDim.x) * blockDim.x) {
        const int32_t f = T.free_of[g];
#pragma unroll
        for (int c = 0; c < D; ++c) { Cdir[g * D + c] = f >= 0 ? v[int64_t(f) * D + c] : 0.0; }
    }
}

enum { kCtlGrad = 0, kCtlHvp = 1, kCtlHess = 2 };

// Rank-one direction of node role r in a sample (v = -W^T s or s_k W[k,:]).
template <int D> __device__ __forceinline__ void role_dir(int role, const double* w, const double s[3], double v[3])
{
#pragma unroll
    for (int j = 0; j < D; ++j) {
        if (role == 0) {
            double a = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) { a -= s[k] * w[k * D + j]; }
            v[j] = a;
        } else {
            v[j] = s[role - 1] * w[(role - 1) * D + j];
        }
    }
}

// The directional soft terms' nodal gradient added into the net-node
// gradient y (src/directional.hpp:343-379, src/control_solve.hpp:556-559):
// every node of every sample, at its owner slot; a slot inside a net's block
// adds to that net's node.  The control's Newton model and preconditioner
// stay the shape term's, as in the reference.
template <int D>
__global__ void ctl_dir_scatter_kernel(CtlTables T, const SoftTerm* __restrict__ terms, int64_t n, double eps,
                                       const double* __restrict__ X, double* __restrict__ y)
{
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        SoftTerm t = terms[i];
        const int ar = soft_arity(t.kind);
        for (int m = 0; m < ar; ++m) {
            const int64_t slot = t.node[m];
            int ni = -1;
            for (int q = 0; q < T.n_nets && ni < 0; ++q) {
                if (slot >= T.nets[q].node_off && slot < T.nets[q].node_off + T.nets[q].n_nodes) { ni = q; }
            }
            if (ni < 0) { continue; }
            t.slot = m;
            double g[D], H[D * D], e = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) { g[k] = 0.0; }
#pragma unroll
            for (int k = 0; k < D * D; ++k) { H[k] = 0.0; }
            soft_accumulate<D>(t, X, eps, g, H, e);
            const int64_t row = T.nets[ni].n_off + (slot - T.nets[ni].node_off);
#pragma unroll
            for (int k = 0; k < D; ++k) { atomicAdd(&y[row * D + k], g[k]); }
        }
    }
}

// Hessian-vector product of the 2D metric, from its closed form (metric.cuh)
// without the 4 x 4 Hessian: with P dT = cof(dT) and D' = cof : dT,
//   H dT = 2 f dT + 2 f' (T D' + cof (T : dT)) + s f'' D' cof + s f' P dT.
template <int KIND> __device__ __forceinline__ void mu2_hvp(const double t[4], const double dt[4], double hv[4])
{
    const double cof[4] = {t[3], -t[2], -t[1], t[0]}, pd[4] = {dt[3], -dt[2], -dt[1], dt[0]};
    const double D = det2(t), s = t[0] * t[0] + t[1] * t[1] + t[2] * t[2] + t[3] * t[3];
    const ScaleFn<double> sf = shape_scale(D);
    const double Dd = cof[0] * dt[0] + cof[1] * dt[1] + cof[2] * dt[2] + cof[3] * dt[3];
    const double td = t[0] * dt[0] + t[1] * dt[1] + t[2] * dt[2] + t[3] * dt[3];
    const double a = 2.0 * sf.fp * Dd, b = 2.0 * sf.fp * td + s * sf.fpp * Dd, c = s * sf.fp;
#pragma unroll
    for (int i = 0; i < 4; ++i) { hv[i] = 2.0 * sf.f * dt[i] + a * t[i] + b * cof[i] + c * pd[i]; }
    if constexpr (KIND == kShapeSize) {  // mu = m^2 - 1 + (D - 1)^2, m = s f
        const double m = s * sf.f, md = 2.0 * sf.f * td + c * Dd, dm1 = D - 1.0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double g = 2.0 * sf.f * t[i] + c * cof[i];
            hv[i] = 2.0 * md * g + 2.0 * m * hv[i] + 2.0 * Dd * cof[i] + 2.0 * dm1 * pd[i];
        }
    }
}

// Per-node gradient / Hessian-vector product / contracted Hessian over the
// block's canonical cell stencil (see the file comment).
template <int D, int KIND, int MODE>
__global__ void ctl_node_kernel(CtlTables T, int64_t total_nodes, EnergyStructured2 es, const double* __restrict__ X,
                                const double* __restrict__ corr, double* __restrict__ out,
                                const PcgState* __restrict__ st)
{
    constexpr int NC = 1 << D;  // corners per cell
    constexpr int OUTW = MODE == kCtlHess ? D * D : D;
    for (int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; g < total_nodes;
         g += int64_t(gridDim.x) * blockDim.x) {
        const int ni = net_of(T.node_pfx, T.n_nets, g);
        if (st && st[ni].done) { continue; }
        const CtlNet n = T.nets[ni];
        const int64_t f = g - n.n_off;
        int L[3];
        unravel_node<D>(n, f, L);
        const int n0 = n.node_shape[0], n1 = n.node_shape[1], n2 = D == 3 ? n.node_shape[2] : 1;
        const int c1 = n1 - 1, c2 = D == 3 ? n2 - 1 : 1;
        double acc[OUTW];
#pragma unroll
        for (int i = 0; i < OUTW; ++i) { acc[i] = 0.0; }
        // cells around the node in ascending cell order (unrolled in 2D: which
        // samples move the node, and in what role, is then known at compile time)
#pragma unroll(D == 2 ? NC : 1)
        for (int cc = 0; cc < NC; ++cc) {
            int cl[3] = {L[0] - 1 + ((cc >> (D - 1)) & 1), L[1] - 1 + ((cc >> (D - 2)) & 1),
                         D == 3 ? L[2] - 1 + (cc & 1) : 0};
            if (cl[0] < 0 || cl[0] > n0 - 2 || cl[1] < 0 || cl[1] > n1 - 2) { continue; }
            if (D == 3 && (cl[2] < 0 || cl[2] > n2 - 2)) { continue; }
            const int q = cc ^ (NC - 1);  // node's corner index inside the cell (axis 0 most significant)
            const int64_t lc = (int64_t(cl[0]) * c1 + cl[1]) * c2 + (D == 3 ? cl[2] : 0);
            const int64_t cell = n.cell_off + lc;
            const int64_t base = n.node_off + (int64_t(cl[0]) * n1 + cl[1]) * n2 + (D == 3 ? cl[2] : 0);
#pragma unroll(D == 2 ? NC : 1)
            for (int b = 0; b < NC; ++b) {
                int role = -1;
                if (q == b) {
                    role = 0;
                } else {
#pragma unroll
                    for (int k = 0; k < D; ++k) {
                        if (q == (b ^ (1 << (D - 1 - k)))) { role = k + 1; }
                    }
                }
                if (role < 0) { continue; }
                const int64_t sid = cell * NC + b;
                const double* w = es.W + sid * es.w_stride;
                const double wt = es.wt[sid * es.wt_stride];
                double s[3];
#pragma unroll
                for (int k = 0; k < D; ++k) { s[k] = (b & (1 << (D - 1 - k))) ? -1.0 : 1.0; }
                auto corner_slot = [&](int a) {
                    if (D == 2) { return base + int64_t((a >> 1) & 1) * n1 + (a & 1); }
                    return base + (int64_t((a >> 2) & 1) * n1 + ((a >> 1) & 1)) * n2 + (a & 1);
                };
                double v[3];
                role_dir<D>(role, w, s, v);
                if constexpr (D == 2) {
                    const int64_t sc = corner_slot(b), sa = corner_slot(b ^ 2), sb = corner_slot(b ^ 1);
                    const double2* X2 = reinterpret_cast<const double2*>(X);
                    double t[4], detA;
                    assemble_T(X2[sc], X2[sa], X2[sb], s[0], s[1], w, t, detA);
                    double mu, gT[4], H[16];
                    if constexpr (MODE != kCtlHvp) { mu_eval<double>(KIND, t, 0.0, mu, gT, H); }
                    if constexpr (MODE == kCtlGrad) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) { acc[i] += wt * (gT[2 * i] * v[0] + gT[2 * i + 1] * v[1]); }
                    } else if constexpr (MODE == kCtlHvp) {
                        // dT from corr at the same corners (net-node indexed)
                        const int64_t gc = n.n_off + (sc - n.node_off), ga = n.n_off + (sa - n.node_off),
                                      gb = n.n_off + (sb - n.node_off);
                        const double2 dc = make_double2(corr[2 * gc], corr[2 * gc + 1]);
                        const double2 da = make_double2(corr[2 * ga], corr[2 * ga + 1]);
                        const double2 db = make_double2(corr[2 * gb], corr[2 * gb + 1]);
                        double dt[4], dd;
                        assemble_T(dc, da, db, s[0], s[1], w, dt, dd);
                        double hv[4];
                        mu2_hvp<KIND>(t, dt, hv);
#pragma unroll
                        for (int i = 0; i < 2; ++i) { acc[i] += wt * (hv[2 * i] * v[0] + hv[2 * i + 1] * v[1]); }
                    } else {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                double h = 0.0;
#pragma unroll
                                for (int a = 0; a < 2; ++a) {
#pragma unroll
                                    for (int c = 0; c < 2; ++c) { h += H[(2 * i + a) * 4 + 2 * j + c] * v[a] * v[c]; }
                                }
                                acc[2 * i + j] += wt * h;
                            }
                        }
                    }
                } else {
                    const int32_t ic = int32_t(corner_slot(b));
                    const int32_t in[3] = {int32_t(corner_slot(b ^ 4)), int32_t(corner_slot(b ^ 2)),
                                           int32_t(corner_slot(b ^ 1))};
                    const double none[3] = {0, 0, 0};
                    double t[9], detA;
                    assemble_T3(X, ic, in, s, w, -1, none, t, detA);
                    Shared3<double> S3;
                    shared3<double>(KIND, t, 0.0, S3);
                    if constexpr (MODE == kCtlGrad) {
                        double gT[9];
                        mu3_grad<double>(KIND, S3, gT);
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            acc[i] += wt * (gT[3 * i] * v[0] + gT[3 * i + 1] * v[1] + gT[3 * i + 2] * v[2]);
                        }
                    } else if constexpr (MODE == kCtlHvp) {
                        // corr is net-node indexed: shift store slots into the net-node space
                        const int64_t sh = n.n_off - n.node_off;
                        const int32_t icn = int32_t(ic + sh);
                        const int32_t inn[3] = {int32_t(in[0] + sh), int32_t(in[1] + sh), int32_t(in[2] + sh)};
                        double dt[9], dd;
                        assemble_T3(corr, icn, inn, s, w, -1, none, dt, dd);
                        double hv[9];
                        mu3_hvp<double>(KIND, S3, dt, hv);
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            acc[i] += wt * (hv[3 * i] * v[0] + hv[3 * i + 1] * v[1] + hv[3 * i + 2] * v[2]);
                        }
                    } else {
                        double gg[3], h6[6];
                        role3<double>(KIND, S3, v, gg, h6);
                        const double hm[9] = {h6[0], h6[1], h6[2], h6[1], h6[3], h6[4], h6[2], h6[4], h6[5]};
#pragma unroll
                        for (int i = 0; i < 9; ++i) { acc[i] += wt * hm[i]; }
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < OUTW; ++i) { out[g * OUTW + i] = acc[i]; }
    }
}

// Tensor support of one control: per axis the CSR list of (node, weight).
template <int D> struct Support {
    const int32_t* node[3];
    const double* w[3];
    int len[3];
};

template <int D>
__device__ __forceinline__ Support<D> support_of(const CtlTables& T, const CtlNet& n, const int a[3])
{
    Support<D> sp;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int32_t* so = T.sup_off + n.sup_base[k];
        const int32_t b0 = so[a[k]], b1 = so[a[k] + 1];
        sp.node[k] = T.sup_node + b0;
        sp.w[k] = T.sup_w + b0;
        sp.len[k] = b1 - b0;
    }
    return sp;
}

// Free-control pullback out_f = sum_{n in supp(f)} w_n y_n (+ lam v_f), or the
// Jacobi block P_f = sum w_n^2 h_n (PRECOND).  A control's support is a box of
// a few hundred nodes.  WARP: its warp's lanes stride over the box, consecutive
// lanes along the last axis, and add up by butterfly; otherwise one thread
// adds in the reference's order, a serial chain of loads (257^2 block, 64^2
// net: 53 us against 7.5).  With many nets most are done while the last ones
// iterate; a warp finds which of its controls are left 32 at a time (256 nets,
// 822 k controls, few of them left: 19 us, 129 one control after another).
// Topologies and walled nets keep the serial
// order: their frames amplify a last bit (a sphere's chart near its pole,
// 7e7-fold), and their nets are small.
template <int D, bool PRECOND, bool WARP>
__global__ void ctl_pullback_kernel(CtlTables T, int64_t total_free, const double* __restrict__ y,
                                    double* __restrict__ out, const double* __restrict__ v,
                                    const PcgState* __restrict__ st)
{
    constexpr int W = PRECOND ? D * D : D, G = WARP ? 32 : 1;
    const int lane = threadIdx.x & (G - 1);
    const int64_t ngroup = (int64_t(gridDim.x) * blockDim.x) / G;
    const int64_t g0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G;
    auto active = [&](int64_t g, int& ni) {
        if (g >= total_free) { return false; }
        ni = net_of(T.free_pfx, T.n_nets, g);
        return PRECOND || st == nullptr || !st[ni].done;
    };
    auto pull = [&](int64_t g, int ni) {
        const CtlNet n = T.nets[ni];
        int a[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < D; ++k) { a[k] = T.free_midx[g * D + k]; }
        const Support<D> sp = support_of<D>(T, n, a);
        double acc[W];
#pragma unroll
        for (int i = 0; i < W; ++i) { acc[i] = 0.0; }
        const int ll = sp.len[D - 1], l1 = D == 3 ? sp.len[1] : 1;
        const int rows = sp.len[0] * l1;
        for (int e = lane; e < rows * ll; e += G) {
            const int row = e / ll, tl = e - row * ll;
            const int t0 = D == 3 ? row / l1 : row;
            double w = sp.w[0][t0];
            int64_t nd = sp.node[0][t0];
            if constexpr (D == 3) {
                w *= sp.w[1][row - t0 * l1];
                nd = nd * n.node_shape[1] + sp.node[1][row - t0 * l1];
            }
            w *= sp.w[D - 1][tl];
            nd = nd * n.node_shape[D - 1] + sp.node[D - 1][tl];
            const int64_t gn = n.n_off + nd;
            if (PRECOND) { w *= w; }
#pragma unroll
            for (int i = 0; i < W; ++i) { acc[i] += w * y[gn * W + i]; }
        }
#pragma unroll
        for (int i = 0; i < W; ++i) { acc[i] = group_sum<G>(acc[i]); }
        if (!PRECOND && st && st[ni].lam > 0.0) {
#pragma unroll
            for (int i = 0; i < W; ++i) { acc[i] += st[ni].lam * v[g * W + i]; }
        }
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < W; ++i) { out[g * W + i] = acc[i]; }
        }
    };
    int ni = 0;
    if constexpr (WARP) {
        // a warp's controls of 32 rounds at once: each lane looks one of them up
        for (int64_t b = g0; b < total_free; b += 32 * ngroup) {
            unsigned todo = __ballot_sync(0xffffffffu, active(b + lane * ngroup, ni));
            while (todo != 0u) {
                const int q = __ffs(int(todo)) - 1;
                todo &= todo - 1u;
                pull(b + q * ngroup, __shfl_sync(0xffffffffu, ni, q));
            }
        }
    } else {
        for (int64_t g = g0; g < total_free; g += ngroup) {
            if (active(g, ni)) { pull(g, ni); }
        }
    }
}

// z = (P_f + lam I)^{-1} r with the Newton-solve fallbacks (src/solve.hpp).
template <int D> __device__ __forceinline__ void ctl_precond(const double* P, double lam, const double r[D], double z[D])
{
    double rhs[3], x[3];
#pragma unroll
    for (int i = 0; i < D; ++i) { rhs[i] = -r[i]; }
    if constexpr (D == 2) {
        const double H[4] = {P[0] + lam, P[1], P[2], P[3] + lam};
        solve2<double>(H, rhs, x);
    } else {
        const double h6[6] = {P[0] + lam, P[1], P[2], P[4] + lam, P[5], P[8] + lam};
        solve3<double>(h6, rhs, x);
    }
#pragma unroll
    for (int i = 0; i < D; ++i) { z[i] = x[i]; }
}

// Per-net reductions over the stacked free vector (one CTA per net, fixed
// order, compensated).
enum {
    kRedAmax = 0,  // out[net] = max |x|
    kRedTrace,     // out[net] = sum of diagonals of the D x D blocks of x
};

template <int D, int OP>
__global__ void ctl_reduce_kernel(CtlTables T, const double* __restrict__ x, double* __restrict__ out)
{
    const int ni = blockIdx.x;
    Comp acc {0.0, 0.0};
    double mx = 0.0;
    for (int64_t g = T.free_pfx[ni] + threadIdx.x; g < T.free_pfx[ni + 1]; g += blockDim.x) {
#pragma unroll
        for (int i = 0; i < D; ++i) {
            if (OP == kRedAmax) {
                mx = fmax(mx, fabs(x[g * D + i]));
            } else {
                comp_add(acc, x[g * D * D + i * (D + 1)]);
            }
        }
    }
    // max via the min slot of the shared reducer
    double mn = -mx;
    if (!block_reduce(acc, mn)) { return; }
    out[ni] = OP == kRedAmax ? -mn : acc.s + acc.c;
}

// The vector part of a PCG iteration (src/control_solve.hpp:761-819): dot
// products, updates and preconditioner in one launch, a cluster of kCgCluster
// CTAs per net.  Each dot product is reduced per CTA, exchanged through
// distributed shared memory and added in rank order, so every thread holds the
// same total and takes the same decisions.  A CG iteration on a 64^2 net took
// 10 launches and 105 us (three one-CTA reductions among them), in one CTA of
// 512 threads 4 launches and 44 us, with the cluster 31.
constexpr int kCgCluster = 8;
constexpr int kCgThreads = 512;

struct CgShared {
    Comp part[3];
    double total[3];
};

// The cluster's totals of acc[0 .. N), exchange slots first .. first + N.
template <int N>
__device__ __forceinline__ void ctl_cluster_total(CgShared& sh, int first, const Comp (&acc)[N], double (&out)[N])
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
#pragma unroll
    for (int k = 0; k < N; ++k) {
        Comp a = acc[k];
        double mn = 0.0;
        if (block_reduce(a, mn)) { sh.part[first + k] = a; }
        __syncthreads();  // the reducer's storage is free again
    }
    cl.sync();
    if (threadIdx.x < N) {
        Comp t {0.0, 0.0};
        for (unsigned q = 0; q < unsigned(kCgCluster); ++q) {
            t = comp_merge(t, cl.map_shared_rank(&sh, q)->part[first + threadIdx.x]);
        }
        sh.total[first + threadIdx.x] = t.s + t.c;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) { out[k] = sh.total[first + k]; }
}

// Start: dC = 0, r = -G, z = P^{-1} r, p = z (also scattered to the lattice,
// Cdir), b.b, r.z; the net's relative tolerance arrives in stop2.
template <int D>
__global__ void __cluster_dims__(kCgCluster, 1, 1) __launch_bounds__(kCgThreads)
  ctl_cg_start_kernel(CtlTables T, const double* __restrict__ G, const double* __restrict__ prec,
                      double* __restrict__ dC, double* __restrict__ r, double* __restrict__ p,
                      double* __restrict__ Cdir, PcgState* __restrict__ st)
{
    __shared__ CgShared sh;
    const int ni = blockIdx.x / kCgCluster, rank = blockIdx.x % kCgCluster;
    PcgState& s = st[ni];
    const bool lead = rank == 0 && threadIdx.x == 0;
    if (!s.active) {  // uniform across the cluster
        if (lead) { s.done = 1; }
        return;
    }
    const double lam = s.lam, tol = s.stop2;
    const int max_iter = s.max_iter;
    const int64_t c_off = T.nets[ni].c_off;
    Comp acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int64_t g = T.free_pfx[ni] + rank * kCgThreads + threadIdx.x; g < T.free_pfx[ni + 1];
         g += kCgCluster * kCgThreads) {
        double rr[D], z[D];
#pragma unroll
        for (int i = 0; i < D; ++i) { rr[i] = -G[g * D + i]; }
        ctl_precond<D>(prec + g * D * D, lam, rr, z);
        const int64_t ci = c_off + T.free_idx[g];
#pragma unroll
        for (int i = 0; i < D; ++i) {
            dC[g * D + i] = 0.0;
            r[g * D + i] = rr[i];
            p[g * D + i] = z[i];
            Cdir[ci * D + i] = z[i];
            comp_add(acc[0], rr[i] * rr[i]);
            comp_add(acc[1], rr[i] * z[i]);
        }
    }
    double t[2];
    ctl_cluster_total<2>(sh, 0, acc, t);
    if (lead) {
        s.b_norm2 = t[0];
        s.r_norm2 = t[0];
        s.stop2 = tol * tol * t[0];
        s.rz = t[1];
        s.it = 0;
        s.its = 0;
        s.done = (t[0] == 0.0 || max_iter <= 0) ? 1 : 0;
    }
    cooperative_groups::this_cluster().sync();  // no CTA leaves while its partials are read
}

// One iteration after Ap: p.Ap (stop on non-positive curvature), dC += alpha p,
// r -= alpha Ap, r.r (stop at stop2), z = P^{-1} r, r.z, p = z + beta p.
template <int D>
__global__ void __cluster_dims__(kCgCluster, 1, 1) __launch_bounds__(kCgThreads)
  ctl_cg_step_kernel(CtlTables T, const double* __restrict__ prec, const double* __restrict__ Ap,
                     double* __restrict__ dC, double* __restrict__ r, double* __restrict__ z, double* __restrict__ p,
                     double* __restrict__ Cdir, PcgState* __restrict__ st)
{
    __shared__ CgShared sh;
    const int ni = blockIdx.x / kCgCluster, rank = blockIdx.x % kCgCluster;
    PcgState& s = st[ni];
    if (s.done) { return; }  // uniform: the lead thread writes it past two cluster barriers
    const bool lead = rank == 0 && threadIdx.x == 0;
    const double rz_old = s.rz, lam = s.lam, stop2 = s.stop2;
    const int it = s.it, max_iter = s.max_iter;
    const int64_t lo = T.free_pfx[ni] + rank * kCgThreads + threadIdx.x, hi = T.free_pfx[ni + 1];
    constexpr int64_t step = kCgCluster * kCgThreads;
    Comp pp[1] = {{0.0, 0.0}};
    for (int64_t g = lo; g < hi; g += step) {
#pragma unroll
        for (int i = 0; i < D; ++i) { comp_add(pp[0], p[g * D + i] * Ap[g * D + i]); }
    }
    double pap[1];
    ctl_cluster_total<1>(sh, 0, pp, pap);
    const bool down = !(pap[0] > 0.0);
    const double alpha = rz_old / pap[0];
    Comp acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
    if (!down) {
        for (int64_t g = lo; g < hi; g += step) {
            double rv[D], zv[D];
#pragma unroll
            for (int i = 0; i < D; ++i) {
                const int64_t e = g * D + i;
                dC[e] += alpha * p[e];
                rv[i] = r[e] - alpha * Ap[e];
                r[e] = rv[i];
                comp_add(acc[0], rv[i] * rv[i]);
            }
            ctl_precond<D>(prec + g * D * D, lam, rv, zv);
#pragma unroll
            for (int i = 0; i < D; ++i) {
                z[g * D + i] = zv[i];
                comp_add(acc[1], rv[i] * zv[i]);
            }
        }
    }
    double t[2];
    ctl_cluster_total<2>(sh, 1, acc, t);
    const bool small = t[0] <= stop2, last = it + 1 >= max_iter;
    if (lead) {
        if (down) {
            s.its = it;
            s.done = 1;
        } else {
            s.alpha = alpha;
            s.r_norm2 = t[0];
            if (!small) {
                s.beta = t[1] / rz_old;
                s.rz = t[1];
                s.it = it + 1;
            }
            if (small || last) {
                s.its = it + 1;
                s.done = 1;
            }
        }
    }
    if (!(down || small || last)) {
        const double beta = t[1] / rz_old;
        const int64_t c_off = T.nets[ni].c_off;
        for (int64_t g = lo; g < hi; g += step) {
            const int64_t ci = c_off + T.free_idx[g];
#pragma unroll
            for (int i = 0; i < D; ++i) {
                const double v = z[g * D + i] + beta * p[g * D + i];
                p[g * D + i] = v;
                Cdir[ci * D + i] = v;
            }
        }
    }
    cooperative_groups::this_cluster().sync();  // no CTA leaves while its partials are read
}

// Trial / commit on the net nodes: out[slot] = X[slot] + alpha[net] corr[node]
// (out may alias X for the commit).
template <int D>
__global__ void ctl_step_kernel(CtlTables T, int64_t total_nodes, const double* X, const double* __restrict__ corr,
                                const double* __restrict__ alpha, double* out)
{
    for (int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; g < total_nodes;
         g += int64_t(gridDim.x) * blockDim.x) {
        const int ni = net_of(T.node_pfx, T.n_nets, g);
        const double al = alpha[ni];
        if (al == 0.0) { continue; }
        const CtlNet n = T.nets[ni];
        const int64_t slot = n.node_off + (g - n.n_off);
#pragma unroll
        for (int c = 0; c < D; ++c) { out[slot * D + c] = X[slot * D + c] + al * corr[g * D + c]; }
    }
}

// C[lattice(free)] += alpha[net] dC[free].
template <int D>
__global__ void ctl_commit_c_kernel(CtlTables T, int64_t total_free, const double* __restrict__ dC,
                                    const double* __restrict__ alpha, double* __restrict__ C)
{
    for (int64_t g = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; g < total_free;
         g += int64_t(gridDim.x) * blockDim.x) {
        const int ni = net_of(T.free_pfx, T.n_nets, g);
        const double al = alpha[ni];
        if (al == 0.0) { continue; }
        const CtlNet n = T.nets[ni];
        const int64_t ci = n.c_off + T.free_idx[g];
#pragma unroll
        for (int c = 0; c < D; ++c) { C[ci * D + c] += al * dC[g * D + c]; }
    }
}

}  // namespace egg_b200
