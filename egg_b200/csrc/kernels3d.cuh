// 3D sweep kernels of the egg_b200 core (sm_100a).
//
// Store: blocks are dense row-major (n0, n1, n2) node arrays, three doubles
// per node, packed back to back (same conventions as the 2D store).
//
// interior3_kernel: one CTA = a TI x TJ x TK tile of structured-interior DOFs;
// the (TI+2)(TJ+2)(TK+2) node window is staged in shared memory (with its fp32
// forward edges in the mixed path) and each thread relaxes one DOF over its
// 64-occurrence patch (8 cells x 8 corner samples,
// src/structured_patch.hpp:89-258): dof3.cuh evaluates the 32 samples that
// move it, grouped by the edge that moves; the 32 that do not move it only
// rule a step out, from per-cell bits; then the 3x3 Newton step, <= 10 halvings
// on the moving samples, omega blend (src/sweep.hpp:1534-1650).
#pragma once

#include "dof3.cuh"
#include "entity3.cuh"
#include "kernels2d.cuh"
#include "metric3.cuh"

namespace egg_b200
{

struct Tile3 {
    int32_t block;
    int32_t i0, j0, k0;  // first DOF (logical, >= 1)
};

// Corner-index bit of axis k (axis 0 most significant).
__host__ __device__ constexpr int bit3(int k) { return 4 >> k; }

template <int TI, int TJ, int TK> struct Win3 {
    static constexpr int WI = TI + 2, WJ = TJ + 2, WK = TK + 2;
    static constexpr int N = WI * WJ * WK;
    static constexpr int S0 = WJ * WK, S1 = WK, S2 = 1;  // node strides of the axes
    static constexpr int NC = (WI - 1) * (WJ - 1) * (WK - 1);  // cells of the window
    __device__ static int idx(int u, int v, int w) { return (u * WJ + v) * WK + w; }
    __device__ static int cidx(int u, int v, int w) { return (u * (WJ - 1) + v) * (WK - 1) + w; }
};

template <int TI, int TJ, int TK> struct Tile3Shared {
    double P[3][Win3<TI, TJ, TK>::N];  // node window, SoA per coordinate
};

// Edge vectors of sample b of the cell whose base is window node (bu, bv, bw);
// node `a` of the cell may be replaced by `trial` (a < 0: no substitution).
// A[i][k] = s_k (X[nbr_k] - X[corner])_i, returned row-major in t[9] (fp64).
template <int TI, int TJ, int TK>
__device__ __forceinline__ void edges3(const Tile3Shared<TI, TJ, TK>& sm, int bu, int bv, int bw, int b, int a,
                                       const double trial[3], double t[9])
{
    using W = Win3<TI, TJ, TK>;
    auto node = [&](int c, double p[3]) {
        if (c == a) {
            p[0] = trial[0];
            p[1] = trial[1];
            p[2] = trial[2];
        } else {
            const int id = W::idx(bu + (c >> 2), bv + ((c >> 1) & 1), bw + (c & 1));
            p[0] = sm.P[0][id];
            p[1] = sm.P[1][id];
            p[2] = sm.P[2][id];
        }
    };
    double pc[3];
    node(b, pc);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double pn[3];
        node(b ^ bit3(k), pn);
        const double sk = (b & bit3(k)) ? -1.0 : 1.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) { t[3 * i + k] = sk * (pn[i] - pc[i]); }
    }
}

// Whether a corner sample of the cell with base window node n is inverted or
// badly shaped: det T <= 0 or det^2 < kBadCell^2 times its columns' squared
// lengths, from the window's fp32 forward edges fe[(3 k + i) N + node] =
// (X[node + e_k] - X[node])_i.  Sample b's columns are the cell's edges along
// axis k at the corner b without bit k, so the cell's 12 edges and their
// lengths are formed once, and the two samples along axis 2 share one
// instruction (a sample at a time from 9 loads each took 11% of the kernel).
template <class W> __device__ __forceinline__ bool cell_bad3(const float* __restrict__ fe, int n)
{
    using L = Lane<F2>;
    const EdgeF<W::N> E {fe};
    F2 e0[2][3], n0[2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        E.get(0, n + b * W::WK, n + b * W::WK + 1, e0[b]);
        n0[b] = dotv(e0[b], e0[b]);
    }
    bool bad = false;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int m = n + a * W::WJ * W::WK;
        F2 e1[3], m1[3];
        E.get(3 * W::N, m, m + 1, e1);
        negv(e1, m1);
        const F2 n1 = dotv(e1, e1);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            F2 e2[3], c[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) { e2[i] = L::set(fe[(6 + i) * W::N + m + b * W::WK]); }
            crossv(m1, e1, e0[b], c);  // e0 x e1
            const F2 D = dotv(e2, c), nn = n0[b] * n1 * dotv(e2, e2);
            const F2 t = vfma(D, D, L::set(-float(kBadCell * kBadCell)) * nn);
            bad = bad || !(D.v.x > 0.0f) || !(D.v.y > 0.0f) || t.v.x < 0.0f || t.v.y < 0.0f;
        }
    }
    return bad;
}

// fp64 metric change of one near-degenerate trial sample (cell base
// (bu, bv, bw), corner b, the DOF at corner a moved from pos by d), from the
// staged fp64 positions.  Out of line: it runs rarely and its fp64
// temporaries would otherwise weigh on the fp32 line search's registers.
template <int TI, int TJ, int TK, int KIND>
__device__ __noinline__ float dmu3_guard64(const Tile3Shared<TI, TJ, TK>& sm, int bu, int bv, int bw, int b, int a,
                                           const double pos[3], const double d[3], double delta, float& dn)
{
    const double none[3] = {0.0, 0.0, 0.0};
    const double trial[3] = {pos[0] + d[0], pos[1] + d[1], pos[2] + d[2]};
    double t0[9], t1[9], d0, d1;
    edges3<TI, TJ, TK>(sm, bu, bv, bw, b, -1, none, t0);
    edges3<TI, TJ, TK>(sm, bu, bv, bw, b, a, trial, t1);
    const double m0 = mu3_value<double>(KIND, t0, delta, d0);
    const double m1 = mu3_value<double>(KIND, t1, delta, d1);
    dn = d1 > 0.0 ? fmaxf(float(d1), 1e-38f) : (d1 < 0.0 ? fminf(float(d1), -1e-38f) : 0.0f);
    return float(m1 - m0);
}

// Whether one corner sample admits a move of the DOFs that do not move it:
// its metric is finite and, outside the untangle phase, its det positive.
template <int KIND> __device__ __forceinline__ bool sample_ok64(const double t[9], double delta)
{
    const double c0 = t[4] * t[8] - t[5] * t[7], c1 = t[5] * t[6] - t[3] * t[8], c2 = t[3] * t[7] - t[4] * t[6];
    const double D = t[0] * c0 + t[1] * c1 + t[2] * c2;
    if constexpr (KIND != kUntangle) {
        if (!(D > 0.0)) { return false; }
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) { s += t[k] * t[k]; }
        // q <= s^2 / 3, so the metric cannot overflow here
        if (s < 1e100 && D * D > 1e-280 * (s * s * s)) { return true; }
    }
    double d;
    return isfinite(mu3_value<double>(KIND, t, delta, d));
}

// Bit b set: sample b of the cell with base node n of window P fails
// sample_ok64.
template <class W, int KIND> __device__ __forceinline__ unsigned cell_stop64(const double* P, int n, double delta)
{
    const int st[3] = {W::S0, W::S1, W::S2};
    unsigned mask = 0u;
#pragma unroll 2
    for (int b = 0; b < 8; ++b) {
        const int at = n + ((b & 4) ? W::S0 : 0) + ((b & 2) ? W::S1 : 0) + ((b & 1) ? W::S2 : 0);
        double t[9];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int lo = (b & bit3(k)) ? at - st[k] : at;
#pragma unroll
            for (int i = 0; i < 3; ++i) { t[3 * i + k] = P[i * W::N + lo + st[k]] - P[i * W::N + lo]; }
        }
        if (!sample_ok64<KIND>(t, delta)) { mask |= 1u << b; }
    }
    return mask;
}

// The samples of a cell that do not move its corner a, as bits of cell_stop64.
__device__ __forceinline__ constexpr unsigned still_bits(int a)
{
    return (1u << (a ^ 7)) | (1u << (a ^ 6)) | (1u << (a ^ 5)) | (1u << (a ^ 3));
}

// fp64 update (or, grad_only, gradient) of the DOF at node p of window P, by
// its NH threads (dof3_system).  `stop`: a sample around it that it does not
// move rules every step out.  The accept test compares the energies of the 32
// samples it moves; the other 32 add the same constant to both sides.
template <class W, int KIND, int NH>
__device__ __forceinline__ void dof3_fp64(const double* P, int p, int half, bool stop, const double tau[3],
                                          double delta, double omega, double out[3], bool grad_only)
{
    const EdgeD<W::N> E {P};
    double g[3], h[6], e0;
    if (grad_only) {
        dof3_system<W, KIND, NH, true>(E, p, half, delta, g, h, e0);
#pragma unroll
        for (int q = 0; q < 3; ++q) { out[q] = g[q] - tau[q]; }
        return;
    }
    dof3_system<W, KIND, NH, false>(E, p, half, delta, g, h, e0);
#pragma unroll
    for (int q = 0; q < 3; ++q) { g[q] -= tau[q]; }
#pragma unroll
    for (int q = 0; q < 3; ++q) { out[q] = P[q * W::N + p]; }
    if (stop) { return; }
    double dl[3];
    solve3<double>(h, g, dl);
    double alpha = 1.0;
#pragma unroll 1
    for (int it = 0; it < 10; ++it) {
        const double d[3] = {alpha * dl[0], alpha * dl[1], alpha * dl[2]};
        double md = INFINITY;
        const double e =
          dof3_trial<W, KIND, NH>(E, p, half, d, delta, md) - (tau[0] * d[0] + tau[1] * d[1] + tau[2] * d[2]);
        md = pair_min<NH>(md);
        if (isfinite(e) && e <= e0 + Tol<double>::energy && (KIND == kUntangle || md > 0.0)) {
#pragma unroll
            for (int q = 0; q < 3; ++q) { out[q] += omega * d[q]; }
            return;
        }
        alpha *= 0.5;
    }
}

// The mixed path's DOFs next to an inverted or badly shaped sample: fp64, out
// of line so that its registers do not weigh on the fp32 path.
template <int TI, int TJ, int TK, int KIND>
__device__ __noinline__ void dof3_fallback64(const Tile3Shared<TI, TJ, TK>& sm, int ti, int tj, int tk,
                                             const double tau[3], double delta, double omega, double out[3],
                                             bool grad_only)
{
    using W = Win3<TI, TJ, TK>;
    bool stop = false;
#pragma unroll 1
    for (int cell = 0; cell < 8 && !grad_only; ++cell) {
        const int n = W::idx(ti + (cell >> 2), tj + ((cell >> 1) & 1), tk + (cell & 1));
        stop = stop || (cell_stop64<W, KIND>(&sm.P[0][0], n, delta) & still_bits(7 - cell)) != 0u;
    }
    dof3_fp64<W, KIND, 1>(&sm.P[0][0], W::idx(ti + 1, tj + 1, tk + 1), 0, stop, tau, delta, omega, out, grad_only);
}

// The line search's pass over near-degenerate trial samples, out of line: the
// fp32 sum without them plus their changes differenced in fp64.
template <int TI, int TJ, int TK, int KIND>
__device__ __noinline__ float dof3_line_guard(const Tile3Shared<TI, TJ, TK>& sm, const float* __restrict__ fe, int ti,
                                              int tj, int tk, const float d[3], double delta, float& md)
{
    using W = Win3<TI, TJ, TK>;
    const EdgeF<W::N> E {fe};
    const int p = W::idx(ti + 1, tj + 1, tk + 1);
    float low = 0.0f, add = 0.0f;
    unsigned guard = 0u;
    md = INFINITY;
    const float ds = dof3_line<W, KIND, true>(E, p, d, float(delta), md, low, guard);
    const double pos[3] = {sm.P[0][p], sm.P[1][p], sm.P[2][p]};
    const double d3[3] = {double(d[0]), double(d[1]), double(d[2])};
    while (guard != 0u) {
        const int bit = __ffs(int(guard)) - 1;
        guard &= guard - 1u;
        const int cell = bit & 7, r = bit >> 3, a = 7 - cell, b = r == 0 ? a : (a ^ bit3(r - 1));
        float dn;
        add += dmu3_guard64<TI, TJ, TK, KIND>(sm, ti + (cell >> 2), tj + ((cell >> 1) & 1), tk + (cell & 1), b, a,
                                              pos, d3, delta, dn);
        md = fminf(md, dn);
    }
    return ds + add;
}

// fp32 update (or gradient) of a DOF whose 8 cells hold no bad sample: the
// samples that it does not move then have positive dets, and the accept test
// sums metric changes, with the fp64 energy tolerance.  Near-degenerate trial
// samples are differenced in fp64.
template <int TI, int TJ, int TK, int KIND>
__device__ __forceinline__ void dof3_fp32(const Tile3Shared<TI, TJ, TK>& sm, const float* __restrict__ fe, int ti,
                                          int tj, int tk, const double tau[3], double delta, double omega,
                                          double out[3], bool grad_only)
{
    using W = Win3<TI, TJ, TK>;
    const EdgeF<W::N> E {fe};
    const int p = W::idx(ti + 1, tj + 1, tk + 1);
    const float fd = float(delta);
    float g[3], h[6];
    const float ft[3] = {float(tau[0]), float(tau[1]), float(tau[2])};
    if (grad_only) {
        dof3_system<W, KIND, true>(E, p, fd, g, h);
#pragma unroll
        for (int q = 0; q < 3; ++q) { out[q] = double(g[q] - ft[q]); }
        return;
    }
    dof3_system<W, KIND, false>(E, p, fd, g, h);
#pragma unroll
    for (int q = 0; q < 3; ++q) { g[q] -= ft[q]; }
    float dl[3];
    solve3<float>(h, g, dl);
    float alpha = 1.0f;
#pragma unroll 1
    for (int it = 0; it < 10; ++it) {
        const float d[3] = {alpha * dl[0], alpha * dl[1], alpha * dl[2]};
        float md = INFINITY, low = INFINITY;
        unsigned none_guard = 0u;
        float ds = dof3_line<W, KIND, false>(E, p, d, fd, md, low, none_guard);
        if (!(low > 0.0f) || !isfinite(ds)) {
            ds = dof3_line_guard<TI, TJ, TK, KIND>(sm, fe, ti, tj, tk, d, delta, md);
        }
        ds -= ft[0] * d[0] + ft[1] * d[1] + ft[2] * d[2];
        if (isfinite(ds) && ds <= float(Tol<double>::energy) && (KIND == kUntangle || md > 0.0f)) {
#pragma unroll
            for (int q = 0; q < 3; ++q) { out[q] = sm.P[q][p] + omega * double(d[q]); }
            return;
        }
        alpha *= 0.5f;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) { out[q] = sm.P[q][p]; }
}

template <int TI, int TJ, int TK, int MINB, int KIND, class C>
__global__ void __launch_bounds__(TI* TJ* TK, MINB)
  interior3_kernel(const double* __restrict__ Xin, double* __restrict__ Xout, const Tile3* __restrict__ tiles,
                   const BlockInfo* __restrict__ blocks, const uint8_t* __restrict__ active,
                   const double* __restrict__ tau, double delta, double omega, double* __restrict__ grad_out)
{
    using W = Win3<TI, TJ, TK>;
    __shared__ Tile3Shared<TI, TJ, TK> sm;
    __shared__ float fe[std::is_same_v<C, float> ? 9 * W::N : 1];  // fp32 forward edges (mixed)
    __shared__ uint8_t cbad[W::NC];  // per window cell: bad-sample bits (mixed), stop bits (fp64)
    const Tile3 tile = tiles[blockIdx.x];
    const BlockInfo bi = blocks[tile.block];
    const int n0 = bi.n[0], n1 = bi.n[1], n2 = bi.n[2];
    const int u0 = tile.i0 - 1, v0 = tile.j0 - 1, w0 = tile.k0 - 1;
    constexpr int NT = TI * TJ * TK;
    for (int id = threadIdx.x; id < W::N; id += NT) {
        const int u = id / (W::WJ * W::WK), v = (id / W::WK) % W::WJ, w = id % W::WK;
        const int gi = u0 + u, gj = v0 + v, gk = w0 + w;
        double p0 = 0.0, p1 = 0.0, p2 = 0.0;
        if (gi < n0 && gj < n1 && gk < n2) {
            const int64_t node = bi.off + (int64_t(gi) * n1 + gj) * n2 + gk;
            p0 = Xin[3 * node];
            p1 = Xin[3 * node + 1];
            p2 = Xin[3 * node + 2];
        }
        sm.P[0][id] = p0;
        sm.P[1][id] = p1;
        sm.P[2][id] = p2;
    }
    __syncthreads();
    if constexpr (std::is_same_v<C, float>) {
        // forward edge along k of every window node that has a +k neighbour
        for (int id = threadIdx.x; id < W::N; id += NT) {
            const int cu = id / (W::WJ * W::WK), cv = (id / W::WK) % W::WJ, cw = id % W::WK;
            const bool has[3] = {cu + 1 < W::WI, cv + 1 < W::WJ, cw + 1 < W::WK};
            const int step[3] = {W::WJ * W::WK, W::WK, 1};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    fe[(3 * k + i) * W::N + id] = has[k] ? float(sm.P[i][id + step[k]] - sm.P[i][id]) : 0.0f;
                }
            }
        }
        __syncthreads();
        // each window cell's 8 samples checked once for the whole tile (a
        // DOF's patch covers all 8 samples of its 8 cells); cells reaching
        // past the block hold zero positions and are read by no DOF
        for (int c = threadIdx.x; c < W::NC; c += NT) {
            const int cu = c / ((W::WJ - 1) * (W::WK - 1)), cv = (c / (W::WK - 1)) % (W::WJ - 1), cw = c % (W::WK - 1);
            cbad[c] = cell_bad3<W>(fe, W::idx(cu, cv, cw)) ? 1 : 0;
        }
    } else {
        for (int c = threadIdx.x; c < W::NC; c += NT) {
            const int cu = c / ((W::WJ - 1) * (W::WK - 1)), cv = (c / (W::WK - 1)) % (W::WJ - 1), cw = c % (W::WK - 1);
            cbad[c] = uint8_t(cell_stop64<W, KIND>(&sm.P[0][0], W::idx(cu, cv, cw), delta));
        }
    }
    __syncthreads();
    const int ti = threadIdx.x / (TJ * TK), tj = (threadIdx.x / TK) % TJ, tk = threadIdx.x % TK;
    const int gi = tile.i0 + ti, gj = tile.j0 + tj, gk = tile.k0 + tk;
    if (gi > n0 - 2 || gj > n1 - 2 || gk > n2 - 2) { return; }
    const int64_t slot = bi.off + (int64_t(gi) * n1 + gj) * n2 + gk;
    if (!active[slot]) { return; }
    double tv[3] = {0.0, 0.0, 0.0};
    if (tau != nullptr) {
        tv[0] = tau[3 * slot];
        tv[1] = tau[3 * slot + 1];
        tv[2] = tau[3 * slot + 2];
    }
    double out[3];
    const bool go = grad_out != nullptr;
    unsigned bad = 0u;
#pragma unroll
    for (int cell = 0; cell < 8; ++cell) {
        const unsigned m = cbad[W::cidx(ti + (cell >> 2), tj + ((cell >> 1) & 1), tk + (cell & 1))];
        bad |= std::is_same_v<C, float> ? m : m & still_bits(7 - cell);
    }
    if constexpr (std::is_same_v<C, double>) {
        dof3_fp64<W, KIND, 1>(&sm.P[0][0], W::idx(ti + 1, tj + 1, tk + 1), 0, bad != 0u, tv, delta, omega, out, go);
    } else if (bad != 0u) {
        dof3_fallback64<TI, TJ, TK, KIND>(sm, ti, tj, tk, tv, delta, omega, out, go);
    } else {
        dof3_fp32<TI, TJ, TK, KIND>(sm, fe, ti, tj, tk, tv, delta, omega, out, go);
    }
    double* dst = go ? grad_out : Xout;
    dst[3 * slot] = out[0];
    dst[3 * slot + 1] = out[1];
    dst[3 * slot + 2] = out[2];
}

// ---------------------------------------------------------------------------
// Stored-patch sweep, 3D (fp64, general W_inv).
// ---------------------------------------------------------------------------
struct StoredPatch3 {
    int64_t n;
    const int32_t* slot;
    const int64_t* off;
    const int32_t* gc;
    const int32_t* gn0;
    const int32_t* gn1;
    const int32_t* gn2;
    const int8_t* s0;
    const int8_t* s1;
    const int8_t* s2;
    const int32_t* role;
    const double* W;  // [occ*9] or [9]
    int32_t w_stride;
    const double* wt;
    int32_t wt_stride;
    const int8_t* etag;  // [n] entity tag of each DOF, or NULL (all Free)
    const double* epar;  // [n * EGG_B200_ENTITY_FIELDS] entity records
    int cold;            // first sweep of a run call: parametric entities project in world space
    SoftTable soft;      // directional terms per DOF (off == NULL: none)
    const double* arena; // entity arena (B-spline surfaces)
    double* seeds;       // [n * 2] last foot parameter of each B-spline-surface DOF (NaN: none)
    Copies copies;
};

__device__ __forceinline__ void assemble_T3(const double* X, int32_t ic, const int32_t in[3], const double s[3],
                                            const double* w, int32_t dslot, const double tr[3], double t[9],
                                            double& detA)
{
    auto ld = [&](int32_t n, double p[3]) {
        if (n == dslot) {
            p[0] = tr[0];
            p[1] = tr[1];
            p[2] = tr[2];
        } else {
            p[0] = X[3 * int64_t(n)];
            p[1] = X[3 * int64_t(n) + 1];
            p[2] = X[3 * int64_t(n) + 2];
        }
    };
    double c[3], A[9];
    ld(ic, c);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double p[3];
        ld(in[k], p);
#pragma unroll
        for (int i = 0; i < 3; ++i) { A[3 * i + k] = s[k] * (p[i] - c[i]); }
    }
    detA = det3(A);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            t[3 * i + k] = A[3 * i] * w[k] + A[3 * i + 1] * w[3 + k] + A[3 * i + 2] * w[6 + k];
        }
    }
}

// Stored DOFs whose patch is a plain 3 x 3 x 3 lattice with identity target
// and unit weight: nodes off every block edge where two blocks meet (and, on
// the FAS levels, the same nodes).  Blocks may be turned against one another;
// the table lists each DOF's 27 node slots in one right-handed order of its
// own, so the structured update applies (dof3_fp64, two threads per DOF)
// instead of 64 gathered samples with a general target.
struct Lattice3 {
    int64_t n;            // DOFs
    const int32_t* node;  // [27][n] node slots, entry 13 the DOF
    Copies copies;
};
constexpr int kLatDofs = 64;  // DOFs per CTA of 2 kLatDofs threads
struct WinLat3 {
    static constexpr int N = 27 * kLatDofs, S0 = 9 * kLatDofs, S1 = 3 * kLatDofs, S2 = kLatDofs;
};

template <int KIND>
__device__ __noinline__ void lattice3_cta(double* P, Lattice3 lat, int64_t d0, const double* __restrict__ Xin,
                                          double* __restrict__ Xout, const double* __restrict__ tau, double delta,
                                          double omega, double* __restrict__ grad_out)
{
    using W = WinLat3;
    for (int i = threadIdx.x; i < W::N; i += 2 * kLatDofs) {
        const int64_t d = d0 + i % kLatDofs;
        if (d >= lat.n) { continue; }
        const int64_t s = lat.node[(i / kLatDofs) * lat.n + d];
#pragma unroll
        for (int q = 0; q < 3; ++q) { P[q * W::N + i] = Xin[3 * s + q]; }
    }
    __syncthreads();
    const int t = threadIdx.x >> 1, half = threadIdx.x & 1, p = 13 * kLatDofs + t;
    const int64_t d = d0 + t;
    if (d >= lat.n) { return; }
    const int64_t slot = lat.node[13 * lat.n + d];
    const bool go = grad_out != nullptr;
    double tv[3] = {0.0, 0.0, 0.0}, out[3];
    if (tau != nullptr) {
#pragma unroll
        for (int q = 0; q < 3; ++q) { tv[q] = tau[3 * slot + q]; }
    }
    unsigned stop = 0u;
#pragma unroll 1
    for (int c = 0; c < 4 && !go; ++c) {
        const int cell = 4 * half + c;
        const int n = p + ((cell & 4) ? 0 : -W::S0) + ((cell & 2) ? 0 : -W::S1) + ((cell & 1) ? 0 : -W::S2);
        stop |= cell_stop64<W, KIND>(P, n, delta) & still_bits(7 - cell);
    }
    stop |= __shfl_xor_sync(pair_mask(), stop, 1, 2);
    dof3_fp64<W, KIND, 2>(P, p, half, stop != 0u, tv, delta, omega, out, go);
    if (half) { return; }
    double* dst = go ? grad_out : Xout;
#pragma unroll
    for (int q = 0; q < 3; ++q) { dst[3 * slot + q] = out[q]; }
    if (!go && lat.copies.off != nullptr) {
        for (int32_t c = lat.copies.off[d]; c < lat.copies.off[d + 1]; ++c) {
            for (int q = 0; q < 3; ++q) { Xout[3 * int64_t(lat.copies.dst[c]) + q] = out[q]; }
        }
    }
}

// Stored-patch sweep, 3D, G lanes per DOF (see stored_patch_kernel): the
// lanes split the DOF's samples and reduce across the group.  CLS says what is
// compiled in: 0 general patches alone, 1 lattice DOFs too, 2 constrained DOFs
// too.  The first `nb` CTAs take the stored DOFs, the others the lattice DOFs.
//
// The lattice part takes a kernel without entity code from 124 to 158
// registers, 4 to 3 CTAs per SM (with entities it is 236 either way): levels
// without lattice DOFs, such as every DOF of a target that is no multiple of
// the identity, launch class 0 (65^3 cube, general target: 700 us a sweep,
// 775 with one class for both).
template <int KIND, int G, int CLS>
__global__ void stored3_kernel(StoredPatch3 sp, int nb, Lattice3 lat, const double* __restrict__ Xin,
                               double* __restrict__ Xout, const double* __restrict__ tau, double delta, double omega,
                               double* __restrict__ grad_out)
{
    constexpr bool CON = CLS == 2;
    if constexpr (CLS > 0) {
        if (int(blockIdx.x) >= nb) {
            extern __shared__ __align__(16) unsigned char lat_smem[];
            lattice3_cta<KIND>(reinterpret_cast<double*>(lat_smem), lat, int64_t(blockIdx.x - nb) * kLatDofs, Xin,
                               Xout, tau, delta, omega, grad_out);
            return;
        }
    }
    const int lane = threadIdx.x & (G - 1);
    const int64_t ngroups = (int64_t(nb) * blockDim.x) / G;
    const double none[3] = {0, 0, 0};
    for (int64_t d = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G; d < sp.n; d += ngroups) {
        const int32_t slot = sp.slot[d];
        const double pos[3] = {Xin[3 * int64_t(slot)], Xin[3 * int64_t(slot) + 1], Xin[3 * int64_t(slot) + 2]};
        const int64_t p0 = sp.off[d], p1 = sp.off[d + 1];
        double g[3] = {0, 0, 0}, h[6] = {0, 0, 0, 0, 0, 0}, e0 = 0.0;
        for (int64_t p = p0 + lane; p < p1; p += G) {
            const double* w = sp.W + p * sp.w_stride;
            const double s[3] = {double(sp.s0[p]), double(sp.s1[p]), double(sp.s2[p])};
            const int32_t in[3] = {sp.gn0[p], sp.gn1[p], sp.gn2[p]};
            double t[9], detA;
            assemble_T3(Xin, sp.gc[p], in, s, w, -1, none, t, detA);
            Shared3<double> S;
            shared3<double>(KIND, t, delta, S);
            const double wt = sp.wt[p * sp.wt_stride];
            e0 += wt * mu3_from<double>(KIND, S);
            const int role = sp.role[p];
            if (role < 0) { continue; }
            double v[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v[c] = role == 0 ? -(s[0] * w[c] + s[1] * w[3 + c] + s[2] * w[6 + c]) : s[role - 1] * w[3 * (role - 1) + c];
            }
            double gg[3], hh[6];
            role3<double>(KIND, S, v, gg, hh);
#pragma unroll
            for (int q = 0; q < 3; ++q) { g[q] += wt * gg[q]; }
#pragma unroll
            for (int q = 0; q < 6; ++q) { h[q] += wt * hh[q]; }
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) { g[q] = group_sum<G>(g[q]); }
#pragma unroll
        for (int q = 0; q < 6; ++q) { h[q] = group_sum<G>(h[q]); }
        e0 = group_sum<G>(e0);
        // Directional soft terms (src/sweep.hpp:1307-1327,1491-1512), added
        // entry by entry to the full 3x3 Hessian.
        const int etag = (CON && sp.etag != nullptr) ? int(sp.etag[d]) : 0;
        if (sp.soft.off != nullptr) {
            double H9[9] = {h[0], h[1], h[2], h[1], h[3], h[4], h[2], h[4], h[5]};
            soft_dof_accumulate<3>(sp.soft, d, false, Xin, g, H9, e0);
            h[0] = H9[0];
            h[1] = H9[1];
            h[2] = H9[2];
            h[3] = H9[4];
            h[4] = H9[5];
            h[5] = H9[8];
        }
        double tv[3] = {0, 0, 0};
        if (tau != nullptr) {
            for (int q = 0; q < 3; ++q) { tv[q] = tau[3 * int64_t(slot) + q]; }
            for (int q = 0; q < 3; ++q) {
                g[q] -= tv[q];
                e0 -= tv[q] * pos[q];
            }
        }
        if (grad_out != nullptr) {
            if (lane == 0) {
                for (int q = 0; q < 3; ++q) { grad_out[3 * int64_t(slot) + q] = g[q]; }
            }
            continue;
        }
        // Constrained DOFs (src/sweep.hpp:1286-1403, 1718-1876): the step on
        // the entity's tangent space, damped by omega before the line
        // search, every trial on the entity; a parametric entity after the
        // first sweep of a run call searches in its parameters.
        const double* er = sp.epar + (etag != 0 ? d * EGG_B200_ENTITY_FIELDS : 0);
        // A B-spline surface carries its foot parameter from sweep to sweep
        // (src/sweep.hpp:1221-1265): the first sweep of a run call steps on
        // the seeded foot's frame and projects every trial from the seed,
        // which each projection advances; later sweeps search in its
        // parameters, every trial clamped onto the trim polygon
        // (src/sweep.hpp:1820-1832: the clamp applies inside the trim too).
        const bool bsurf = etag == EGG_B200_TAG_BSPLINESURF;
        double seed[2] = {NAN, NAN};
        if (bsurf) {
            seed[0] = sp.seeds[2 * d];
            seed[1] = sp.seeds[2 * d + 1];
        }
        const bool warm_param = (is_param3(etag) || (bsurf && isfinite(seed[0]))) && !sp.cold;
        double dl[3] = {0.0, 0.0, 0.0};
        double qs[2] = {0.0, 0.0}, dq[2] = {0.0, 0.0};
        if (etag == 0) {
            solve3<double>(h, g, dl);
        } else if (bsurf && warm_param) {
            bsurf_dof(kBsurfWarm, er, sp.arena, h, g, pos, omega, 0.0, seed, qs, dq, nullptr, nullptr);
        } else if (bsurf) {
            bsurf_dof(kBsurfCold, er, sp.arena, h, g, pos, omega, 0.0, seed, qs, dq, dl, nullptr);
            for (int q = 0; q < 3; ++q) { dl[q] *= omega; }
        } else if (warm_param) {
            param3_warm_step(etag, er, h, g, pos, omega, qs, dq);
        } else {
            entity3_newton_step(etag, er, h, g, pos, dl);
            for (int q = 0; q < 3; ++q) { dl[q] *= omega; }
        }
        double alpha = 1.0;
        double cur[3] = {pos[0], pos[1], pos[2]};
        for (int it = 0; it < 10; ++it) {
            double tr[3] = {pos[0] + alpha * dl[0], pos[1] + alpha * dl[1], pos[2] + alpha * dl[2]};
            if (bsurf) {
                bsurf_dof(warm_param ? kBsurfWarmTrial : kBsurfColdTrial, er, sp.arena, h, g, pos, omega, alpha,
                          seed, qs, dq, tr, nullptr);
            } else if (warm_param) {
                double qt[2] = {qs[0] + alpha * dq[0], qs[1] + alpha * dq[1]};
                p3_clamp(etag, er, qt);
                p3_eval(etag, er, qt, tr);
            } else if (etag != 0) {
                const double raw[3] = {tr[0], tr[1], tr[2]};
                entity3_project(etag, er, raw, tr);
            }
            double e = 0.0, md = INFINITY;
            for (int64_t p = p0 + lane; p < p1; p += G) {
                const double s[3] = {double(sp.s0[p]), double(sp.s1[p]), double(sp.s2[p])};
                const int32_t in[3] = {sp.gn0[p], sp.gn1[p], sp.gn2[p]};
                double t[9], detA;
                assemble_T3(Xin, sp.gc[p], in, s, sp.W + p * sp.w_stride, slot, tr, t, detA);
                double dd;
                e += sp.wt[p * sp.wt_stride] * mu3_value<double>(KIND, t, delta, dd);
                md = fmin(md, detA);
            }
            e = group_sum<G>(e);
            if (sp.soft.off != nullptr) { e += soft_dof_trial<3>(sp.soft, d, false, Xin, tr); }
            e -= tv[0] * tr[0] + tv[1] * tr[1] + tv[2] * tr[2];
            md = group_min<G>(md);
            if (isfinite(e) && e <= e0 + Tol<double>::energy && (KIND == kUntangle || md > 0.0)) {
                cur[0] = tr[0];
                cur[1] = tr[1];
                cur[2] = tr[2];
                break;
            }
            alpha *= 0.5;
        }
        if (lane == 0) {
            for (int q = 0; q < 3; ++q) {
                cur[q] = etag != 0 ? cur[q] : pos[q] + omega * (cur[q] - pos[q]);
                Xout[3 * int64_t(slot) + q] = cur[q];
            }
            if (sp.copies.off != nullptr) {
                for (int32_t c = sp.copies.off[d]; c < sp.copies.off[d + 1]; ++c) {
                    for (int q = 0; q < 3; ++q) { Xout[3 * int64_t(sp.copies.dst[c]) + q] = cur[q]; }
                }
            }
            if (bsurf) {
                sp.seeds[2 * d] = seed[0];
                sp.seeds[2 * d + 1] = seed[1];
            }
        }
    }
}

// Owner -> non-owner copy refresh, three doubles per node.
__global__ void broadcast3_kernel(double* __restrict__ X, const int32_t* __restrict__ src,
                                  const int32_t* __restrict__ dst, int64_t n)
{
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n; e += int64_t(gridDim.x) * blockDim.x) {
        const int64_t s = 3 * int64_t(src[e]), d = 3 * int64_t(dst[e]);
        X[d] = X[s];
        X[d + 1] = X[s + 1];
        X[d + 2] = X[s + 2];
    }
}

// Energy / min det over the canonical cell stencil of the blocks (3D).
template <int KIND>
__global__ void energy_structured3_kernel(EnergyStructured2 es, const double* __restrict__ X, double delta,
                                          double* part_s, double* part_c, double* part_m, ReduceOut out = {})
{
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    int64_t c_lo, c_hi;
    segment_range(es.seg, es.ncell, c_lo, c_hi);
    for (int64_t c = c_lo + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; c < c_hi;
         c += int64_t(gridDim.x) * blockDim.x) {
        int lo = 0, hi = es.nblocks - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (es.cell_off[mid] <= c) {
                lo = mid;
            } else {
                hi = mid - 1;
            }
        }
        const BlockInfo bi = es.blocks[lo];
        const uint32_t lc = uint32_t(c - es.cell_off[lo]);  // a store holds < 2^31 nodes
        const uint32_t c1 = uint32_t(bi.n[1] - 1), c2 = uint32_t(bi.n[2] - 1), ij = lc / c2;
        const int i = int(ij / c1), j = int(ij % c1), k = int(lc % c2);
        const int32_t base = int32_t(bi.off + (int64_t(i) * bi.n[1] + j) * bi.n[2] + k);
        int32_t nd[8];
#pragma unroll
        for (int a = 0; a < 8; ++a) { nd[a] = base + ((a >> 2) * bi.n[1] + ((a >> 1) & 1)) * bi.n[2] + (a & 1); }
        const double none[3] = {0, 0, 0};
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int64_t sid = c * 8 + b;
            const double s[3] = {(b & 4) ? -1.0 : 1.0, (b & 2) ? -1.0 : 1.0, (b & 1) ? -1.0 : 1.0};
            const int32_t in[3] = {nd[b ^ 4], nd[b ^ 2], nd[b ^ 1]};
            double t[9], detA;
            assemble_T3(X, nd[b], in, s, es.W + sid * es.w_stride, -1, none, t, detA);
            double dd;
            comp_add(acc, es.wt[sid * es.wt_stride] * mu3_value<double>(KIND, t, delta, dd));
            mn = fmin(mn, detA);
        }
    }
    block_reduce_store(acc, mn, part_s, part_c, part_m, out);
}

struct EnergyStored3 {
    int64_t n;
    const int32_t* gc;
    const int32_t* gn0;
    const int32_t* gn1;
    const int32_t* gn2;
    const int8_t* s0;
    const int8_t* s1;
    const int8_t* s2;
    const double* W;
    int32_t w_stride;
    const double* wt;
    int32_t wt_stride;
    const int64_t* seg = nullptr;  // per-mesh sample prefix offsets or null
};

template <int KIND>
__global__ void energy_stored3_kernel(EnergyStored3 es, const double* __restrict__ X, double delta, double* part_s,
                                      double* part_c, double* part_m, ReduceOut out = {})
{
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    const double none[3] = {0, 0, 0};
    int64_t i_lo, i_hi;
    segment_range(es.seg, es.n, i_lo, i_hi);
    for (int64_t i = i_lo + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < i_hi;
         i += int64_t(gridDim.x) * blockDim.x) {
        const double s[3] = {double(es.s0[i]), double(es.s1[i]), double(es.s2[i])};
        const int32_t in[3] = {es.gn0[i], es.gn1[i], es.gn2[i]};
        double t[9], detA;
        assemble_T3(X, es.gc[i], in, s, es.W + i * es.w_stride, -1, none, t, detA);
        double dd;
        comp_add(acc, es.wt[i * es.wt_stride] * mu3_value<double>(KIND, t, delta, dd));
        mn = fmin(mn, detA);
    }
    block_reduce_store(acc, mn, part_s, part_c, part_m, out);
}

// Device metric probe (tests): mu, gradient over vec(T) (9) and the contracted
// Hessian along e_i v^T (6) for n (t, v) pairs.
__global__ void metric3_probe_kernel(int kind, double delta, const double* t, const double* v, int64_t n,
                                     double* mu, double* g9, double* hv)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) { return; }
    Shared3<double> S;
    shared3<double>(kind, t + 9 * i, delta, S);
    mu[i] = mu3_from<double>(kind, S);
    for (int c = 0; c < 3; ++c) {
        const double e[3] = {c == 0 ? 1.0 : 0.0, c == 1 ? 1.0 : 0.0, c == 2 ? 1.0 : 0.0};
        double gg[3], hh[6];
        role3<double>(kind, S, e, gg, hh);
        for (int r = 0; r < 3; ++r) { g9[9 * i + 3 * r + c] = gg[r]; }
    }
    double gg[3];
    role3<double>(kind, S, v + 3 * i, gg, hv + 6 * i);
}

}  // namespace egg_b200
