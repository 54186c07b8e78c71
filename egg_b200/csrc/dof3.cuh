// One structured-interior DOF of a 3D sweep from its node window: Newton
// system and line search over the 32 corner samples that move it (W_inv = I).
//
// The DOF sits at window node p.  Every sample that moves it is three edges
// (the columns of T) at p or at one of its six neighbours:
//
//   axis k, side +-  the sample's corner is the neighbour n = p +- e_k, its
//                    column k the edge between n and p, its columns i, j the
//                    edges of n along the other two axes (2 x 2 signs): 24
//                    samples.  A move d of the DOF changes column k alone, by
//                    w = +d (n below p) or -d (n above).
//   corner           the DOF is the corner; with the outward edges
//                    o_l = X_nbr - X_p every column moves by -d: 8 samples.
//
// mu + 1 = s q F(D) / 9 (metric3.cuh), with t_k the moving column, c = t_i x
// t_j, x_e = t_e x t_k and u_e = x_e x t_e for the two other edges e, n = |t|^2:
//
//   D = t_k.c,  s = n_i + n_j + n_k,  q = |c|^2 + |x_i|^2 + |x_j|^2,
//   dD = c,  ds = 2 t_k,  dq = 2 kb with kb = u_i + u_j,
//   d2s = 2 I,  d2q = 2 (M_i + M_j) with M_e = |t_e|^2 I - t_e t_e^T,  d2D = 0,
//
// so the 24 axis samples need no cofactor matrix: each costs one cross product
// and a few scalars; x_e, u_e and the lengths belong to an edge and are shared
// by the samples of a (k, side) group.  The sums over a group factor further:
// the M_e parts collect one coefficient per edge, the t_k (.)^T parts one
// vector per group.  For the corner, with the cofactors C_l = o_i x o_j (cyclic)
// and the differences f_l = o_i - o_j: c = sum C_l, q = sum |C_l|^2,
// kb = sum C_l x f_l and M = sum |f_l|^2 I - f_l f_l^T.
//
// Every second-order term is a cross product or a sum of squares (the diagonal
// of M_e is the sum of the other two components' squares).  Expanded into
// products of lengths and dot products (q = |c|^2 + (n_i + n_j) n_k - d_ik^2 -
// d_jk^2, kb = (n_i + n_j) t_k - ..., (n_i + n_j) I - ...) the same quantities
// cancel to (short / long)^2 of their terms where a cell's edges differ in
// length or lie near one line: the fp32 step of 1 : 0.01 : 0.01 cells was then
// off by 8e-4 of the short spacing (median), and is by 8e-7 in this form, for
// 3% of the kernel (129^3 cube, mixed: 545 us a sweep, now 560).
//
// V is double, or F2: two fp32 lanes evaluated by one instruction (x2.cuh).
// The lanes are the two sides of an axis group, and the two directions of
// axis 2 at the corner.  The functions also compile for the host, where the
// tests hold them against extended precision.
#pragma once

#include "metric3.cuh"
#include "x2.cuh"

namespace egg_b200
{

struct F2 {
    float2 v;
};

EGG_HD F2 operator+(F2 a, F2 b) { return F2 {add2(a.v, b.v)}; }
EGG_HD F2 operator-(F2 a, F2 b) { return F2 {sub2(a.v, b.v)}; }
EGG_HD F2 operator*(F2 a, F2 b) { return F2 {mul2(a.v, b.v)}; }
EGG_HD F2 vfma(F2 a, F2 b, F2 c) { return F2 {fma2(a.v, b.v, c.v)}; }
EGG_HD double vfma(double a, double b, double c) { return fma(a, b, c); }

template <class V> struct Lane;
template <> struct Lane<F2> {
    using R = float;
    static EGG_HD F2 set(float a) { return F2 {p2(a)}; }
    static EGG_HD F2 set(float a, float b) { return F2 {make_float2(a, b)}; }
    static EGG_HD float sum(F2 a) { return a.v.x + a.v.y; }
};
template <> struct Lane<double> {
    using R = double;
    static EGG_HD double set(double a) { return a; }
    static EGG_HD double sum(double a) { return a; }
};

// Two scalar negations: cheaper than a packed product with -1, which would
// take the FMA pipe for two cycles.
EGG_HD F2 vneg(F2 a) { return F2 {make_float2(-a.v.x, -a.v.y)}; }
EGG_HD double vneg(double a) { return -a; }

template <class V> EGG_HD V dotv(const V a[3], const V b[3])
{
    return vfma(a[2], b[2], vfma(a[1], b[1], a[0] * b[0]));
}

// n = -a
template <class V> EGG_HD void negv(const V a[3], V n[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i) { n[i] = vneg(a[i]); }
}

// o = a x b, given na = -a (a packed subtraction would spend an instruction
// on each sign).
template <class V> EGG_HD void crossv(const V a[3], const V na[3], const V b[3], V o[3])
{
    o[0] = vfma(a[1], b[2], na[2] * b[1]);
    o[1] = vfma(a[2], b[0], na[0] * b[2]);
    o[2] = vfma(a[0], b[1], na[1] * b[0]);
}

// F = 1/D^2 (or 1/Dh^2, untangle), f3 = -F'/2 and f4 = F''/6; the divisions
// and roots round as IEEE prescribes.  Products that feed a sum are fused by
// hand, so that every instance of a kernel rounds alike.
template <int KIND, class R> EGG_HD void scale3(R D, R delta, R& F, R& f3, R& f4)
{
    if constexpr (KIND == kUntangle) {
        const R r = sqrt(fma(D, D, R(4) * delta * delta));
        const R Dh = R(0.5) * (D + r);
        const R d1 = Dh / r, d2 = R(2) * delta * delta / (r * r * r);
        const R inv = R(1) / Dh;
        const R inv2 = inv * inv, inv3 = inv2 * inv;
        F = inv2;
        f3 = d1 * inv3;
        f4 = fma(d1 * d1, inv2 * inv2, R(-1.0 / 3.0) * d2 * inv3);
    } else {
        const R inv = R(1) / D;
        F = inv * inv;
        f3 = F * inv;
        f4 = F * F;
    }
}

template <int KIND> EGG_HD void scale3v(double D, double delta, double& F, double& f3, double& f4)
{
    scale3<KIND, double>(D, delta, F, f3, f4);
}
template <int KIND> EGG_HD void scale3v(F2 D, float delta, F2& F, F2& f3, F2& f4)
{
    if constexpr (KIND == kUntangle) {
        scale3<KIND, float>(D.v.x, delta, F.v.x, f3.v.x, f4.v.x);
        scale3<KIND, float>(D.v.y, delta, F.v.y, f3.v.y, f4.v.y);
    } else {
        const F2 inv = Lane<F2>::set(1.0f / D.v.x, 1.0f / D.v.y);
        F = inv * inv;
        f3 = F * inv;
        f4 = F * F;
    }
}

// Sums over samples of 9 times the gradient, Hessian and metric.  A holds
// sums of x y^T + y x^T as x_i y_i on the diagonal and x_i y_j + x_j y_i off
// it; H = 2 hI I + A, its diagonal doubled.
template <class V> struct Sys3 {
    V g[3], A[6], hI, e;
    EGG_HD void clear()
    {
        const V z = Lane<V>::set(0);
#pragma unroll
        for (int q = 0; q < 3; ++q) { g[q] = z; }
#pragma unroll
        for (int q = 0; q < 6; ++q) { A[q] = z; }
        hI = z;
        e = z;
    }
};

template <class V> EGG_HD void sym_add(V A[6], const V x[3], const V y[3])
{
    A[0] = vfma(x[0], y[0], A[0]);
    A[1] = vfma(x[0], y[1], vfma(x[1], y[0], A[1]));
    A[2] = vfma(x[0], y[2], vfma(x[2], y[0], A[2]));
    A[3] = vfma(x[1], y[1], A[3]);
    A[4] = vfma(x[1], y[2], vfma(x[2], y[1], A[4]));
    A[5] = vfma(x[2], y[2], A[5]);
}

// H += 2 coef (|x|^2 I - x x^T), given m2 = -2 coef: the products off the
// diagonal into A, -2 coef times the squares into sq, which spread_sq gives to
// the diagonal's other two entries.
template <class V> EGG_HD void cross_add(V A[6], V sq[3], const V x[3], V m2)
{
    V y[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        y[m] = m2 * x[m];
        sq[m] = vfma(y[m], x[m], sq[m]);
    }
    A[1] = vfma(y[0], x[1], A[1]);
    A[2] = vfma(y[0], x[2], A[2]);
    A[4] = vfma(y[1], x[2], A[4]);
}
template <class V> EGG_HD void spread_sq(V A[6], const V sq[3])
{
    const V mh = Lane<V>::set(-0.5f);
    A[0] = vfma(mh, sq[1] + sq[2], A[0]);
    A[3] = vfma(mh, sq[0] + sq[2], A[3]);
    A[5] = vfma(mh, sq[0] + sq[1], A[5]);
}

// An edge t of a group, nt = -t: |x|^2 of x = t x t_k, and v = t x x (= -u:
// the sign is left to the caller's constants).
template <class V> EGG_HD void edge_cross(const V t[3], const V nt[3], const V tk[3], V& xx, V v[3])
{
    V x[3];
    crossv(t, nt, tk, x);
    xx = dotv(x, x);
    crossv(t, nt, x, v);
}

// The four samples of one (axis, side) group, both sides in the lanes of F2:
// tk the edge to the neighbour, ti[2], tj[2] the neighbour's edges (below,
// above) along the other axes.  sgn is the sign of w: +1 below, -1 above.
// Constant factors are left to the end of the group: with Q = q f3
// and v = -kb,
//   g   = 2 hI t_k - 2 G,  hI = sum q F,  G = sum (s Q) c + sum (sF) v,
//   P   = -4 sum (F v + Q c)          (t_k P^T + P t_k^T)
//   r   = 3 s q f4 c + 4 s f3 v       (c r^T + r c^T).
template <int KIND, bool GRAD, class V>
EGG_HD void axis_system(const V tk[3], const V ti[2][3], const V tj[2][3], V sgn, typename Lane<V>::R delta,
                        Sys3<V>& S)
{
    using L = Lane<V>;
    const V z = L::set(0), one = L::set(-1);
    const V nk = dotv(tk, tk);
    V P[3] = {z, z, z}, G[3] = {z, z, z}, sq[3] = {z, z, z}, gj[2], hI = z;
    V nj[2], xj[2], vj[2][3];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        V nt[3];
        negv(tj[b], nt);
        edge_cross(tj[b], nt, tk, xj[b], vj[b]);
        nj[b] = dotv(tj[b], tj[b]);
        gj[b] = z;
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        V gi = z, nt[3], xi, vi[3];
        negv(ti[a], nt);
        edge_cross(ti[a], nt, tk, xi, vi);
        const V ni = nk + dotv(ti[a], ti[a]);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            V c[3], r[3];
            crossv(ti[a], nt, tj[b], c);
            const V D = dotv(tk, c), s = ni + nj[b];
            const V q = vfma(c[2], c[2], vfma(c[1], c[1], vfma(c[0], c[0], xi + xj[b])));
            V F, f3, f4;
            scale3v<KIND>(D, delta, F, f3, f4);
            const V sF = s * F, Q = q * f3;
            V sQ = s * Q, rc = (s * q) * (f4 * L::set(3));
            const V rk = (s * L::set(4)) * f3;
            S.e = vfma(sF, q, S.e);
            hI = vfma(q, F, hI);
            gi = gi + sF;
            gj[b] = gj[b] + sF;
            if constexpr (KIND == kShapeSize) {  // + (D - 1)^2
                const V dm1 = D + one;
                sQ = vfma(L::set(-9), dm1, sQ);
                rc = rc + L::set(9);
                S.e = vfma(L::set(9) * dm1, dm1, S.e);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                G[m] = vfma(sQ, c[m], G[m]);
                if constexpr (GRAD) { continue; }
                const V v = vi[m] + vj[b][m];
                P[m] = vfma(F, v, vfma(Q, c[m], P[m]));
                r[m] = vfma(rc, c[m], rk * v);
            }
            if constexpr (!GRAD) { sym_add(S.A, c, r); }
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) { G[m] = vfma(gi, vi[m], G[m]); }
        if constexpr (!GRAD) { cross_add(S.A, sq, ti[a], gi * L::set(-2)); }
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
#pragma unroll
        for (int m = 0; m < 3; ++m) { G[m] = vfma(gj[b], vj[b][m], G[m]); }
        if constexpr (!GRAD) { cross_add(S.A, sq, tj[b], gj[b] * L::set(-2)); }
    }
    const V s2 = sgn * L::set(2), m2 = sgn * L::set(-2);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        S.g[m] = vfma(s2 * hI, tk[m], vfma(m2, G[m], S.g[m]));
        P[m] = P[m] * L::set(-4);
    }
    if constexpr (!GRAD) {
        sym_add(S.A, tk, P);
        spread_sq(S.A, sq);
    }
    S.hI = S.hI + hI;
}

// The corner's cofactors C_l = o_i x o_j (cyclic).
template <class V> EGG_HD void corner_cofactors(const V o0[3], const V o1[3], const V o2[3], V C[3][3])
{
    V m0[3], m1[3];
    negv(o0, m0);
    negv(o1, m1);
    crossv(o1, m1, o2, C[0]);
    crossv(m0, o0, o2, C[1]);  // o2 x o0 = -o0 x o2
    crossv(o0, m0, o1, C[2]);
}

// One corner sample (two lanes of F2 along axis 2): outward edges o0, o1, o2
// and the sign sig of T's determinant over theirs.
template <int KIND, bool GRAD, class V>
EGG_HD void corner_system(const V o0[3], const V o1[3], const V o2[3], V sig, typename Lane<V>::R delta, Sys3<V>& S)
{
    using L = Lane<V>;
    const V one = L::set(-1), three = L::set(3);
    V C[3][3], f[3][3], c[3], kb[3], q = L::set(0);
    corner_cofactors(o0, o1, o2, C);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        f[0][m] = o1[m] - o2[m];
        f[1][m] = o2[m] - o0[m];
        f[2][m] = o0[m] - o1[m];
    }
#pragma unroll
    for (int l = 0; l < 3; ++l) {
        V n[3], k[3];
        negv(C[l], n);
        crossv(C[l], n, f[l], k);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            q = vfma(C[l][m], C[l][m], q);
            c[m] = l ? c[m] + C[l][m] : C[l][m];
            kb[m] = l ? kb[m] + k[m] : k[m];
        }
    }
    const V D = sig * dotv(o2, C[2]);
    const V s = dotv(o0, o0) + dotv(o1, o1) + dotv(o2, o2);
    V F, f3, f4;
    scale3v<KIND>(D, delta, F, f3, f4);
    const V sF = s * F, qF = q * F, Q = q * (sig * f3);
    S.e = vfma(sF, q, S.e);
    S.hI = vfma(three, qF, S.hI);
    V sQ = s * Q, rc = (s * q) * (f4 * three);
    if constexpr (KIND == kShapeSize) {
        const V dm1 = D + one;
        sQ = vfma(L::set(-9) * sig, dm1, sQ);
        rc = rc + L::set(9);
        S.e = vfma(L::set(9) * dm1, dm1, S.e);
    }
    const V two = L::set(2), pk = L::set(4) * F, pc = L::set(-4) * Q, rk = (L::set(-4) * s) * (sig * f3);
    const V ga = L::set(-2) * qF, gk = L::set(-2) * sF, gc = two * sQ;
    V a[3], p[3], r[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        a[m] = o0[m] + o1[m] + o2[m];
        S.g[m] = vfma(ga, a[m], vfma(gk, kb[m], vfma(gc, c[m], S.g[m])));
        if constexpr (GRAD) { continue; }
        p[m] = vfma(pk, kb[m], pc * c[m]);
        r[m] = vfma(rc, c[m], rk * kb[m]);
    }
    if constexpr (!GRAD) {
        sym_add(S.A, a, p);
        sym_add(S.A, c, r);
        V sq[3] = {L::set(0), L::set(0), L::set(0)};
#pragma unroll
        for (int l = 0; l < 3; ++l) { cross_add(S.A, sq, f[l], gk); }
        spread_sq(S.A, sq);
    }
}

// Edge sources.  fe: fp32 forward edges of the window, fe[(3 k + i) N + node]
// = (X[node + e_k] - X[node])_i; P: fp64 positions, P[i N + node].
template <int N> struct EdgeF {
    const float* fe;
    // forward edge at nodes (na, nb) of the axis whose block starts at ax = 3 k N
    EGG_HD void get(int ax, int na, int nb, F2 o[3]) const
    {
#pragma unroll
        for (int i = 0; i < 3; ++i) { o[i] = F2 {make_float2(fe[ax + i * N + na], fe[ax + i * N + nb])}; }
    }
};

template <int N> struct EdgeD {
    const double* P;
    // X[b] - X[a]
    EGG_HD void get(int a, int b, double o[3]) const
    {
#pragma unroll
        for (int i = 0; i < 3; ++i) { o[i] = P[i * N + b] - P[i * N + a]; }
    }
};

// The axis of one pass of the axis loop and the other two, in cyclic order:
// node strides, fe blocks and corner-index bits.
struct AxisTurn {
    int sk, si, sj, fk, fi, fj, bk, bi, bj;
    EGG_HD void next()
    {
        int t = sk;
        sk = si, si = sj, sj = t;
        t = fk;
        fk = fi, fi = fj, fj = t;
        t = bk;
        bk = bi, bi = bj, bj = t;
    }
};
template <class W> EGG_HD AxisTurn axis_turn()
{
    return AxisTurn {W::S0, W::S1, W::S2, 0, 3 * W::N, 6 * W::N, 4, 2, 1};
}

// Newton system of the DOF at window node p: gradient g[3] and Hessian h[6]
// = (xx, xy, xz, yy, yz, zz); GRAD: the gradient alone (h is not the Hessian).
template <class W, int KIND, bool GRAD>
EGG_HD void dof3_system(const EdgeF<W::N>& E, int p, float delta, float g[3], float h[6])
{
    using L = Lane<F2>;
    Sys3<F2> S;
    S.clear();
    {
        F2 o2[3];
        E.get(6 * W::N, p - 1, p, o2);
#pragma unroll
        for (int m = 0; m < 3; ++m) { o2[m].v.x = -o2[m].v.x; }
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            const float s0 = (c & 2) ? 1.0f : -1.0f, s1 = (c & 1) ? 1.0f : -1.0f;
            const int na = (c & 2) ? p : p - W::S0, nb = (c & 1) ? p : p - W::S1;
            F2 o0[3], o1[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                o0[m] = L::set(s0 * E.fe[m * W::N + na]);
                o1[m] = L::set(s1 * E.fe[(3 + m) * W::N + nb]);
            }
            corner_system<KIND, GRAD>(o0, o1, o2, L::set(-s0 * s1, s0 * s1), delta, S);
        }
    }
    AxisTurn t = axis_turn<W>();
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const int na = p - t.sk, nb = p + t.sk;
        F2 tk[3], ti[2][3], tj[2][3];
        E.get(t.fk, na, p, tk);
        E.get(t.fi, na - t.si, nb - t.si, ti[0]);
        E.get(t.fi, na, nb, ti[1]);
        E.get(t.fj, na - t.sj, nb - t.sj, tj[0]);
        E.get(t.fj, na, nb, tj[1]);
        axis_system<KIND, GRAD>(tk, ti, tj, L::set(1.0f, -1.0f), delta, S);
        t.next();
    }
    constexpr float n9 = float(1.0 / 9.0);
    const float hI = 2.0f * L::sum(S.hI);
#pragma unroll
    for (int m = 0; m < 3; ++m) { g[m] = fmul_rn(n9, L::sum(S.g[m])); }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const float A = L::sum(S.A[m]);
        h[m] = fmul_rn(n9, (m == 0 || m == 3 || m == 5) ? fmaf(2.0f, A, hI) : A);
    }
}

// fp64; e: the energy of the 32 moving samples without their constant -1.
// NH = 2: two neighbouring threads share the DOF, each with one side of every
// group and one direction of axis 2 at the corner (`half`); both end with the
// same totals and take the same decisions.
#ifdef __CUDACC__
__device__ __forceinline__ unsigned pair_mask() { return 3u << (threadIdx.x & 30u); }
#endif
template <int NH> EGG_HD double pair_sum(double v)
{
#ifdef __CUDA_ARCH__
    if constexpr (NH == 2) { v += __shfl_xor_sync(pair_mask(), v, 1, 2); }
#endif
    return v;
}
template <int NH> EGG_HD double pair_min(double v)
{
#ifdef __CUDA_ARCH__
    if constexpr (NH == 2) { v = fmin(v, __shfl_xor_sync(pair_mask(), v, 1, 2)); }
#endif
    return v;
}

template <class W, int KIND, int NH, bool GRAD>
EGG_HD void dof3_system(const EdgeD<W::N>& E, int p, int half, double delta, double g[3],
                                            double h[6], double& e)
{
    Sys3<double> S;
    S.clear();
#pragma unroll 1
    for (int c = 4 * half; c < 4 * half + 8 / NH; ++c) {
        double o0[3], o1[3], o2[3];
        E.get(p, (c & 2) ? p + W::S0 : p - W::S0, o0);
        E.get(p, (c & 1) ? p + W::S1 : p - W::S1, o1);
        E.get(p, (c & 4) ? p + W::S2 : p - W::S2, o2);
        const double sig = ((c ^ (c >> 1) ^ (c >> 2)) & 1) ? 1.0 : -1.0;  // product of the three edge signs
        corner_system<KIND, GRAD>(o0, o1, o2, sig, delta, S);
    }
    AxisTurn t = axis_turn<W>();
#pragma unroll 1
    for (int k = 0; k < 6 / NH; ++k) {
        const bool up = NH == 2 ? half != 0 : (k & 1) != 0;
        const int n = up ? p + t.sk : p - t.sk;
        double tk[3], ti[2][3], tj[2][3];
        E.get(up ? p : n, up ? n : p, tk);
        E.get(n - t.si, n, ti[0]);
        E.get(n, n + t.si, ti[1]);
        E.get(n - t.sj, n, tj[0]);
        E.get(n, n + t.sj, tj[1]);
        axis_system<KIND, GRAD>(tk, ti, tj, up ? -1.0 : 1.0, delta, S);
        if (NH == 2 || up) { t.next(); }
    }
    constexpr double n9 = 1.0 / 9.0;
#pragma unroll
    for (int m = 0; m < 3; ++m) { g[m] = n9 * pair_sum<NH>(S.g[m]); }
    if constexpr (!GRAD) {
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            h[m] = n9 * pair_sum<NH>((m == 0 || m == 3 || m == 5) ? 2.0 * (S.A[m] + S.hI) : S.A[m]);
        }
        e = n9 * pair_sum<NH>(S.e);
    }
}

// ---------------------------------------------------------------------------
// Line search, fp32: the summed metric changes of the 32 moving samples when
// the DOF moves by d, free of the cancellation of e' - e.  With w the change of
// t_k: dD = w.c, ds = 2 w.t_k + |w|^2 and dq = sum y_e.(2 x_e + y_e) with
// y_e = t_e x w; at the corner C_l changes by y_l = d x f_l = d x o_i - d x o_j.
// ---------------------------------------------------------------------------

// mu(T') - mu(T) (times 9) from s, q, D and their changes; dn = D + dD.
template <int KIND> EGG_HD F2 dmu3_pair(F2 s, F2 q, F2 D, F2 ds, F2 dq, F2 dD, float delta, F2& dn)
{
    using L = Lane<F2>;
    dn = D + dD;
    F2 x = D, xn = dn, dx = dD;
    if constexpr (KIND == kUntangle) {
        float xo[2], xno[2], dxo[2];
        const float Dl[2] = {D.v.x, D.v.y}, nl[2] = {dn.v.x, dn.v.y}, cl[2] = {dD.v.x, dD.v.y};
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const float d2 = 4.0f * delta * delta;
            const float r = sqrtf(fmaf(Dl[l], Dl[l], d2)), rn = sqrtf(fmaf(nl[l], nl[l], d2));
            xo[l] = untangle_dh_stable(Dl[l], r, delta);
            xno[l] = untangle_dh_stable(nl[l], rn, delta);
            dxo[l] = untangle_ddh(Dl[l], nl[l], r, rn, cl[l], delta);
        }
        x = L::set(xo[0], xo[1]);
        xn = L::set(xno[0], xno[1]);
        dx = L::set(dxo[0], dxo[1]);
    }
    // s' q' F(x') - s q F(x) = d(sq) / x'^2 - s q dx (x + x') / (x x')^2, on the
    // one quotient g = 1 / (x x'): x g = 1 / x'
    const F2 g = F2 {ldiv2(p2(1.0f), (x * xn).v)};
    const F2 dsq = vfma(ds, q + dq, s * dq), ixn = x * g;
    F2 dm = vfma(ixn * ixn, dsq, (vneg(s * q) * g) * ((dx * g) * (x + xn)));
    if constexpr (KIND == kShapeSize) { dm = vfma(L::set(9.0f) * dD, dn + D + L::set(-2.0f), dm); }
    return dm;
}

// Folds one pair of trial samples into the sums.  A sample whose det is below
// kGuard times its columns' lengths is near-degenerate: dn^2 - kGuard^2 nnn is
// then negative.  The first pass only keeps the smallest such value, `low`; a
// pass with GUARD (rare) leaves those samples out and sets their bits in
// `guard` (bx, by) for the caller to difference them in fp64.
template <bool GUARD>
EGG_HD void line_fold(F2 dm, F2 dn, F2 nnn, unsigned bx, unsigned by, F2& dsum, float& md,
                                          float& low, unsigned& guard)
{
    const F2 t = vfma(dn, dn, Lane<F2>::set(-float(kGuard * kGuard)) * nnn);
    if constexpr (GUARD) {
        const bool gx = !(fabsf(dn.v.x) > 0.0f) || t.v.x < 0.0f, gy = !(fabsf(dn.v.y) > 0.0f) || t.v.y < 0.0f;
        guard |= (gx ? bx : 0u) | (gy ? by : 0u);
        dsum = dsum + Lane<F2>::set(gx ? 0.0f : dm.v.x, gy ? 0.0f : dm.v.y);
        md = fminf(md, fminf(gx ? INFINITY : dn.v.x, gy ? INFINITY : dn.v.y));
    } else {
        dsum = dsum + dm;
        md = fminf(md, fminf(dn.v.x, dn.v.y));
        low = fminf(low, fminf(t.v.x, t.v.y));
    }
}

// |x|^2 of x = t x t_k and its change when t_k moves by w.
EGG_HD void edge_change(const F2 t[3], const F2 nt[3], const F2 tk[3], const F2 w[3], F2& xx, F2& dx)
{
    F2 x[3], y[3];
    crossv(t, nt, tk, x);
    crossv(t, nt, w, y);
    xx = dotv(x, x);
    const F2 two = Lane<F2>::set(2.0f);
#pragma unroll
    for (int m = 0; m < 3; ++m) { x[m] = vfma(two, x[m], y[m]); }
    dx = dotv(y, x);
}

// Guard bits: bit 8 role + cell, role 0 the corner and 1 + k the axis-k
// samples, cell = the cell's side along each axis (bit 4 axis 0).
template <class W, int KIND, bool GUARD>
EGG_HD float dof3_line(const EdgeF<W::N>& E, int p, const float d[3], float delta, float& md,
                                           float& low, unsigned& guard)
{
    using L = Lane<F2>;
    const F2 two = L::set(2.0f), mtwo = L::set(-2.0f);
    const F2 dd = L::set(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    F2 dsum = L::set(0.0f);
    {
        const F2 D3[3] = {L::set(d[0]), L::set(d[1]), L::set(d[2])};
        const F2 N3[3] = {L::set(-d[0]), L::set(-d[1]), L::set(-d[2])};
        F2 o2[3];
        E.get(6 * W::N, p - 1, p, o2);
#pragma unroll
        for (int m = 0; m < 3; ++m) { o2[m].v.x = -o2[m].v.x; }
        const F2 n2 = dotv(o2, o2), x2 = dotv(o2, D3);
        F2 v[3][3];  // d x o_l
        crossv(D3, N3, o2, v[2]);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            const float s0 = (c & 2) ? 1.0f : -1.0f, s1 = (c & 1) ? 1.0f : -1.0f;
            const int na = (c & 2) ? p : p - W::S0, nb = (c & 1) ? p : p - W::S1;
            F2 o0[3], o1[3], C[3][3], cs[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                o0[m] = L::set(s0 * E.fe[m * W::N + na]);
                o1[m] = L::set(s1 * E.fe[(3 + m) * W::N + nb]);
            }
            const F2 sig = L::set(-s0 * s1, s0 * s1);
            corner_cofactors(o0, o1, o2, C);
            crossv(D3, N3, o0, v[0]);
            crossv(D3, N3, o1, v[1]);
            F2 q = L::set(0.0f), dq = q;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                cs[m] = C[0][m] + C[1][m] + C[2][m];
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const F2 y = v[(l + 1) % 3][m] - v[(l + 2) % 3][m];
                    q = vfma(C[l][m], C[l][m], q);
                    dq = vfma(y, vfma(two, C[l][m], y), dq);
                }
            }
            const F2 D = sig * dotv(o2, C[2]), dD = vneg(sig * dotv(D3, cs));
            const F2 n0 = dotv(o0, o0), n1 = dotv(o1, o1), s = n0 + n1 + n2;
            const F2 x0 = dotv(o0, D3), x1 = dotv(o1, D3);
            const F2 ds = vfma(L::set(3.0f), dd, mtwo * (x0 + x1 + x2));
            F2 dn;
            const F2 dm = dmu3_pair<KIND>(s, q, D, ds, dq, dD, delta, dn);
            const F2 nn = (vfma(mtwo, x0, n0) + dd) * (vfma(mtwo, x1, n1) + dd) * (vfma(mtwo, x2, n2) + dd);
            // cell bits: side of axis 0 (4), axis 1 (2), axis 2 (lane)
            const unsigned cell = unsigned((c & 2) << 1 | (c & 1) << 1);
            line_fold<GUARD>(dm, dn, nn, 1u << cell, 1u << (cell | 1u), dsum, md, low, guard);
        }
    }
    AxisTurn t = axis_turn<W>();
    const F2 w[3] = {L::set(d[0], -d[0]), L::set(d[1], -d[1]), L::set(d[2], -d[2])};
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const int na = p - t.sk, nb = p + t.sk;
        F2 tk[3], tj[2][3], nj[2], xj[2], dj[2];
        E.get(t.fk, na, p, tk);
        const F2 nk = dotv(tk, tk), ds = vfma(two, dotv(w, tk), dd), nkn = nk + ds;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            E.get(t.fj, b ? na : na - t.sj, b ? nb : nb - t.sj, tj[b]);
            F2 nt[3];
            negv(tj[b], nt);
            nj[b] = dotv(tj[b], tj[b]);
            edge_change(tj[b], nt, tk, w, xj[b], dj[b]);
        }
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            F2 ti[3], nt[3], xi, di;
            E.get(t.fi, a ? na : na - t.si, a ? nb : nb - t.si, ti);
            negv(ti, nt);
            edge_change(ti, nt, tk, w, xi, di);
            const F2 ni = dotv(ti, ti), nki = nkn * ni;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                F2 c[3];
                crossv(ti, nt, tj[b], c);
                const F2 D = dotv(tk, c), dD = dotv(w, c), s = nk + (ni + nj[b]);
                const F2 q = vfma(c[2], c[2], vfma(c[1], c[1], vfma(c[0], c[0], xi + xj[b])));
                const F2 dq = di + dj[b];
                F2 dn;
                const F2 dm = dmu3_pair<KIND>(s, q, D, ds, dq, dD, delta, dn);
                const unsigned cell = unsigned(8 * (k + 1) + (a ? t.bi : 0) + (b ? t.bj : 0));
                line_fold<GUARD>(dm, dn, nki * nj[b], 1u << cell, 1u << (cell + t.bk), dsum, md, low, guard);
            }
        }
        t.next();
    }
    return fmul_rn(float(1.0 / 9.0), L::sum(dsum));
}

// fp64: the energy of the 32 moving samples (without their constant -1) with
// the DOF moved by d (summed over its NH threads), and this thread's smallest det.
template <class W, int KIND, int NH>
EGG_HD double dof3_trial(const EdgeD<W::N>& E, int p, int half, const double d[3], double delta,
                                             double& md)
{
    auto value = [&](double s, double q, double D) {
        double x = D;
        if constexpr (KIND == kUntangle) { x = 0.5 * (D + sqrt(D * D + 4.0 * delta * delta)); }
        const double inv = 1.0 / x;
        double v = s * q * (inv * inv) * (1.0 / 9.0);
        if constexpr (KIND == kShapeSize) { v += (D - 1.0) * (D - 1.0); }
        md = fmin(md, D);
        return v;
    };
    double e = 0.0;
#pragma unroll 1
    for (int c = 4 * half; c < 4 * half + 8 / NH; ++c) {
        double o0[3], o1[3], o2[3], C[3][3];
        E.get(p, (c & 2) ? p + W::S0 : p - W::S0, o0);
        E.get(p, (c & 1) ? p + W::S1 : p - W::S1, o1);
        E.get(p, (c & 4) ? p + W::S2 : p - W::S2, o2);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            o0[m] -= d[m];
            o1[m] -= d[m];
            o2[m] -= d[m];
        }
        corner_cofactors(o0, o1, o2, C);
        const double D = (((c ^ (c >> 1) ^ (c >> 2)) & 1) ? 1.0 : -1.0) * dotv(o2, C[2]);
        e += value(dotv(o0, o0) + dotv(o1, o1) + dotv(o2, o2),
                   dotv(C[0], C[0]) + dotv(C[1], C[1]) + dotv(C[2], C[2]), D);
    }
    AxisTurn t = axis_turn<W>();
#pragma unroll 1
    for (int k = 0; k < 6 / NH; ++k) {
        const bool up = NH == 2 ? half != 0 : (k & 1) != 0;
        const int n = up ? p + t.sk : p - t.sk;
        double tk[3], tj[2][3], nj[2], xj[2];
        E.get(up ? p : n, up ? n : p, tk);
#pragma unroll
        for (int m = 0; m < 3; ++m) { tk[m] += up ? -d[m] : d[m]; }
        const double nk = dotv(tk, tk);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            E.get(b ? n : n - t.sj, b ? n + t.sj : n, tj[b]);
            double nt[3], x[3];
            negv(tj[b], nt);
            crossv(tj[b], nt, tk, x);
            nj[b] = dotv(tj[b], tj[b]);
            xj[b] = dotv(x, x);
        }
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            double ti[3], nt[3], x[3];
            E.get(a ? n : n - t.si, a ? n + t.si : n, ti);
            negv(ti, nt);
            crossv(ti, nt, tk, x);
            const double ni = dotv(ti, ti), xi = dotv(x, x);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                double c[3];
                crossv(ti, nt, tj[b], c);
                e += value(nk + (ni + nj[b]), dotv(c, c) + (xi + xj[b]), dotv(tk, c));
            }
        }
        if (NH == 2 || up) { t.next(); }
    }
    return pair_sum<NH>(e);
}

}  // namespace egg_b200
