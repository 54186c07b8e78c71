// Packed-fp32 structured-interior sweep for mixed precision (sm_100a).
//
// One CTA = CI x CJ DOFs, one per thread, over the (CI+1) x (CJ+1) cells
// around them, on Blackwell's two-lane fp32 instructions (x2.cuh):
//   phase 1  every window node's fp64 position goes to shared memory (for the
//            fp64 fallbacks) and its two forward edges with it, each the fp64
//            difference of two positions rounded once to fp32 (the neighbours
//            come from L1);
//   phase 2  one thread per cell (a second, partial round covers the cells
//            beyond the CTA's CI x CJ threads; one thread per cell in whole
//            warps measured slower, fewer CTAs fitting per SM) evaluates the
//            cell's four samples as two lane pairs (samples 0|1 and 2|3 share
//            their axis-0 edges) and stores the role contributions per corner
//            -- in a layout shifted by one cell (below) so that a DOF gathers
//            each row of its cells with one 64-bit load -- and a flag for an
//            inverted or badly shaped sample;
//   phase 3  one thread per DOF sums its 4 corners, solves, and line-searches
//            its 12 moving samples as 6 lane pairs (cells (ci, 0) | (ci, 1),
//            same role) on the 12 edges around it, accepting on summed exact
//            metric changes with the fp64 tolerance.  Trial samples with
//            |det| < kGuard |a0||a1| are redone in fp64 from the fp64 window;
//            DOFs next to a flagged cell relax entirely in fp64
//            (warp_dofs_fp64).
// The sample semantics are src/structured_patch.hpp:89-258 and
// src/sweep.hpp:1534-1650.
#pragma once

#include "kernels2d.cuh"
#include "x2.cuh"

namespace egg_b200
{

template <int CI, int CJ> struct TileSharedX2 {
    static constexpr int CH = CI + 1, CW = CJ + 1;  // cells staged
    static constexpr int NC = CH * CW;
    static constexpr int PW = CW + 1;                // window row length (nodes)
    static constexpr int PH = CH + 1;                // window rows
    static constexpr int NN = PH * PW;               // window nodes
    static constexpr int NT = CI * CJ;               // threads: one per DOF
    double2 P[NN];                                   // fp64 window
    float f0x[NN], f0y[NN], f1x[NN], f1y[NN];        // forward edges along axis 0 / axis 1
    // Corner values of cell c, shifted: g[p][q][c] = (corner 2p+1 of cell c,
    // corner 2p of cell c+1), q = gx, gy, hxx, hxy, hyy; a DOF whose cells
    // are c00, c01 (row 0) and c10, c11 (row 1) takes corners 3 | 2 from
    // g[1][q][c00] and 1 | 0 from g[0][q][c10].
    float2 g[2][5][NC];
    uint8_t bad[NC];  // cell with an inverted or badly shaped sample
};

// Summed metric changes of the 12 moving samples for the DOF moved by (dx, dy),
// as 6 lane pairs: cells (ci, 0) | (ci, 1), same role.  Without GUARD the
// smallest det^2 - kGuard^2 |a0|^2 |a1|^2 of a trial sample comes back in
// `low`; with it, the samples below zero are left out and set their bits.
//
// w is the window node up and left of the DOF.  The edges are read from shared
// memory sample pair by sample pair (volatile, so that the loads are not
// hoisted): holding all 24 of them spilled, 253 us a 2049^2 sweep against
// 228.
template <class S, int KIND, bool GUARD>
__device__ __forceinline__ float x2_line(const S& sm, int w, float dx, float dy, float fdelta, float& md, float& low,
                                         unsigned& guard)
{
    constexpr int PW = S::PW;
    const volatile float* F0x = sm.f0x + w;
    const volatile float* F0y = sm.f0y + w;
    const volatile float* F1x = sm.f1x + w;
    const volatile float* F1y = sm.f1y + w;
    const float kg = float(kGuard * kGuard);
    const float2 DX = p2(dx), DY = p2(dy), NX = p2(-dx), NY = p2(-dy);
    const float2 RX = make_float2(dx, -dx), RY = make_float2(dy, -dy);
    const float2 dd = p2(dx * dx + dy * dy);
    float2 dsum2 = p2(0.0f);
#pragma unroll
    for (int ci = 0; ci < 2; ++ci) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            // column edges at columns j - 1 | j + 1 of cell row ci (r = 2) or
            // the one at column j; row edges west | east of the DOF's row, or
            // of the outer row (r = 1)
            const int v = ci * PW + (r == 2 ? 0 : 1), h = (r == 1 ? 2 * ci : 1) * PW;
            const float2 t0 = r == 2 ? make_float2(F0x[v], F0x[v + 2]) : p2(F0x[v]);
            const float2 t2 = r == 2 ? make_float2(F0y[v], F0y[v + 2]) : p2(F0y[v]);
            const float2 t1 = make_float2(F1x[h], F1x[h + 1]), t3 = make_float2(F1y[h], F1y[h + 1]);
            const float2 N0 = fma2(t0, t0, mul2(t2, t2)), N1 = fma2(t1, t1, mul2(t3, t3));
            const float2 Sv = add2(N0, N1);
            const float2 D = fma2(t0, t3, neg2(mul2(t1, t2)));
            // the moved columns: column 0 by s0 d (r = 1), column 1 by s1 d
            // (r = 2), both by -s d (the corner); s0 is -1 in the upper
            // cells' corner samples, s1 is -1 | 1 there
            float2 ds, dD, n0t, n1t;
            if (r == 1) {
                const float2 ex = ci ? NX : DX, ey = ci ? NY : DY;
                ds = fma2(p2(2.0f), fma2(t0, ex, mul2(t2, ey)), dd);
                dD = fma2(ex, t3, neg2(mul2(ey, t1)));
                const float2 cx = add2(t0, ex), cy = add2(t2, ey);
                n0t = fma2(cx, cx, mul2(cy, cy));
                n1t = N1;
            } else if (r == 2) {
                const float2 ex = RX, ey = RY;
                ds = fma2(p2(2.0f), fma2(t1, ex, mul2(t3, ey)), dd);
                dD = fma2(t0, ey, neg2(mul2(ex, t2)));
                const float2 cx = add2(t1, ex), cy = add2(t3, ey);
                n0t = N0;
                n1t = fma2(cx, cx, mul2(cy, cy));
            } else {  // det dT = 0
                const float2 e0x = ci ? NX : DX, e0y = ci ? NY : DY, e1x = RX, e1y = RY;
                const float2 dot = add2(fma2(t0, e0x, mul2(t2, e0y)), fma2(t1, e1x, mul2(t3, e1y)));
                ds = fma2(p2(2.0f), dot, add2(dd, dd));
                dD = add2(fma2(e0x, t3, neg2(mul2(e0y, t1))), fma2(t0, e1y, neg2(mul2(e1x, t2))));
                const float2 cx = add2(t0, e0x), cy = add2(t2, e0y), fx = add2(t1, e1x), fy = add2(t3, e1y);
                n0t = fma2(cx, cx, mul2(cy, cy));
                n1t = fma2(fx, fx, mul2(fy, fy));
            }
            const float2 M2 = KIND == kShapeSize ? ldiv2(Sv, D) : p2(0.0f);
            float2 dn;
            const float2 dm = dmu2_pair<KIND>(Sv, D, add2(D, D), M2, ds, dD, fdelta, dn);
            const float2 gq = fma2(dn, dn, mul2(p2(-kg), mul2(n0t, n1t)));
            if constexpr (GUARD) {
                const bool gx = gq.x < 0.0f, gy = gq.y < 0.0f;
                guard |= (gx ? 1u << (ci * 6 + r) : 0u) | (gy ? 1u << (ci * 6 + 3 + r) : 0u);
                dsum2 = add2(dsum2, make_float2(gx ? 0.0f : dm.x, gy ? 0.0f : dm.y));
                md = fminf(md, fminf(gx ? INFINITY : dn.x, gy ? INFINITY : dn.y));
            } else {
                dsum2 = add2(dsum2, dm);
                md = fminf(md, fminf(dn.x, dn.y));
                low = fminf(low, fminf(gq.x, gq.y));
            }
        }
    }
    return dsum2.x + dsum2.y;
}

// Near-degenerate trial samples in fp64, out of line: inlined, their fp64
// temporaries would raise the register demand of the whole kernel.  k = 6 ci +
// 3 cj + r: role r of cell (ci, cj) around the DOF, P the upper left of its
// 3 x 3 nodes.
template <int KIND>
__device__ __noinline__ float x2_guard64(const double2* P, int PW, int k, double dx, double dy, double delta, float& dn)
{
    const int ci = k / 6, cj = (k / 3) % 2, r = k % 3;
    const int a = (1 - ci) * 2 + (1 - cj);
    const int b = (r == 0) ? a : ((r == 1) ? (a ^ 2) : (a ^ 1));
    auto node = [&](int c) { return P[(ci + (c >> 1)) * PW + cj + (c & 1)]; };
    return dmu2_guard64<KIND>(node(b), node(b ^ 2), node(b ^ 1), r, dx, dy, (b & 2) ? -1.0 : 1.0,
                              (b & 1) ? -1.0 : 1.0, delta, dn);
}

template <class S, int KIND>
__device__ __noinline__ float x2_line_guard(const S& sm, const double2* P, int w, float dx, float dy, double delta, float& md)
{
    float low = 0.0f;
    unsigned guard = 0u;
    md = INFINITY;
    float ds = x2_line<S, KIND, true>(sm, w, dx, dy, float(delta), md, low, guard);
#pragma unroll 1
    for (int k = 0; guard && k < 12; ++k) {
        if (!((guard >> k) & 1u)) { continue; }
        float dn;
        ds += x2_guard64<KIND>(P, S::PW, k, double(dx), double(dy), delta, dn);
        md = fminf(md, dn);
    }
    return ds;
}

template <int CI, int CJ, int MINB, int KIND>
__global__ void __launch_bounds__(TileSharedX2<CI, CJ>::NT, MINB)
  interior_x2_kernel(const double2* __restrict__ Xin, double2* __restrict__ Xout, const Tile2* __restrict__ tiles,
                     const uint8_t* __restrict__ active, const double2* __restrict__ tau, double delta, double omega,
                     double2* __restrict__ grad_out)
{
    using S = TileSharedX2<CI, CJ>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S& sm = *reinterpret_cast<S*>(smem_raw);
    constexpr int NT = S::NT, PW = S::PW, NN = S::NN, CW = S::CW, NC = S::NC;
    const float fdelta = float(delta);

    const Tile2 tile = tiles[blockIdx.x];
    const int n0 = tile.n0, n1 = tile.n1;
    const int r0 = tile.i0 - 1, c0 = tile.j0 - 1;  // window origin (always inside the block)
    const int tid = threadIdx.x;

    // Phase 1.  Nodes outside the block, and edges that leave it or the window,
    // are zero: never part of a valid cell.
    for (int k = tid; k < NN; k += NT) {
        const int r = k / PW, c = k % PW;
        const int wi = r0 + r, wj = c0 + c;
        double2 v = make_double2(0.0, 0.0);
        float2 f0 = make_float2(0.0f, 0.0f), f1 = f0;
        if (wi < n0 && wj < n1) {
            const double2* p = Xin + tile.off + int64_t(wi) * n1 + wj;
            v = *p;
            if (r < S::PH - 1 && wi + 1 < n0) {
                const double2 d = p[n1];
                f0 = make_float2(float(d.x - v.x), float(d.y - v.y));
            }
            if (c < PW - 1 && wj + 1 < n1) {
                const double2 d = p[1];
                f1 = make_float2(float(d.x - v.x), float(d.y - v.y));
            }
        }
        sm.P[k] = v;
        sm.f0x[k] = f0.x;
        sm.f0y[k] = f0.y;
        sm.f1x[k] = f1.x;
        sm.f1y[k] = f1.y;
    }
    // This thread's DOF, its active flag and tau, in flight during phase 2.
    const int ti = tid / CJ, tj = tid % CJ;
    const int gi = tile.i0 + ti, gj = tile.j0 + tj;
    const int64_t slot = tile.off + int64_t(gi) * n1 + gj;
    const bool mine = gi <= n0 - 2 && gj <= n1 - 2 && active[slot];
    double2 tv = make_double2(0.0, 0.0);
    if (mine && tau != nullptr) { tv = tau[slot]; }
    __syncthreads();

    // Phase 2: thread t takes cells t, t + NT, ...  Cell (ci, cj) has its base
    // at window node (ci, cj).
    for (int cell = tid; cell < NC; cell += NT) {
        const int ci = cell / CW, cj = cell % CW;
        if (r0 + ci > n0 - 2 || c0 + cj > n1 - 2) { continue; }  // read by no DOF
        const int a = ci * PW + cj;
        // edges as lane pairs over the two sides: axis 0 (00->10 | 01->11),
        // axis 1 (00->01 | 10->11)
        const float2 e0x = make_float2(sm.f0x[a], sm.f0x[a + 1]), e0y = make_float2(sm.f0y[a], sm.f0y[a + 1]);
        const float2 e1x = make_float2(sm.f1x[a], sm.f1x[a + PW]), e1y = make_float2(sm.f1y[a], sm.f1y[a + PW]);
        // shifted stores: lane y of pair p goes to slot cell (.x), lane x to
        // slot cell - 1 (.y), which no DOF reads when cj = 0
        float* gs = reinterpret_cast<float*>(&sm.g[0][0][0]);
        auto put_g = [&](int p, int q, float2 v) {
            gs[2 * ((p * 5 + q) * NC + cell)] = v.y;
            if (cj > 0) { gs[2 * ((p * 5 + q) * NC + cell - 1) + 1] = v.x; }
        };
        // corner c receives sample c in role 0, sample c^2 in role 1 and
        // sample c^1 in role 2.  Samples 0 | 1 first, folded at once into the
        // corner pairs 0 | 1 and 2 | 3 so that fewer values stay live.
        const float kb = float(kBadCell * kBadCell);
        float2 G01[5], G23[5];
        bool bad;
        {
            Roles2 P;  // columns (axis-0 side 0 | 1, axis-1 side 0)
            roles2<KIND>(e0x, p2(e1x.x), e0y, p2(e1y.x), p2(1.0f), make_float2(1.0f, -1.0f), fdelta, P);
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                G01[q] = make_float2(P.r0[q].x + P.r2[q].y, P.r0[q].y + P.r2[q].x);
                G23[q] = P.r1[q];
            }
            // inverted or badly shaped sample (sine of a corner below kBadCell)
            const float2 bp = fma2(P.D, P.D, mul2(p2(-kb), mul2(P.n0, P.n1)));
            bad = !(fminf(P.D.x, P.D.y) > 0.0f) || !(fminf(bp.x, bp.y) >= 0.0f) || P.D.x != P.D.x || P.D.y != P.D.y;
        }
        {
            Roles2 Q;  // samples 2 | 3: columns (axis-0 side 0 | 1, axis-1 side 1)
            roles2<KIND>(e0x, p2(e1x.y), e0y, p2(e1y.y), p2(-1.0f), make_float2(1.0f, -1.0f), fdelta, Q);
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                put_g(0, q, add2(G01[q], Q.r1[q]));
                const float2 B = add2(G23[q], Q.r0[q]);
                put_g(1, q, make_float2(B.x + Q.r2[q].y, B.y + Q.r2[q].x));
            }
            const float2 bq = fma2(Q.D, Q.D, mul2(p2(-kb), mul2(Q.n0, Q.n1)));
            bad = bad || !(fminf(Q.D.x, Q.D.y) > 0.0f) || !(fminf(bq.x, bq.y) >= 0.0f) || Q.D.x != Q.D.x ||
                  Q.D.y != Q.D.y;
        }
        sm.bad[cell] = bad ? 1 : 0;
    }
    __syncthreads();

    // Phase 3.
    const int c00 = ti * CW + tj, c10 = c00 + CW;
    const double2* P = sm.P + ti * PW + tj;  // the DOF's 3 x 3 nodes
    bool bad = false;
    if (mine) { bad = (sm.bad[c00] | sm.bad[c00 + 1] | sm.bad[c10] | sm.bad[c10 + 1]) != 0; }
    if (mine && !bad) {
        float gsum[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {  // corner of each cell: (0,0) -> 3, (0,1) -> 2, (1,0) -> 1, (1,1) -> 0
            const float2 v = add2(sm.g[1][q][c00], sm.g[0][q][c10]);
            gsum[q] = v.x + v.y;
        }
        const float tx = float(tv.x), ty = float(tv.y);
        const float gv[2] = {gsum[0] - tx, gsum[1] - ty};
        if (grad_out != nullptr) {
            grad_out[slot] = make_double2(double(gv[0]), double(gv[1]));
        } else {
            const float Hm[4] = {gsum[2], gsum[3], gsum[3], gsum[4]};
            float dl[2];
            solve2<float>(Hm, gv, dl);
            float alpha = 1.0f;
            double2 out = P[PW + 1];
#pragma unroll 1
            for (int it = 0; it < 10; ++it) {
                const int w = ti * PW + tj;
                const float dx = alpha * dl[0], dy = alpha * dl[1];
                float md = INFINITY, low = INFINITY;
                unsigned guard = 0u;
                float ds = x2_line<S, KIND, false>(sm, w, dx, dy, fdelta, md, low, guard);
                if (!(low >= 0.0f) || !isfinite(ds)) {  // a near-degenerate trial sample: rare
                    ds = x2_line_guard<S, KIND>(sm, P, w, dx, dy, delta, md);
                }
                ds -= tx * dx + ty * dy;
                if (isfinite(ds) && ds <= float(Tol<double>::energy) && (KIND == kUntangle || md > 0.0f)) {
                    out.x += omega * double(dx);
                    out.y += omega * double(dy);
                    break;
                }
                alpha *= 0.5f;
            }
            Xout[slot] = out;
        }
    }
    __syncwarp();
    warp_dofs_fp64<KIND>(bad, P, PW, slot, tv, delta, omega, Xout, grad_out);
}

}  // namespace egg_b200
