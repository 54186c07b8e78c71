// 2D sweep kernels of the egg_b200 core (sm_100a).
//
// Store layout: every block is a dense row-major (n0, n1) array of nodes with
// the two coordinates interleaved (double2 per node); blocks are packed back to
// back.  No ghost ring: cross-block reads go to owner slots (stored-patch DOFs)
// or to the block's own refreshed copies of shared interface nodes.
//
// One block-Jacobi sweep (src/sweep.hpp:1938 jacobi_sweep_once) is
//   interior_fp64_kernel structured-interior DOFs (patch synthesized, W_inv = I;
//                        mixed precision: interior_x2_kernel)
//   stored_patch_kernel  every other moving DOF (ragged stored patch); it also
//                        writes the DOF's copies in other blocks
// Both read X_in (frozen snapshot) and write X_out.  Nodes that no DOF moves
// keep the copies that both buffers start with (broadcast2_kernel).
#pragma once

#include "entity2.cuh"
#include "metric.cuh"
#include "soft.cuh"

#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

namespace egg_b200
{

struct BlockInfo {
    int64_t off;  // first node slot of the block in the packed store
    int32_t n[3]; // node counts per axis (n[2] = 1 in 2D)
    int32_t pad;
};

// A tile of structured-interior DOFs with its block's data, so that a CTA
// starts on one load instead of two dependent ones.
struct __align__(16) Tile2 {
    int64_t off;     // first node slot of the block
    int32_t n0, n1;  // the block's node counts
    int32_t i0;      // first DOF row (logical, >= 1)
    int32_t j0;      // first DOF column
    int32_t pad[2];
};

__device__ __forceinline__ double2 ld2(const double2* p) { return *p; }

// ---------------------------------------------------------------------------
// One sample from its two edge vectors e0 = s0 (n0 - c), e1 = s1 (n1 - c)
// (already signed).  vec(T) = [e0.x, e1.x, e0.y, e1.y] (A[:,k] = e_k, W = I).
// ---------------------------------------------------------------------------
template <class C> struct SampleOut {
    C mu, det;
    C g[4];
    C H[16];
};

template <int KIND, class C>
__device__ __forceinline__ void sample_full_c(C ax, C bx, C ay, C by, C delta, SampleOut<C>& o)
{
    const C t[4] = {ax, bx, ay, by};
    mu_eval<C>(KIND, t, delta, o.mu, o.g, o.H);
    o.det = det2(t);
}

// Value + det only (line-search trials), working precision C with fp64 guard.
template <int KIND, class C>
__device__ __forceinline__ C sample_mu_c(C ax, C bx, C ay, C by, C delta, C& det)
{
    const C t[4] = {ax, bx, ay, by};
    det = det2(t);
    return mu_value<C>(KIND, t, delta);
}

// Per-sample contributions to the three nodes a sample moves, without forming
// the full 4x4 metric Hessian: only its 10 distinct entries enter
//   role 1 (axis-0 neighbour)  grad s0 (g0, g2),  jhj (H00, H02, H22)
//   role 2 (axis-1 neighbour)  grad s1 (g1, g3),  jhj (H11, H13, H33)
//   role 0 (corner)            grad -(role1 + role2),
//                              jhj  role1 + role2 + s0 s1 (2 H01, H03 + H12, 2 H23)
// (role_Jb / accumulate_sample of src/patch.hpp:204-320 with W_inv = I).
template <class C> struct RoleOut {
    C mu, det;
    C r[3][5];  // [role 0, 1, 2][gx, gy, hxx, hxy, hyy]
};

template <int KIND, class C>
__device__ __forceinline__ void sample_roles_c(C a, C b, C c, C d, C s0, C s1, C delta, RoleOut<C>& o)
{
    const C t[4] = {a, b, c, d};
    const C cof[4] = {d, -c, -b, a};
    const C D = a * d - b * c;
    const C s = a * a + b * b + c * c + d * d;
    ScaleFn<C> sf = (KIND == kUntangle) ? untangle_scale(D, delta) : shape_scale(D);
    const C m = s * sf.f;
    C g2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { g2[i] = C(2) * sf.f * t[i] + s * sf.fp * cof[i]; }
    const C dm1 = D - C(1);
    auto P = [](int i, int j) -> C {
        const int k = i * 4 + j;
        return (k == 3 || k == 12) ? C(1) : ((k == 6 || k == 9) ? C(-1) : C(0));
    };
    // i, j are constants after inlining: the terms whose factor is an exact
    // zero (off-diagonal 2f, P(i, j) = 0) are left out rather than multiplied
    // by 0, which IEEE arithmetic would not let the compiler drop.
    auto H = [&](int i, int j) -> C {
        const C p = P(i, j);
        C h2 = C(2) * sf.fp * (t[i] * cof[j] + cof[i] * t[j]);
        if (i == j) { h2 = C(2) * sf.f + h2; }
        h2 = h2 + s * sf.fpp * cof[i] * cof[j];
        if (p != C(0)) { h2 = h2 + s * sf.fp * p; }
        if (KIND != kShapeSize) { return h2; }
        C h = C(2) * g2[i] * g2[j] + C(2) * m * h2 + C(2) * cof[i] * cof[j];
        if (p != C(0)) { h = h + C(2) * dm1 * p; }
        return h;
    };
    C g[4];
    if (KIND == kShapeSize) {
        o.mu = m * m - C(1) + dm1 * dm1;
#pragma unroll
        for (int i = 0; i < 4; ++i) { g[i] = C(2) * m * g2[i] + C(2) * dm1 * cof[i]; }
    } else {
        o.mu = m - C(1);
#pragma unroll
        for (int i = 0; i < 4; ++i) { g[i] = g2[i]; }
    }
    o.det = D;
    const C h00 = H(0, 0), h01 = H(0, 1), h02 = H(0, 2), h03 = H(0, 3), h11 = H(1, 1);
    const C h12 = H(1, 2), h13 = H(1, 3), h22 = H(2, 2), h23 = H(2, 3), h33 = H(3, 3);
    o.r[1][0] = s0 * g[0];
    o.r[1][1] = s0 * g[2];
    o.r[1][2] = h00;
    o.r[1][3] = h02;
    o.r[1][4] = h22;
    o.r[2][0] = s1 * g[1];
    o.r[2][1] = s1 * g[3];
    o.r[2][2] = h11;
    o.r[2][3] = h13;
    o.r[2][4] = h33;
    const C ss = s0 * s1;
    o.r[0][0] = -(o.r[1][0] + o.r[2][0]);
    o.r[0][1] = -(o.r[1][1] + o.r[2][1]);
    o.r[0][2] = h00 + h11 + C(2) * ss * h01;
    o.r[0][3] = h02 + h13 + ss * (h03 + h12);
    o.r[0][4] = h22 + h33 + C(2) * ss * h23;
}

// ---------------------------------------------------------------------------
// Owner -> non-owner copy refresh (src/structured_halo.hpp:197 fused_halo_broadcast).
// ---------------------------------------------------------------------------
__global__ void broadcast2_kernel(double2* __restrict__ X, const int32_t* __restrict__ src,
                                  const int32_t* __restrict__ dst, int64_t n)
{
    for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n;
         e += int64_t(gridDim.x) * blockDim.x) {
        X[dst[e]] = X[src[e]];
    }
}

// Mixed precision: a DOF whose patch touches a cell with an inverted sample or
// a corner angle below asin(kBadCell) is relaxed entirely in fp64 (patch,
// Newton step and line search), since accept/reject decisions next to such
// cells are ill-conditioned in fp32.
constexpr double kBadCell = 0.1;

// Complete fp64 update (or, grad_only, gradient) of one DOF by 16 lanes, one
// per sample of its 2 x 2 cells (mask: those lanes, l this lane's sample):
// P points to the upper left of its 3 x 3 nodes, PW the row length.  Every
// lane returns the same point.  W_inv = I; 2x2 Newton step, <= 10 halvings,
// omega blend.
//
// The accept test compares the energies of the 12 samples the DOF moves; the
// four others add the same constant to both sides, and one of them that is
// inverted (outside untangle) or has no finite metric rules every step out.  A
// trial with a det <= 0 is refused (outside untangle) before its energies.
//
// One lane alone took some 5000 instructions for such a DOF (16 full samples
// in fp64, and ten trials of 16 where an inverted sample keeps it in place)
// while the rest of its warp waited: on a +-0.3 h grid, where 1% of the DOFs
// touch a bad cell, that was a third of the sweep (2049^2: 280 us a sweep
// against 208 at +-0.2 h; with 16 lanes 228).
template <int KIND>
__device__ __noinline__ double2 dof_fp64_lanes(const double2* __restrict__ P, int PW, int l, unsigned mask, double tx,
                                               double ty, double delta, double omega, bool grad_only)
{
    const int ci = l >> 3, cj = (l >> 2) & 1, b = l & 3;
    const int a = (1 - ci) * 2 + (1 - cj);
    auto node = [&](int c) { return P[(ci + (c >> 1)) * PW + cj + (c & 1)]; };
    auto sum = [&](double v) {
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) { v += __shfl_xor_sync(mask, v, o, 16); }
        return v;
    };
    const double s0 = (b & 2) ? -1.0 : 1.0, s1 = (b & 1) ? -1.0 : 1.0;
    const int role = b == a ? 0 : ((b ^ 2) == a ? 1 : ((b ^ 1) == a ? 2 : -1));
    const double2 pc = node(b), p0 = node(b ^ 2), p1 = node(b ^ 1), pos = P[PW + 1];
    const double ax = s0 * (p0.x - pc.x), bx = s1 * (p1.x - pc.x), ay = s0 * (p0.y - pc.y), by = s1 * (p1.y - pc.y);
    SampleOut<double> o;
    sample_full_c<KIND, double>(ax, bx, ay, by, delta, o);
    double g0 = 0.0, g1 = 0.0, hxx = 0.0, hxy = 0.0, hyy = 0.0;
    if (role == 0) {
        g0 = -(s0 * o.g[0] + s1 * o.g[1]);
        g1 = -(s0 * o.g[2] + s1 * o.g[3]);
        hxx = o.H[0] + o.H[5] + s0 * s1 * (o.H[1] + o.H[4]);
        hxy = o.H[2] + o.H[7] + s0 * s1 * (o.H[3] + o.H[6]);
        hyy = o.H[10] + o.H[15] + s0 * s1 * (o.H[11] + o.H[14]);
    } else if (role == 1) {
        g0 = s0 * o.g[0];
        g1 = s0 * o.g[2];
        hxx = o.H[0];
        hxy = o.H[2];
        hyy = o.H[10];
    } else if (role == 2) {
        g0 = s1 * o.g[1];
        g1 = s1 * o.g[3];
        hxx = o.H[5];
        hxy = o.H[7];
        hyy = o.H[15];
    }
    const double gv[2] = {sum(g0) - tx, sum(g1) - ty};
    if (grad_only) { return make_double2(gv[0], gv[1]); }
    hxx = sum(hxx);
    hxy = sum(hxy);
    hyy = sum(hyy);
    const double e0 = sum(role >= 0 ? o.mu : 0.0);
    if (__any_sync(mask, role < 0 && (!isfinite(o.mu) || (KIND != kUntangle && !(o.det > 0.0))))) { return pos; }
    const double Hm[4] = {hxx, hxy, hxy, hyy};
    double dl[2];
    solve2<double>(Hm, gv, dl);
    // this lane's columns move by k0 d and k1 d
    const double k0 = role == 0 ? -s0 : (role == 1 ? s0 : 0.0), k1 = role == 0 ? -s1 : (role == 2 ? s1 : 0.0);
    double alpha = 1.0;
#pragma unroll 1
    for (int it = 0; it < 10; ++it, alpha *= 0.5) {
        const double dx = alpha * dl[0], dy = alpha * dl[1];
        const double t[4] = {ax + k0 * dx, bx + k1 * dx, ay + k0 * dy, by + k1 * dy};
        if (KIND != kUntangle && __any_sync(mask, role >= 0 && !(det2(t) > 0.0))) { continue; }
        const double e = sum(role >= 0 ? mu_value<double>(KIND, t, delta) : 0.0) - (tx * dx + ty * dy);
        if (isfinite(e) && e <= e0 + Tol<double>::energy) {
            return make_double2(pos.x + omega * dx, pos.y + omega * dy);
        }
    }
    return pos;
}

// The DOFs of a warp that need fp64 (`bad` on their lanes), two at a time by
// dof_fp64_lanes; each lane passes its own DOF's window, slot and tau.  All 32
// lanes call this.
template <int KIND>
__device__ __forceinline__ void warp_dofs_fp64(bool bad, const double2* P, int PW, int64_t slot, double2 tau,
                                               double delta, double omega, double2* __restrict__ Xout,
                                               double2* __restrict__ grad_out)
{
    unsigned todo = __ballot_sync(0xffffffffu, bad);
    const int half = (threadIdx.x >> 4) & 1;
    while (todo != 0u) {
        const int first = __ffs(int(todo)) - 1;
        todo &= todo - 1u;
        const int second = todo != 0u ? __ffs(int(todo)) - 1 : -1;
        todo &= todo - 1u;  // 0 stays 0
        const int src = half == 0 ? first : (second >= 0 ? second : first);
        const double2* Ps = reinterpret_cast<const double2*>(
          __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(P), src));
        const int64_t sl = __shfl_sync(0xffffffffu, slot, src);
        const double tx = __shfl_sync(0xffffffffu, tau.x, src), ty = __shfl_sync(0xffffffffu, tau.y, src);
        if (half == 0 || second >= 0) {
            const double2 r = dof_fp64_lanes<KIND>(Ps, PW, threadIdx.x & 15, half ? 0xffff0000u : 0x0000ffffu, tx, ty,
                                                   delta, omega, grad_out != nullptr);
            if ((threadIdx.x & 15) == 0) { (grad_out != nullptr ? grad_out : Xout)[sl] = r; }
        }
        __syncwarp();
    }
}

// fp64 metric change of one near-degenerate trial sample, from the staged
// fp64 positions of its corner qc and neighbours q0, q1; the moving node
// (role 0 corner, 1 axis-0 neighbour, 2 axis-1 neighbour) is displaced by
// (dx, dy).  Called from a separate loop after the fp32 pass, so its fp64
// temporaries do not weigh on the fp32 line search's registers.
template <int KIND>
__device__ float dmu2_guard64(double2 qc, double2 q0, double2 q1, int role, double dx, double dy,
                                           double s0, double s1, double delta, float& dn)
{
    double d0, d1;
    const double m0 = sample_mu_c<KIND, double>(s0 * (q0.x - qc.x), s1 * (q1.x - qc.x), s0 * (q0.y - qc.y),
                                                s1 * (q1.y - qc.y), delta, d0);
    if (role == 0) {
        qc.x += dx;
        qc.y += dy;
    } else if (role == 1) {
        q0.x += dx;
        q0.y += dy;
    } else {
        q1.x += dx;
        q1.y += dy;
    }
    const double m1 = sample_mu_c<KIND, double>(s0 * (q0.x - qc.x), s1 * (q1.x - qc.x), s0 * (q0.y - qc.y),
                                                s1 * (q1.y - qc.y), delta, d1);
    dn = d1 > 0.0 ? fmaxf(float(d1), 1e-38f) : (d1 < 0.0 ? fminf(float(d1), -1e-38f) : 0.0f);
    return float(m1 - m0);
}

// ---------------------------------------------------------------------------
// Fused structured-interior sweep, fp64.  One CTA = one tile of CI x CJ DOFs,
// one per thread, over the (CI+1) x (CJ+1) cells around them.  Phase 1 stages
// the (CI+2) x (CJ+2) node window in shared memory; phase 2 evaluates each
// cell's four corner samples ONCE (the reference re-evaluates every sample for
// each of the 4 DOFs that share it) and stores the sums per cell corner:
// gradient, contracted Hessian, and the energy of the three samples that move
// that corner; phase 3 adds a DOF's four corners, takes the 2x2 Newton step,
// backtracks (<= 10 halvings) on the energy of the 12 samples it moves, applies
// the omega blend and writes X_out.  The four other samples of its patch add
// the same constant to both sides of the accept test; one that is inverted
// (outside untangle) or has no finite metric rules every step out (a bit per
// sample and cell).  Patch semantics follow src/structured_patch.hpp:89-258
// and src/sweep.hpp:1534-1650.
//
// fp64 issue bounds it (2049^2, +-0.3 h: 309 us a sweep; 365 before, 72 against
// 95 at 1025^2).  The line search works on the 12 edges around the DOF
// (only the four that meet there move) and divides once for two samples; after
// a refused trial it looks at the dets first, so that a DOF held in place by an
// inverted sample does not run ten full trials beside its warp.
// The gradient and Hessian keep their order of operations: next to an almost
// degenerate sample H holds (1/sine)^2 against 1, and a last bit there grows
// by an order a sweep (a form with fewer operations ran 294 us, and moved such
// nodes by 1e-1 h within ten sweeps).
// NT > CI CJ: one round of phase 2 for every cell (small levels, where one
// CTA's chain is the sweep's time).
// ---------------------------------------------------------------------------
template <int CI, int CJ> struct TileShared64 {
    static constexpr int CH = CI + 1, CW = CJ + 1, NC = CH * CW;
    double2 P[(CH + 1) * (CW + 1)];
    double gh[4][6][NC];  // per cell corner: gx, gy, hxx, hxy, hyy, energy
    uint8_t stop[NC];     // bit b: sample b rules out steps of the DOF it does not move
};

// Energies of two samples from their squared lengths and dets: s/(2D) each, on
// one division (untangle with the surrogate dets).
template <int KIND>
__device__ __forceinline__ double pair_energy64(double sa, double Da, double sb, double Db, double delta)
{
    if constexpr (KIND == kShapeSize) {
        const double r = 0.5 / (Da * Db), ma = sa * Db * r, mb = sb * Da * r, da = Da - 1.0, db = Db - 1.0;
        return (ma * ma - 1.0 + da * da) + (mb * mb - 1.0 + db * db);
    } else {
        if constexpr (KIND == kUntangle) {
            Da = untangle_dh(Da, delta);
            Db = untangle_dh(Db, delta);
        }
        return (sa * Db + sb * Da) / (2.0 * (Da * Db)) - 2.0;
    }
}

template <int CI, int CJ, int NT, int MINB, int KIND>
__global__ void __launch_bounds__(NT, MINB)
  interior_fp64_kernel(const double2* __restrict__ Xin, double2* __restrict__ Xout, const Tile2* __restrict__ tiles,
                       const uint8_t* __restrict__ active, const double2* __restrict__ tau, double delta, double omega,
                       double2* __restrict__ grad_out)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using S = TileShared64<CI, CJ>;
    S& sm = *reinterpret_cast<S*>(smem_raw);
    constexpr int NC = S::NC, CW = S::CW, PW = CW + 1;
    const Tile2 tile = tiles[blockIdx.x];
    const int n0 = tile.n0, n1 = tile.n1;
    const int r0 = tile.i0 - 1, c0 = tile.j0 - 1;  // node window origin
    const int tid = threadIdx.x;

    // Phase 1: node window.
    for (int k = tid; k < (S::CH + 1) * PW; k += NT) {
        const int r = k / PW, c = k % PW;
        const int gi = r0 + r, gj = c0 + c;
        double2 v = make_double2(0.0, 0.0);
        if (gi < n0 && gj < n1) { v = Xin[tile.off + int64_t(gi) * n1 + gj]; }
        sm.P[k] = v;
    }
    // this thread's DOF, its flag and tau: in flight while phase 2 runs
    const int ti = tid / CJ, tj = tid % CJ;
    const int gi = tile.i0 + ti, gj = tile.j0 + tj;
    const int64_t slot = tile.off + int64_t(gi) * n1 + gj;
    const bool mine = tid < CI * CJ && gi <= n0 - 2 && gj <= n1 - 2 && active[slot];
    double2 tv = make_double2(0.0, 0.0);
    if (mine && tau != nullptr) { tv = tau[slot]; }
    __syncthreads();

    // Phase 2: cell (ci, cj) has its base at window node (ci, cj).
    for (int cell = tid; cell < NC; cell += NT) {
        const int ci = cell / CW, cj = cell % CW;
        if (r0 + ci > n0 - 2 || c0 + cj > n1 - 2) { continue; }  // read by no DOF
        double acc[4][5], em[4];  // role contributions and moved energies per cell corner
        unsigned stop = 0u;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int q = 0; q < 5; ++q) { acc[a][q] = 0.0; }
            em[a] = 0.0;
        }
        // Sample b's columns are the axis-0 edge on side (b & 1) and the axis-1
        // edge on side (b >> 1): the sample signs cancel the edge orientation.
        const double2 p00 = sm.P[ci * PW + cj], p01 = sm.P[ci * PW + cj + 1];
        const double2 p10 = sm.P[(ci + 1) * PW + cj], p11 = sm.P[(ci + 1) * PW + cj + 1];
        const double e0x[2] = {p10.x - p00.x, p11.x - p01.x}, e0y[2] = {p10.y - p00.y, p11.y - p01.y};
        const double e1x[2] = {p01.x - p00.x, p11.x - p10.x}, e1y[2] = {p01.y - p00.y, p11.y - p10.y};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const double s0 = (b & 2) ? -1.0 : 1.0;
            const double s1 = (b & 1) ? -1.0 : 1.0;
            RoleOut<double> o;
            sample_roles_c<KIND, double>(e0x[b & 1], e1x[b >> 1], e0y[b & 1], e1y[b >> 1], s0, s1, delta, o);
            if (!isfinite(o.mu) || (KIND != kUntangle && !(o.det > 0.0))) { stop |= 1u << b; }
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                acc[b][q] += o.r[0][q];
                acc[b ^ 2][q] += o.r[1][q];
                acc[b ^ 1][q] += o.r[2][q];
            }
            em[b] += o.mu;
            em[b ^ 2] += o.mu;
            em[b ^ 1] += o.mu;
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int q = 0; q < 5; ++q) { sm.gh[a][q][cell] = acc[a][q]; }
            sm.gh[a][5][cell] = em[a];
        }
        sm.stop[cell] = uint8_t(stop);
    }
    __syncthreads();

    // Phase 3: DOFs.
    if (!mine) { return; }
    const int c00 = ti * CW + tj;
    double sum[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    unsigned stop = 0u;
#pragma unroll
    for (int ci = 0; ci < 2; ++ci) {
#pragma unroll
        for (int cj = 0; cj < 2; ++cj) {
            const int cell = c00 + ci * CW + cj, a = (1 - ci) * 2 + (1 - cj);
#pragma unroll
            for (int q = 0; q < 6; ++q) { sum[q] += sm.gh[a][q][cell]; }
            stop |= sm.stop[cell] & (1u << (a ^ 3));
        }
    }
    const double gv[2] = {sum[0] - tv.x, sum[1] - tv.y};
    if (grad_out != nullptr) {  // gradient-only mode (FAS restriction / tau)
        grad_out[slot] = make_double2(gv[0], gv[1]);
        return;
    }
    double2 out = sm.P[(ti + 1) * PW + tj + 1];
    if (stop != 0u) {
        Xout[slot] = out;
        return;
    }
    const double Hm[4] = {sum[2], sum[3], sum[3], sum[4]};
    double dl[2];
    solve2<double>(Hm, gv, dl);

    // The 12 edges around the DOF: V[c][k] down column tj + k from window row
    // ti + c, H[r][k] along row ti + r from column tj + k; V[.][1] and H[1][.]
    // meet at the DOF.
    double Vx[2][3], Vy[2][3], Hx[3][2], Hy[3][2];
    {
        double2 up[3], at[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                at[k] = sm.P[(ti + r) * PW + tj + k];
                if (r) {
                    Vx[r - 1][k] = at[k].x - up[k].x;
                    Vy[r - 1][k] = at[k].y - up[k].y;
                }
                if (k) {
                    Hx[r][k - 1] = at[k].x - at[k - 1].x;
                    Hy[r][k - 1] = at[k].y - at[k - 1].y;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) { up[k] = at[k]; }
        }
    }
    double alpha = 1.0;
#pragma unroll 1
    for (int it = 0; it < 10; ++it, alpha *= 0.5) {
        const double dx = alpha * dl[0], dy = alpha * dl[1];
        // the moved edges: the upper and west ones end at the DOF, the others
        // start there
        const double vx[2] = {Vx[0][1] + dx, Vx[1][1] - dx}, vy[2] = {Vy[0][1] + dy, Vy[1][1] - dy};
        const double hx[2] = {Hx[1][0] + dx, Hx[1][1] - dx}, hy[2] = {Hy[1][0] + dy, Hy[1][1] - dy};
        // sample (ci, cj, r): the corner itself (both moved edges), the
        // axis-0 neighbour (moved column edge, row edge of the outer row), the
        // axis-1 neighbour (moved row edge, outer column edge)
        auto sample = [&](int ci, int cj, int r, double& ax, double& ay, double& bx, double& by) {
            ax = r == 2 ? Vx[ci][2 * cj] : vx[ci];
            ay = r == 2 ? Vy[ci][2 * cj] : vy[ci];
            bx = r == 1 ? Hx[2 * ci][cj] : hx[cj];
            by = r == 1 ? Hy[2 * ci][cj] : hy[cj];
        };
        if (KIND != kUntangle && it > 0) {
            double md = INFINITY;
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                double ax, ay, bx, by;
                sample(k / 6, (k / 3) & 1, k % 3, ax, ay, bx, by);
                md = fmin(md, ax * by - bx * ay);
            }
            if (!(md > 0.0)) { continue; }
        }
        double e = 0.0, md = INFINITY;
#pragma unroll
        for (int k = 0; k < 6; ++k) {  // samples (0, cj, r) and (1, cj, r)
            double s[2], D[2];
#pragma unroll
            for (int ci = 0; ci < 2; ++ci) {
                double ax, ay, bx, by;
                sample(ci, k / 3, k % 3, ax, ay, bx, by);
                s[ci] = (ax * ax + ay * ay) + (bx * bx + by * by);
                D[ci] = ax * by - bx * ay;
                md = fmin(md, D[ci]);
            }
            e += pair_energy64<KIND>(s[0], D[0], s[1], D[1], delta);
        }
        e -= tv.x * dx + tv.y * dy;
        if (isfinite(e) && e <= sum[5] + Tol<double>::energy && (KIND == kUntangle || md > 0.0)) {
            out.x += omega * dx;
            out.y += omega * dy;
            break;
        }
    }
    Xout[slot] = out;
}

// ---------------------------------------------------------------------------
// Stored-patch sweep (fp64): one thread per DOF over its ragged occurrence
// slice; general W_inv, per-sample weights and the FAS tau shift.  Mirrors
// src/patch.hpp:325 patch_eval + src/sweep.hpp:1534 interior_update_kernel.
// ---------------------------------------------------------------------------
// The non-owner copies of stored DOFs (slots dst[off[d] .. off[d + 1]) of DOF d,
// off == NULL: none).  A relaxed node is written to its copies with it, so a
// sweep needs no owner -> copy launch of its own (3 us of the 12 us sweep of a
// 5 x 65^2 disk); a node that no DOF moves keeps the copies it started with.
struct Copies {
    const int32_t* off;
    const int32_t* dst;
};

struct StoredPatch2 {
    int64_t n;              // DOFs
    const int32_t* slot;    // [n] owner slot of each DOF
    const int64_t* off;     // [n+1] occurrence ranges
    const int32_t* gc;      // [occ] owner slots
    const int32_t* gn0;
    const int32_t* gn1;
    const int8_t* s0;       // [occ] +-1
    const int8_t* s1;
    const int32_t* role;    // [occ]
    const double* W;        // [occ*4] or [4]
    int32_t w_stride;       // 4 or 0
    const double* wt;       // [occ] or [1]
    int32_t wt_stride;      // 1 or 0
    const int8_t* etag;     // [n] entity tag of each DOF, or NULL (all Free)
    const double* epar;     // [n * EGG_B200_ENTITY_FIELDS] entity records (constrained DOFs)
    int cold;               // first sweep of a run call: trimmed arcs project in world space
    const double* arena;    // entity arena (B-spline knots, control points, weights)
    double* seeds;          // [n] last foot parameter of each B-spline DOF (NaN: none)
    SoftTable soft;         // directional / curvature terms per DOF (off == NULL: none)
    Copies copies;
};

__device__ __forceinline__ void assemble_T(const double2 c, const double2 n0, const double2 n1,
                                           double s0, double s1, const double* w, double t[4],
                                           double& detA)
{
    const double A00 = s0 * (n0.x - c.x), A01 = s1 * (n1.x - c.x);
    const double A10 = s0 * (n0.y - c.y), A11 = s1 * (n1.y - c.y);
    detA = A00 * A11 - A01 * A10;
    t[0] = A00 * w[0] + A01 * w[2];
    t[1] = A00 * w[1] + A01 * w[3];
    t[2] = A10 * w[0] + A11 * w[2];
    t[3] = A10 * w[1] + A11 * w[3];
}

template <int KIND>
__device__ void stored_patch_eval(const StoredPatch2& sp, const double2* X, int64_t d, double delta,
                                  double g[2], double h[4], double& e0, double& mdet)
{
    g[0] = g[1] = 0.0;
    h[0] = h[1] = h[2] = h[3] = 0.0;
    e0 = 0.0;
    mdet = INFINITY;
    for (int64_t p = sp.off[d]; p < sp.off[d + 1]; ++p) {
        const double* w = sp.W + p * sp.w_stride;
        const double s0 = sp.s0[p], s1 = sp.s1[p];
        double t[4], detA;
        assemble_T(X[sp.gc[p]], X[sp.gn0[p]], X[sp.gn1[p]], s0, s1, w, t, detA);
        mdet = fmin(mdet, detA);
        const double wt = sp.wt[p * sp.wt_stride];
        const int role = sp.role[p];
        double mu, gg[4], H[16];
        mu_eval<double>(KIND, t, delta, mu, gg, H);
        e0 += wt * mu;
        if (role < 0) { continue; }
        // Jb (4x2): row a = (i, c): column i holds v_c, v = -(s0 w[0,c] + s1 w[1,c])
        // for the corner, s_ax w[ax, c] for an axis-ax neighbour.
        double v[2];
        for (int c = 0; c < 2; ++c) {
            v[c] = (role == 0) ? -(s0 * w[0 * 2 + c] + s1 * w[1 * 2 + c])
                               : ((role == 1) ? s0 * w[0 * 2 + c] : s1 * w[1 * 2 + c]);
        }
        for (int i = 0; i < 2; ++i) {
            g[i] += wt * (gg[i * 2 + 0] * v[0] + gg[i * 2 + 1] * v[1]);
            for (int j = 0; j < 2; ++j) {
                double acc = 0.0;
                for (int c = 0; c < 2; ++c) {
                    for (int c2 = 0; c2 < 2; ++c2) { acc += v[c] * H[(i * 2 + c) * 4 + (j * 2 + c2)] * v[c2]; }
                }
                h[i * 2 + j] += wt * acc;
            }
        }
    }
}

template <int KIND>
__device__ void stored_trial(const StoredPatch2& sp, const double2* X, int64_t d, int32_t dslot,
                             double2 trial, double delta, double& e, double& md)
{
    e = 0.0;
    md = INFINITY;
    for (int64_t p = sp.off[d]; p < sp.off[d + 1]; ++p) {
        const double* w = sp.W + p * sp.w_stride;
        const int32_t ic = sp.gc[p], i0 = sp.gn0[p], i1 = sp.gn1[p];
        const double2 c = (ic == dslot) ? trial : X[ic];
        const double2 n0 = (i0 == dslot) ? trial : X[i0];
        const double2 n1 = (i1 == dslot) ? trial : X[i1];
        double t[4], detA;
        assemble_T(c, n0, n1, double(sp.s0[p]), double(sp.s1[p]), w, t, detA);
        e += sp.wt[p * sp.wt_stride] * mu_value<double>(KIND, t, delta);
        md = fmin(md, detA);
    }
}

// Reductions over an aligned group of G lanes (G a power of two <= 32) by
// xor butterfly: every lane of the group ends with the same value (each step
// adds a pair in both orders, and fp addition commutes), so the lanes of a
// group take identical Newton steps and accept decisions.
template <int G> __device__ __forceinline__ unsigned group_mask()
{
    if constexpr (G == 32) {
        return 0xffffffffu;
    } else {
        return ((1u << G) - 1u) << ((threadIdx.x & 31u) & ~unsigned(G - 1));
    }
}

template <int G> __device__ __forceinline__ double group_sum(double v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) { v += __shfl_xor_sync(group_mask<G>(), v, o, G); }
    return v;
}

template <int G> __device__ __forceinline__ double group_min(double v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) { v = fmin(v, __shfl_xor_sync(group_mask<G>(), v, o, G)); }
    return v;
}

// Lanes per DOF of the stored-patch sweeps: the widest group (32, 8, 2 or 1)
// whose threads over all stored DOFs stay within a budget.  Few stored DOFs
// (a small multi-block mesh) get a warp each, so the patch is a few rounds of
// parallel work; many (a batch of meshes) get narrow groups, which spend
// fewer issue slots on per-lane redundancy (the solve, the reductions) while
// the interior tiles run beside them.  A 3D patch has 64 samples to split,
// so its budget is larger.  Measured on B200: 256 meshes with 139 k stored
// DOFs run best at 2 lanes (a warp each: -15%); the 7-block 129^3 sphere's
// FAS levels best at 8 lanes on the fine level.
constexpr int64_t kStoredFillThreads2 = 148 * 4096;
constexpr int64_t kStoredFillThreads3 = 148 * 16384;

// Stored-patch sweep, G lanes per DOF: the lanes split the DOF's samples
// (gradient, contracted Hessian, energy; then each line-search trial) and
// reduce across the group, so a ragged patch of 16-64 gathered samples can be
// a few rounds of parallel work instead of one thread's serial loop.
//
// A sweep of a small mesh is one such chain (gathers, metric, reductions,
// projections, trials) in a few warps per SM, so its latency is what counts.
// CON says which entity code is compiled in: 0 none (no DOF is constrained),
// 1 all but B-splines and composites, 2 all of it.  The B-spline Newton solves
// alone take the kernel from 304 to 1408 bytes of stack and from 122 to 164
// registers, which every DOF on an arc paid for (5 x 129^2 disk sliding on
// arcs, 40 sweeps: 1097 us with one class for all entities, now 918).
template <int KIND, int G, int CON>
__global__ void stored_patch_kernel(StoredPatch2 sp, const double2* __restrict__ Xin,
                                    double2* __restrict__ Xout, const double2* __restrict__ tau,
                                    double delta, double omega, double2* __restrict__ grad_out)
{
    const int lane = threadIdx.x & (G - 1);
    const int64_t ngroups = (int64_t(gridDim.x) * blockDim.x) / G;
    for (int64_t d = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G; d < sp.n; d += ngroups) {
        const int32_t slot = sp.slot[d];
        const double2 pos = Xin[slot];
        const int64_t p0 = sp.off[d], p1 = sp.off[d + 1];
        double g0 = 0.0, g1 = 0.0, h00 = 0.0, h01 = 0.0, h10 = 0.0, h11 = 0.0, e0 = 0.0;
        for (int64_t p = p0 + lane; p < p1; p += G) {
            const double* w = sp.W + p * sp.w_stride;
            const double s0 = sp.s0[p], s1 = sp.s1[p];
            double t[4], detA;
            assemble_T(Xin[sp.gc[p]], Xin[sp.gn0[p]], Xin[sp.gn1[p]], s0, s1, w, t, detA);
            const double wt = sp.wt[p * sp.wt_stride];
            const int role = sp.role[p];
            double mu, gg[4], H[16];
            mu_eval<double>(KIND, t, delta, mu, gg, H);
            e0 += wt * mu;
            if (role < 0) { continue; }
            double v[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                v[c] = (role == 0) ? -(s0 * w[c] + s1 * w[2 + c]) : ((role == 1) ? s0 * w[c] : s1 * w[2 + c]);
            }
            double gl[2], hl[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                gl[i] = gg[i * 2] * v[0] + gg[i * 2 + 1] * v[1];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    double acc = 0.0;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
#pragma unroll
                        for (int c2 = 0; c2 < 2; ++c2) { acc += v[c] * H[(i * 2 + c) * 4 + (j * 2 + c2)] * v[c2]; }
                    }
                    hl[i * 2 + j] = acc;
                }
            }
            g0 += wt * gl[0];
            g1 += wt * gl[1];
            h00 += wt * hl[0];
            h01 += wt * hl[1];
            h10 += wt * hl[2];
            h11 += wt * hl[3];
        }
        double g[2] = {group_sum<G>(g0), group_sum<G>(g1)};
        double h[4] = {group_sum<G>(h00), group_sum<G>(h01), group_sum<G>(h10), group_sum<G>(h11)};
        e0 = group_sum<G>(e0);
        // Soft terms fold into the Newton system and the baseline energy
        // (src/sweep.hpp:1461-1512; constrained DOFs take the directional
        // samples only, src/sweep.hpp:1307-1327).  Every lane of the group
        // adds them alike.
        const int etag = (CON && sp.etag != nullptr) ? int(sp.etag[d]) : 0;
        soft_dof_accumulate<2>(sp.soft, d, etag == 0, reinterpret_cast<const double*>(Xin), g, h, e0);
        double tx = 0.0, ty = 0.0;
        if (tau != nullptr) {
            tx = tau[slot].x;
            ty = tau[slot].y;
            g[0] -= tx;
            g[1] -= ty;
            e0 -= tx * pos.x + ty * pos.y;
        }
        if (grad_out != nullptr) {
            if (lane == 0) { grad_out[slot] = make_double2(g[0], g[1]); }
            continue;
        }
        // A constrained DOF (src/sweep.hpp:1286-1403): the Newton step reduced
        // onto its entity's tangent, damped by omega before the line search,
        // and every trial projected onto the entity, so the accepted point
        // stays on the geometry.  A Free DOF: the full step, omega blend after.
        // A trimmed curve after the first sweep of a run call searches in its
        // parameter instead (src/sweep.hpp:1718-1876): trials q* + alpha dq,
        // clamped onto the trim and evaluated on the curve.
        const double* er = sp.epar + (etag != 0 ? d * EGG_B200_ENTITY_FIELDS : 0);
        const bool warm_arc = is_tcurve(etag) && !sp.cold;
        // B-spline DOFs carry a seed (their last foot parameter): every seeded
        // projection starts its Newton solve there and stores its result
        // (src/sweep.hpp:1219-1265).
        const bool bsp = CON == 2 && etag == EGG_B200_TAG_BSPLINE;
        const bool comp = CON == 2 && etag == EGG_B200_TAG_COMPOSITE;
        const double* cslice = comp ? sp.arena + int64_t(er[6]) : nullptr;  // the path's arena slice
        const double* crec = comp ? cslice + int64_t(er[1]) : nullptr;
        const int cseg = comp ? int(er[0]) : 0;
        double seed = bsp ? sp.seeds[d] : 0.0;
        BSplineCurve bc {};
        if (bsp) { bc = bspline_view(er, sp.arena); }
        double dl[2] = {0.0, 0.0};
        double qstar = 0.0, dq = 0.0;
        if (etag == 0) {
            solve2<double>(h, g, dl);
        } else if (comp) {  // one path for every sweep: step on the nearest segment's tangent
            composite_newton_step(cslice, crec, cseg, h, g, pos.x, pos.y, dl);
            dl[0] *= omega;
            dl[1] *= omega;
        } else if (bsp) {
            if (sp.cold) {
                bspline_cold_step(bc, h, g, pos.x, pos.y, seed, dl);
                dl[0] *= omega;
                dl[1] *= omega;
            } else {
                bspline_warm_step(bc, h, g, pos.x, pos.y, omega, seed, qstar, dq);
            }
        } else if (warm_arc) {
            tc_warm_step(etag, er, h, g, pos.x, pos.y, omega, qstar, dq);
        } else {
            entity_newton_step(etag, er, h, g, pos.x, pos.y, dl);
            dl[0] *= omega;
            dl[1] *= omega;
        }
        double alpha = 1.0;
        double2 cur = pos;
        for (int it = 0; it < 10; ++it) {
            double2 trial = make_double2(pos.x + alpha * dl[0], pos.y + alpha * dl[1]);
            if (comp) {
                double tx, ty;
                composite_frame(cslice, crec, cseg, trial.x, trial.y, trial.x, trial.y, tx, ty);
            } else if (bsp) {
                if (sp.cold) {
                    bspline_project_seeded(bc, trial.x, trial.y, seed, trial.x, trial.y);
                } else {
                    bspline_point(bc, bspline_clamp(bc, qstar + alpha * dq), 0, trial.x, trial.y);
                }
            } else if (warm_arc) {
                tc_eval(etag, er, tc_clamp(etag, er, qstar + alpha * dq), 0, trial.x, trial.y);
            } else if (etag != 0) {
                entity_project(etag, er, trial.x, trial.y, trial.x, trial.y);
            }
            double e = 0.0, md = INFINITY;
            for (int64_t p = p0 + lane; p < p1; p += G) {
                const double* w = sp.W + p * sp.w_stride;
                const int32_t ic = sp.gc[p], i0 = sp.gn0[p], i1 = sp.gn1[p];
                const double2 c = (ic == slot) ? trial : Xin[ic];
                const double2 n0 = (i0 == slot) ? trial : Xin[i0];
                const double2 n1 = (i1 == slot) ? trial : Xin[i1];
                double t[4], detA;
                assemble_T(c, n0, n1, double(sp.s0[p]), double(sp.s1[p]), w, t, detA);
                e += sp.wt[p * sp.wt_stride] * mu_value<double>(KIND, t, delta);
                md = fmin(md, detA);
            }
            e = group_sum<G>(e);
            if (sp.soft.off != nullptr) {
                const double tr[2] = {trial.x, trial.y};
                e += soft_dof_trial<2>(sp.soft, d, etag == 0, reinterpret_cast<const double*>(Xin), tr);
            }
            e -= tx * trial.x + ty * trial.y;
            md = group_min<G>(md);
            if (isfinite(e) && e <= e0 + Tol<double>::energy && (KIND == kUntangle || md > 0.0)) {
                cur = trial;
                break;
            }
            alpha *= 0.5;
        }
        if (etag == 0 && omega != 1.0) {
            cur.x = pos.x + omega * (cur.x - pos.x);
            cur.y = pos.y + omega * (cur.y - pos.y);
        }
        if (bsp && lane == 0) { sp.seeds[d] = seed; }
        if (lane == 0) {
            Xout[slot] = cur;
            if (sp.copies.off != nullptr) {
                for (int32_t c = sp.copies.off[d]; c < sp.copies.off[d + 1]; ++c) { Xout[sp.copies.dst[c]] = cur; }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Energy / min-det reductions (fp64, compensated, deterministic two-pass).
// ---------------------------------------------------------------------------
struct Comp {
    double s, c;
};

__device__ __forceinline__ void comp_add(Comp& a, double x)
{
    const double t = a.s + x;
    if (fabs(a.s) >= fabs(x)) {
        a.c += (a.s - t) + x;
    } else {
        a.c += (x - t) + a.s;
    }
    a.s = t;
}

__device__ __forceinline__ Comp comp_merge(Comp a, Comp b)
{
    Comp r = a;
    comp_add(r, b.s);
    r.c += b.c;
    return r;
}

// Block-level reduction of (compensated sum, min); thread 0 returns true and
// holds the block's result in acc / mn.
__device__ __forceinline__ bool block_reduce(Comp& acc, double& mn)
{
    __shared__ double ss[32], sc[32], sm[32];
    for (int o = 16; o > 0; o >>= 1) {
        Comp other;
        other.s = __shfl_down_sync(0xffffffffu, acc.s, o);
        other.c = __shfl_down_sync(0xffffffffu, acc.c, o);
        const double om = __shfl_down_sync(0xffffffffu, mn, o);
        acc = comp_merge(acc, other);
        mn = fmin(mn, om);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        ss[wid] = acc.s;
        sc[wid] = acc.c;
        sm[wid] = mn;
    }
    __syncthreads();
    if (wid != 0) { return false; }
    const int nw = (blockDim.x + 31) >> 5;
    Comp a {0.0, 0.0};
    double m = INFINITY;
    if (lane < nw) {
        a.s = ss[lane];
        a.c = sc[lane];
        m = sm[lane];
    }
    for (int o = 16; o > 0; o >>= 1) {
        Comp other;
        other.s = __shfl_down_sync(0xffffffffu, a.s, o);
        other.c = __shfl_down_sync(0xffffffffu, a.c, o);
        const double om = __shfl_down_sync(0xffffffffu, m, o);
        a = comp_merge(a, other);
        m = fmin(m, om);
    }
    acc = a;
    mn = m;
    return lane == 0;
}

// Where a whole-store reduction leaves its result; ticket counts the CTAs that
// have stored their partials (zero between launches; NULL: a segmented
// reduction, or one that reduce_finalize_kernel ends).
struct ReduceOut {
    double* e = nullptr;
    double* m = nullptr;
    unsigned* ticket = nullptr;
};

// The partials summed in a fixed order by one CTA: out_e = energy, out_m = min det.
__device__ __forceinline__ void reduce_partials(const double* part_s, const double* part_c, const double* part_m,
                                                int n, double* out_e, double* out_m)
{
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        acc = comp_merge(acc, Comp {__ldcg(part_s + i), __ldcg(part_c + i)});
        mn = fmin(mn, __ldcg(part_m + i));
    }
    if (block_reduce(acc, mn)) {
        *out_e = acc.s + acc.c;
        *out_m = mn;
    }
}

// Block reduction into partial slot blockIdx.y * gridDim.x + blockIdx.x
// (blockIdx.y = segment of a segmented reduction, 0 otherwise).  The last CTA to
// store sums the partials, which was a launch of its own (513^2, 4 FAS cycles
// with 12 reductions: 2507 -> 2458 us).  Which CTA is last does not change the
// order of the sum.
__device__ __forceinline__ void block_reduce_store(Comp acc, double mn, double* part_s, double* part_c,
                                                   double* part_m, ReduceOut out)
{
    __shared__ bool last;
    if (block_reduce(acc, mn)) {
        const int64_t slot = int64_t(blockIdx.y) * gridDim.x + blockIdx.x;
        part_s[slot] = acc.s;
        part_c[slot] = acc.c;
        part_m[slot] = mn;
        if (out.ticket != nullptr) {
            __threadfence();
            last = atomicAdd(out.ticket, 1u) == gridDim.x - 1;
        }
    }
    if (out.ticket == nullptr) { return; }
    __syncthreads();
    if (!last) { return; }
    __threadfence();
    reduce_partials(part_s, part_c, part_m, int(gridDim.x), out.e, out.m);
    if (threadIdx.x == 0) { *out.ticket = 0u; }
}

// Item range of this CTA row: segment blockIdx.y of `seg` (prefix offsets),
// or [0, n) without segments.
__device__ __forceinline__ void segment_range(const int64_t* seg, int64_t n, int64_t& lo, int64_t& hi)
{
    lo = seg ? seg[blockIdx.y] : 0;
    hi = seg ? seg[blockIdx.y + 1] : n;
}

struct EnergyStructured2 {
    int32_t nblocks;
    const BlockInfo* blocks;
    const int64_t* cell_off;  // [nblocks+1] prefix of (n0-1)(n1-1)
    int64_t ncell;
    const double* W;          // [4] or [ncell*4*4]
    int32_t w_stride;         // 0 or 4 (per sample)
    const double* wt;         // [1] or [ncell*4]
    int32_t wt_stride;
    const int64_t* seg = nullptr;  // per-mesh cell prefix offsets (segmented reduction) or null
};

template <int KIND>
__global__ void energy_structured2_kernel(EnergyStructured2 es, const double2* __restrict__ X,
                                          double delta, double* part_s, double* part_c,
                                          double* part_m, ReduceOut out = {})
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
        const uint32_t cw = uint32_t(bi.n[1] - 1);
        const int i = int(lc / cw), j = int(lc % cw);
        const int64_t base = bi.off + int64_t(i) * bi.n[1] + j;
        const double2 p[4] = {X[base], X[base + 1], X[base + bi.n[1]], X[base + bi.n[1] + 1]};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int64_t sid = c * 4 + b;
            const double* w = es.W + sid * es.w_stride;
            double t[4], detA;
            assemble_T(p[b], p[b ^ 2], p[b ^ 1], (b & 2) ? -1.0 : 1.0, (b & 1) ? -1.0 : 1.0, w, t,
                       detA);
            comp_add(acc, es.wt[sid * es.wt_stride] * mu_value<double>(KIND, t, delta));
            mn = fmin(mn, detA);
        }
    }
    block_reduce_store(acc, mn, part_s, part_c, part_m, out);
}

struct EnergyStored2 {
    int64_t n;
    const int32_t* gc;
    const int32_t* gn0;
    const int32_t* gn1;
    const int8_t* s0;
    const int8_t* s1;
    const double* W;
    int32_t w_stride;
    const double* wt;
    int32_t wt_stride;
    const int64_t* seg = nullptr;  // per-mesh sample prefix offsets or null
};

template <int KIND>
__global__ void energy_stored2_kernel(EnergyStored2 es, const double2* __restrict__ X, double delta,
                                      double* part_s, double* part_c, double* part_m, ReduceOut out = {})
{
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    int64_t i_lo, i_hi;
    segment_range(es.seg, es.n, i_lo, i_hi);
    for (int64_t i = i_lo + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < i_hi;
         i += int64_t(gridDim.x) * blockDim.x) {
        double t[4], detA;
        assemble_T(X[es.gc[i]], X[es.gn0[i]], X[es.gn1[i]], double(es.s0[i]), double(es.s1[i]),
                   es.W + i * es.w_stride, t, detA);
        comp_add(acc, es.wt[i * es.wt_stride] * mu_value<double>(KIND, t, delta));
        mn = fmin(mn, detA);
    }
    block_reduce_store(acc, mn, part_s, part_c, part_m, out);
}

// Single-CTA final pass over the partials, in the order of the sum that
// block_reduce_store ends with (256 threads).
__global__ void reduce_finalize_kernel(const double* part_s, const double* part_c, const double* part_m, int n,
                                       double* out_e, double* out_m)
{
    reduce_partials(part_s, part_c, part_m, n, out_e, out_m);
}

// Adds the whole-sample directional total to a finished energy report
// (src/directional.hpp:281-299, src/sweep.hpp:1921): one CTA, compensated,
// fixed order, so the reported energy is the composed objective.
template <int D>
__global__ void soft_energy_add_kernel(const SoftTerm* __restrict__ terms, int64_t n, double eps,
                                       const double* __restrict__ X, double* out_e)
{
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const SoftTerm t = terms[i];
        double p[4][3];
        soft_load<D>(t, X, p);
        comp_add(acc, soft_energy<D>(t, p, eps));
    }
    if (block_reduce(acc, mn)) { *out_e += acc.s + acc.c; }
}

// Per-mesh directional totals of a batch: CTA m adds the sum over terms
// [seg[m], seg[m+1]) to out[2m], the mesh's reported energy.
template <int D>
__global__ void soft_energy_add_seg_kernel(const SoftTerm* __restrict__ terms, const int64_t* __restrict__ seg,
                                           double eps, const double* __restrict__ X, double* out)
{
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    for (int64_t i = seg[blockIdx.x] + threadIdx.x; i < seg[blockIdx.x + 1]; i += blockDim.x) {
        const SoftTerm t = terms[i];
        double p[4][3];
        soft_load<D>(t, X, p);
        comp_add(acc, soft_energy<D>(t, p, eps));
    }
    if (block_reduce(acc, mn)) { out[2 * int64_t(blockIdx.x)] += acc.s + acc.c; }
}

// Segmented final pass: CTA m folds partials [m n, (m+1) n) into
// out[2m] = energy and out[2m+1] = min det of segment m.
__global__ void reduce_finalize_seg_kernel(const double* part_s, const double* part_c,
                                           const double* part_m, int n, double* out)
{
    const int64_t base = int64_t(blockIdx.x) * n;
    Comp acc {0.0, 0.0};
    double mn = INFINITY;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        acc = comp_merge(acc, Comp {part_s[base + i], part_c[base + i]});
        mn = fmin(mn, part_m[base + i]);
    }
    if (block_reduce(acc, mn)) {
        out[2 * int64_t(blockIdx.x)] = acc.s + acc.c;
        out[2 * int64_t(blockIdx.x) + 1] = mn;
    }
}

}  // namespace egg_b200
