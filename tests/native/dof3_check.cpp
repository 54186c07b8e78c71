// Checks the grouped 3D forms that the sweep kernels run (egg_b200/csrc/dof3.cuh,
// compiled for the host) on the patch of one DOF, against extended precision:
// stretched boxes in every axis order, and sheared cells whose edges lie near
// one line.  The yardstick is the plain evaluation of metric3.cuh, one sample
// at a time, in the same precision.
//
// Prints one line per check: its name, the cells' index, the objective, then
// median and 99th percentile of the grouped form's error, and the same two of
// the plain form's.
//   step32, step64   Newton step, over the shortest spacing
//   grad32, grad64   gradient, over the sum of the samples' gradient lengths
//   line32           summed metric change of a trial, over the sum of its
//                    samples' changes (plain: dmu3)
//   trial64          energy of a trial, over the energy
// A line "same NAME DIFF" per precision gives the largest difference between
// the gradient with and without the Hessian sums.
#include <math.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "dof3.cuh"

using namespace egg_b200;
using Ext = long double;

namespace egg_b200
{
template <> struct Tol<long double> {
    static constexpr long double energy = 1e-12L;
    static constexpr long double znorm = 1e-30L;
};
}  // namespace egg_b200

struct W {
    static constexpr int N = 27, S0 = 9, S1 = 3, S2 = 1;
};
constexpr int kP = 13;

struct Patch {
    double P[3 * W::N];
    float fe[9 * W::N];
    void edges()
    {
        const int st[3] = {9, 3, 1};
        for (int id = 0; id < 27; ++id) {
            const int at[3] = {id / 9, (id / 3) % 3, id % 3};
            for (int k = 0; k < 3; ++k) {
                for (int i = 0; i < 3; ++i) {
                    fe[(3 * k + i) * 27 + id] = at[k] < 2 ? float(P[i * 27 + id + st[k]] - P[i * 27 + id]) : 0.0f;
                }
            }
        }
    }
};

// The plain forms, sample by sample, over the 32 samples that move the DOF.
// R = float reads the fp32 edges.
template <class R> struct Plain {
    R g[3] = {0, 0, 0}, h[6] = {0, 0, 0, 0, 0, 0}, e = 0;
    double gsum = 0.0;
};

template <class R, class F> void each_sample(const Patch& p, F f)
{
    const int st[3] = {9, 3, 1};
    for (int cell = 0; cell < 8; ++cell) {
        const int a = 7 - cell;
        const int base = (cell >> 2) * 9 + ((cell >> 1) & 1) * 3 + (cell & 1);
        for (int r = 0; r < 4; ++r) {
            const int b = r == 0 ? a : (a ^ (4 >> (r - 1)));
            R t[9], v[3];
            for (int k = 0; k < 3; ++k) {
                const int c = b & ~(4 >> k);
                const int lo = base + (c >> 2) * 9 + ((c >> 1) & 1) * 3 + (c & 1);
                for (int i = 0; i < 3; ++i) {
                    t[3 * i + k] = sizeof(R) == 4 ? R(p.fe[(3 * k + i) * 27 + lo])
                                                  : R(p.P[i * 27 + lo + st[k]]) - R(p.P[i * 27 + lo]);
                }
                const R sk = (b & (4 >> k)) ? R(-1) : R(1);
                v[k] = r == 0 ? -sk : (k == r - 1 ? sk : R(0));
            }
            f(t, v);
        }
    }
}

template <class R> Plain<R> plain(const Patch& p, int kind, R delta)
{
    Plain<R> o;
    each_sample<R>(p, [&](const R* t, const R* v) {
        Shared3<R> S;
        shared3<R>(kind, t, delta, S);
        R g[3], h[6];
        role3<R>(kind, S, v, g, h);
        o.e += mu3_from<R>(kind, S);
        for (int q = 0; q < 3; ++q) { o.g[q] += g[q]; }
        for (int q = 0; q < 6; ++q) { o.h[q] += h[q]; }
        o.gsum += std::sqrt(double(g[0] * g[0] + g[1] * g[1] + g[2] * g[2]));
    });
    return o;
}

struct Err {
    std::vector<double> v[2];
    void add(double grouped, double pl)
    {
        v[0].push_back(grouped);
        v[1].push_back(pl);
    }
    void print(const char* name, int cells, int kind)
    {
        std::printf("%s %d %d", name, cells, kind);
        for (auto& x : v) {
            std::sort(x.begin(), x.end());
            std::printf(" %.3e %.3e", x[x.size() / 2], x[x.size() * 99 / 100]);
        }
        std::printf("\n");
    }
};

template <class A, class B> double dist(const A* a, const B* b)
{
    double s = 0.0;
    for (int q = 0; q < 3; ++q) { s += double(Ext(a[q]) - Ext(b[q])) * double(Ext(a[q]) - Ext(b[q])); }
    return std::sqrt(s);
}

static double g_same[2] = {0.0, 0.0};

template <int KIND> void run(int cells, const double L[3], bool shear, int n)
{
    std::mt19937_64 rng(17 + cells);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    const double h = std::min(L[0], std::min(L[1], L[2]));
    const double vol = shear ? 1e-3 : L[0] * L[1] * L[2];
    // shape+size measures against a target of det 1: scale the cells to it
    const double unit = KIND == kShapeSize ? 1.0 / std::cbrt(vol) : 1.0;
    const double delta = KIND == kUntangle ? 0.3 * vol : 0.0;
    Err step32, step64, grad32, grad64, line32, trial64;
    for (int it = 0; it < n; ++it) {
        Patch p;
        // sheared: columns (1, 0, 0), (1, e, 0), (1, 0, e) plus noise of 0.2 e
        const double e = 0.03;
        for (int id = 0; id < 27; ++id) {
            const double at[3] = {double(id / 9 - 1), double((id / 3) % 3 - 1), double(id % 3 - 1)};
            for (int i = 0; i < 3; ++i) {
                double x = L[i] * at[i] + 0.2 * h * U(rng);
                if (shear) {
                    x = (i == 0 ? at[0] + at[1] + at[2] : e * at[i]) + 0.1 * e * U(rng);
                }
                p.P[i * 27 + id] = unit * x;
            }
        }
        p.edges();
        const double hu = unit * (shear ? e : h);
        const Plain<Ext> x = plain<Ext>(p, KIND, Ext(delta));
        const Plain<double> d = plain<double>(p, KIND, delta);
        const Plain<float> f = plain<float>(p, KIND, float(delta));
        Ext sx[3];
        double sd[3], s64[3], g64[3], h64[6], e64;
        float sf[3], s32[3], g32[3], h32[6];
        solve3<Ext>(x.h, x.g, sx);
        solve3<double>(d.h, d.g, sd);
        solve3<float>(f.h, f.g, sf);
        const EdgeD<W::N> ED {p.P};
        const EdgeF<W::N> EF {p.fe};
        dof3_system<W, KIND, 1, false>(ED, kP, 0, delta, g64, h64, e64);
        dof3_system<W, KIND, false>(EF, kP, float(delta), g32, h32);
        solve3<double>(h64, g64, s64);
        solve3<float>(h32, g32, s32);
        step64.add(dist(s64, sx) / hu, dist(sd, sx) / hu);
        grad64.add(dist(g64, x.g) / x.gsum, dist(d.g, x.g) / x.gsum);
        double go[3], ho[6], eo;
        dof3_system<W, KIND, 1, true>(ED, kP, 0, delta, go, ho, eo);
        g_same[1] = std::fmax(g_same[1], dist(go, g64) / x.gsum);
        // a trial of a quarter step
        const double d64[3] = {0.25 * double(sx[0]), 0.25 * double(sx[1]), 0.25 * double(sx[2])};
        const float df[3] = {float(d64[0]), float(d64[1]), float(d64[2])};
        Patch q = p;
        for (int i = 0; i < 3; ++i) { q.P[i * 27 + kP] += d64[i]; }
        double md = INFINITY;
        const double moved[3] = {q.P[kP] - p.P[kP], q.P[27 + kP] - p.P[27 + kP], q.P[54 + kP] - p.P[54 + kP]};
        const double et = dof3_trial<W, KIND, 1>(ED, kP, 0, moved, delta, md);
        const Plain<Ext> xt = plain<Ext>(q, KIND, Ext(delta));
        const Plain<double> dt = plain<double>(q, KIND, delta);
        const double scale = std::fabs(double(xt.e)) + 32.0;
        trial64.add(std::fabs(double(Ext(et) - 32 - xt.e)) / scale, std::fabs(double(Ext(dt.e) - xt.e)) / scale);
        if (shear) { continue; }  // the fp32 path leaves such cells to fp64
        step32.add(dist(s32, sx) / hu, dist(sf, sx) / hu);
        grad32.add(dist(g32, x.g) / x.gsum, dist(f.g, x.g) / x.gsum);
        float gf[3], hf[6];
        dof3_system<W, KIND, true>(EF, kP, float(delta), gf, hf);
        g_same[0] = std::fmax(g_same[0], dist(gf, g32) / x.gsum);
        // metric changes of the same trial, from the fp32 edges
        Ext ref = 0;
        double sum = 0.0;
        float pl = 0.0f;
        each_sample<float>(p, [&](const float* t, const float* v) {
            Ext tx[9], dx[9], dn;
            float dt9[9], dnf;
            for (int i = 0; i < 3; ++i) {
                for (int k = 0; k < 3; ++k) {
                    tx[3 * i + k] = t[3 * i + k];
                    dt9[3 * i + k] = df[i] * v[k];
                    dx[3 * i + k] = dt9[3 * i + k];
                }
            }
            const Ext m = dmu3<Ext>(KIND, tx, dx, Ext(delta), dn);
            ref += m;
            sum += std::fabs(double(m));
            pl += dmu3<float>(KIND, t, dt9, float(delta), dnf);
        });
        float mdf = INFINITY, low = INFINITY;
        unsigned guard = 0u;
        const float ds = dof3_line<W, KIND, false>(EF, kP, df, float(delta), mdf, low, guard);
        line32.add(std::fabs(double(Ext(ds) - ref)) / sum, std::fabs(double(Ext(pl) - ref)) / sum);
    }
    step64.print("step64", cells, KIND);
    grad64.print("grad64", cells, KIND);
    trial64.print("trial64", cells, KIND);
    if (shear) { return; }
    step32.print("step32", cells, KIND);
    grad32.print("grad32", cells, KIND);
    line32.print("line32", cells, KIND);
}

int main()
{
    const double sp[5][3] = {{1, 1, 1}, {1, 0.1, 0.1}, {1, 0.1, 0.01}, {1, 0.03, 0.03}, {1, 0.01, 0.01}};
    const int turn[3][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}};
    for (int c = 0; c < 5; ++c) {
        for (int t = 0; t < (c ? 3 : 1); ++t) {
            const double L[3] = {sp[c][turn[t][0]], sp[c][turn[t][1]], sp[c][turn[t][2]]};
            run<kShape>(3 * c + t, L, false, 1000);
            run<kUntangle>(3 * c + t, L, false, 1000);
            run<kShapeSize>(3 * c + t, L, false, 1000);
        }
    }
    const double one[3] = {1, 1, 1};
    run<kShape>(15, one, true, 1000);
    run<kUntangle>(15, one, true, 1000);
    std::printf("same grad32 %.3e\nsame grad64 %.3e\n", g_same[0], g_same[1]);
    return 0;
}
