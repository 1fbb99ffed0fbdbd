// bmc_sym.cuh -- one event's exponential by one thread, for generators of up to 7 x 7 (at most one CEST pool).
//
// In the frame turned by the RF phase and in coordinates scaled by d = sqrt(f) per pool (detailed balance: exchange k
// sqrt(f) both ways), the generator equals its own transpose with the signs of the y entries flipped,
//     A[j][i] = sig(i, j) A[i][j],   sig = -1 where exactly one of i, j is a y entry:
// precession and nutation couple y antisymmetrically to x and z, all else is symmetric. Its exponential inherits that,
// and so does the symmetric part of the Frechet derivative H = L(X, v lam^T), which is all that a trace with the
// derivative of such a generator sees. So N (N + 1) / 2 numbers hold a matrix: 28 for one pool, few enough for a thread's
// registers, and a squaring costs 28 x 7 fused multiply-adds (and 28 x 14 for H), without shared memory, shuffles or
// idle lanes.
#pragma once
#include "bmc_chain.cuh"

namespace bmc {

template <int NC>
struct Sym {
    using D0 = Dn<double, 0>;
    using C0 = Chain<NC, double, 0>;
    using L = Layout<NC>;
    static constexpr int N = L::N, P1 = NC + 1;               // entries per axis
    static constexpr bool kFits = NC <= 1;
    static constexpr int X0 = 0, Y0 = P1, Z0 = 2 * P1, M0 = N - 1;

    static constexpr __device__ bool is_y(int i) { return i >= Y0 && i < Z0; }
    // a matrix: entries i <= j of t; the others by the sign
    struct Mat {
        double t[N][N];
        __device__ __forceinline__ double at(int i, int j) const {
            return i <= j ? t[i][j] : (is_y(i) != is_y(j) ? -t[j][i] : t[j][i]);
        }
    };

    // one event's generator and constant column, scaled by its duration over 2^s
    struct Gen {
        double R2w, R1w, offw, w1, km, Rm, cw, cm;
        double k[P1], R2[P1], R1[P1], off[P1], cc[P1];        // per CEST pool (index 0 .. NC - 1)
    };

    // the scale of each pool, and whether the pools have one (no negative fraction)
    static __device__ __forceinline__ bool scales(const double* params, int n_vox, int v, double (&sf)[P1], double& sfm) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const double f = params[(size_t)(L::CF + i) * n_vox + v];
            ok = ok && f >= 0.0;
            sf[i] = sqrt(fmax(f, 1e-30));
        }
        const double fm = params[(size_t)L::MF * n_vox + v];
        ok = ok && fm >= 0.0;
        sfm = sqrt(fmax(fm, 1e-30));
        return ok;
    }

    // from the chain's constants (whose k f are then k sqrt(f) twice); w1: the RF amplitude along x of the turned frame
    static __device__ __forceinline__ void gen(const ChainConst<NC, D0>& cc, const StepCoef<NC, D0>& sc, double w1,
                                               const double (&sf)[P1], double sfm, double h, Gen& g) {
        g.R2w = h * cc.Rw2.v;
        g.R1w = h * cc.Rw1.v;
        g.offw = h * sc.offw.v;
        g.w1 = h * w1;
        g.km = h * (cc.kmt.v * sfm);
        g.Rm = h * sc.Rm1W.v;
        g.cw = h * cc.cw.v;
        g.cm = h * (cc.cm.v / sfm);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            g.k[i] = h * (cc.k[i].v * sf[i]);
            g.R2[i] = h * cc.Rc2[i].v;
            g.R1[i] = h * cc.Rc1[i].v;
            g.off[i] = h * sc.offc[i].v;
            g.cc[i] = h * (cc.cc[i].v / sf[i]);
        }
    }

    // y = A v + C c
    static __device__ __forceinline__ void op(const Gen& g, const double (&v)[N], double c, double (&y)[N]) {
        double px = 0.0, py = 0.0, pz = fma(g.km, v[M0], g.cw * c);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const double x = v[X0 + 1 + i], w = v[Y0 + 1 + i], z = v[Z0 + 1 + i];
            px = fma(g.k[i], x, px);
            py = fma(g.k[i], w, py);
            pz = fma(g.k[i], z, pz);
            y[X0 + 1 + i] = fma(g.k[i], v[X0], -fma(g.R2[i], x, g.off[i] * w));
            y[Y0 + 1 + i] = fma(g.k[i], v[Y0], fma(g.off[i], x, fma(g.w1, z, -(g.R2[i] * w))));
            y[Z0 + 1 + i] = fma(g.k[i], v[Z0], fma(g.cc[i], c, -fma(g.R1[i], z, g.w1 * w)));
        }
        y[X0] = fma(g.offw, v[Y0], fma(-g.R2w, v[X0], px));
        y[Y0] = fma(g.w1, v[Z0], fma(-g.R2w, v[Y0], fma(-g.offw, v[X0], py)));
        y[Z0] = fma(-g.w1, v[Y0], fma(-g.R1w, v[Z0], pz));
        y[M0] = fma(g.km, v[Z0], fma(-g.Rm, v[M0], g.cm * c));
    }

    // T = F = exp - 1 of the generator's N x N block and phi its constant column's: Horner columns, then s squarings F <-
    // F F + 2 F (the slow modes' entries keep their digits, where squaring 1 + F doubles their error each time)
    static __device__ __forceinline__ void expm(const Gen& g, int s, const TaylorTable& tt, Mat& T, double (&phi)[N]) {
#pragma unroll
        for (int j = 0; j <= N; ++j) {
            double v[N];
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = i == j ? 1.0 : 0.0;
#pragma unroll 1
            for (int k = tt.dense_m; k >= 1; --k) {
                double y[N];
                op(g, v, j == N ? 1.0 : 0.0, y);
                const double ik = tt.inv_k[k];
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] = fma(ik, y[i], i == j && k > 1 ? 1.0 : 0.0);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (j == N) phi[i] = v[i];
                else if (i <= j) T.t[i][j] = v[i];
            }
        }
#pragma unroll 1
        for (int q = 0; q < s; ++q) square(T, phi);
    }

    static __device__ __forceinline__ void square(Mat& T, double (&phi)[N]) {
        Mat n;
        double p[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            p[i] = 2.0 * phi[i];
#pragma unroll
            for (int l = 0; l < N; ++l) p[i] = fma(T.at(i, l), phi[l], p[i]);
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = i; j < N; ++j) {
                double x = 2.0 * T.t[i][j];
#pragma unroll
                for (int l = 0; l < N; ++l) x = fma(T.at(i, l), T.at(l, j), x);
                n.t[i][j] = x;
            }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            phi[i] = p[i];
#pragma unroll
            for (int j = i; j < N; ++j) T.t[i][j] = n.t[i][j];
        }
    }

    // (T = F, phi) with the derivative along E = v lam^T, lam = e_zw: H (its symmetric part) and its augmented row h
    static __device__ __forceinline__ void expm_frechet(const Gen& g, int s, double scale, const double (&v0)[N],
                                                        const TaylorTable& tt, Mat& T, double (&phi)[N], Mat& H,
                                                        double (&h)[N]) {
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = i; j < N; ++j) H.t[i][j] = 0.0;
#pragma unroll
        for (int j = 0; j <= N; ++j) {
            double v[N], d[N], dN = 0.0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                v[i] = i == j ? 1.0 : 0.0;
                d[i] = 0.0;
            }
#pragma unroll 1
            for (int k = tt.dense_m; k >= 1; --k) {
                double y[N];
                const double ik = tt.inv_k[k];
                if (j < N) {
                    // the tangent column first: d <- (X d + C dN + E v) / k
                    op(g, d, dN, y);
                    const double dot = scale * v[Z0];
#pragma unroll
                    for (int i = 0; i < N; ++i) d[i] = ik * fma(dot, v0[i], y[i]);
                    dN = ik * dot;
                }
                op(g, v, j == N ? 1.0 : 0.0, y);
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] = fma(ik, y[i], i == j && k > 1 ? 1.0 : 0.0);
            }
            if (j == N) {
#pragma unroll
                for (int i = 0; i < N; ++i) phi[i] = v[i];
            } else {
                h[j < N ? j : 0] = dN;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    if (i <= j) T.t[i][j < N ? j : 0] = v[i];
                    // the symmetric part: entry (i, j) counts half towards itself and half towards (j, i)
                    if (i == j) H.t[i][i] = d[i];
                    else if (i < j) H.t[i][j < N ? j : 0] += 0.5 * d[i];
                    else H.t[j < N ? j : 0][i] += (is_y(i) != is_y(j) ? -0.5 : 0.5) * d[i];
                }
            }
        }
#pragma unroll 1
        for (int q = 0; q < s; ++q) {
            // H <- 2 H + F H + H F + sym(phi h^T), h <- 2 h + h F, then F and phi
            Mat n;
            double hn[N];
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = i; j < N; ++j) {
                    double x = fma(0.5 * phi[i], h[j], 2.0 * H.t[i][j]);
                    x = fma(is_y(i) != is_y(j) ? -0.5 : 0.5, phi[j] * h[i], x);
#pragma unroll
                    for (int l = 0; l < N; ++l) x = fma(T.at(i, l), H.at(l, j), fma(H.at(i, l), T.at(l, j), x));
                    n.t[i][j] = x;
                }
#pragma unroll
            for (int j = 0; j < N; ++j) {
                hn[j] = 2.0 * h[j];
#pragma unroll
                for (int l = 0; l < N; ++l) hn[j] = fma(h[l], T.at(l, j), hn[j]);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                h[i] = hn[i];
#pragma unroll
                for (int j = i; j < N; ++j) H.t[i][j] = n.t[i][j];
            }
            square(T, phi);
        }
    }

    // x <- R(-phase) x over the pools' (x, y) pairs
    static __device__ __forceinline__ void turn(double (&x)[N], double c, double s) {
#pragma unroll
        for (int i = 0; i < P1; ++i) {
            const double a = fma(c, x[X0 + i], s * x[Y0 + i]);
            x[Y0 + i] = fma(c, x[Y0 + i], -(s * x[X0 + i]));
            x[X0 + i] = a;
        }
    }
    // the scale of entry i
    static __device__ __forceinline__ double scale_of(const double (&sf)[P1], double sfm, int i) {
        if (i == M0) return sfm;
        const int p = i % P1;
        return p == 0 ? 1.0 : sf[p > 0 ? p - 1 : 0];
    }
};

// Entries of the scaled start state above this lose digits against the others (a pool with a start magnetisation far
// above its fraction); such chains, and those with a negative fraction, take the general path.
constexpr double kSymLargest = 1e3;
constexpr double kSymLeastFraction = 1e-9;     // of a fraction that is a tangent

// M <- exp(X) [M; 1] by the chain's own thread; false (M untouched) where the chain has to take the general path. Replaces
// the dense path's rounds of 8 lanes per chain: 600,000 chains of a one-pool dictionary (1 s CW block with MT each) took 2.2
// ms in the chain kernel that way, 1.0 ms this way.
template <int NC>
__device__ __noinline__ bool sym_event(const double* params, int n_vox, int v, const ChainConst<NC, Dn<double, 0>>& cc,
                                       const StepCoef<NC, Dn<double, 0>>& sc, const EvRec<double>& rec, double nu,
                                       const TaylorTable& tt, State<NC, Dn<double, 0>>& M) {
    using SY = Sym<NC>;
    using C0 = Chain<NC, double, 0>;
    constexpr int N = SY::N;
    double sf[SY::P1], sfm;
    if (!SY::scales(params, n_vox, v, sf, sfm)) return false;
    double x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = C0::at(M, i).v;
    SY::turn(x, rec.c, rec.s);
    double big = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = x[i] / SY::scale_of(sf, sfm, i);
        big = fmax(big, fabs(x[i]));
    }
    const int s = nu > tt.dense_theta ? (int)ceil(log2(nu / tt.dense_theta)) : 0;
    if (!(big <= kSymLargest) || s > 200) return false;
    typename SY::Gen g;
    SY::gen(cc, sc, rec.w1 * cc.relb1.v, sf, sfm, ldexp(rec.dt, -s), g);
    typename SY::Mat T;
    double phi[N], y[N];
    SY::expm(g, s, tt, T, phi);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        y[i] = phi[i];
#pragma unroll
        for (int l = 0; l < N; ++l) y[i] = fma(T.at(i, l), x[l], y[i]);
        y[i] += x[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) y[i] *= SY::scale_of(sf, sfm, i);
    SY::turn(y, rec.c, -rec.s);
#pragma unroll
    for (int i = 0; i < N; ++i) C0::at(M, i).v = y[i];
    return true;
}

// Every tangent of single-event chains (bmc_adjoint.cuh) with a thread per chain: z, and with kTan dz_p =
// tr(dX_p H) + h . dC_p + (exp(X)^T lam) . dv_p in the turned and scaled coordinates, whose scales move with the
// fractions (dc = dk d + k dd, dv = dm0 / d - v dd / d). A chain that cannot take this form clears done[chain]; the
// group kernel then takes it.
// Bound by the FP64 pipe (28 x 21 multiply-adds a squaring with tangents, 254 registers, 8 warps per SM): 30 iterations over
// 2,048 voxels x 244 rows took 27.9 ms of primal passes in the group kernel and 8.3 ms here, 21.9 and 8.1 ms of tangent
// passes (with the active chains packed, bmc_impl.cu).
template <int NC, bool kTan>
__global__ void __launch_bounds__(128, kTan ? 2 : 3)
sym_kernel(const ChainArgs a, const int* __restrict__ row_ev, int n_tan, const __grid_constant__ TaylorTable tt,
           unsigned char* __restrict__ done) {
    using SY = Sym<NC>;
    using D0 = Dn<double, 0>;
    using D1 = Dn<double, 1>;
    using C0 = Chain<NC, double, 0>;
    using C1 = Chain<NC, double, 1>;
    using L = Layout<NC>;
    constexpr int N = SY::N, P1 = SY::P1, X0 = SY::X0, Y0 = SY::Y0, Z0 = SY::Z0, M0 = SY::M0;
    const long long nch = (long long)a.n_vox * a.n_off;
    long long ci = (long long)blockIdx.x * 128 + threadIdx.x;
    if (ci >= (a.live ? *a.live : nch)) return;
    if (a.order) ci = a.order[ci];
    const int v = (int)(ci / a.n_off), o = (int)(ci % a.n_off);
    if (a.active && a.active[v] == 0) return;
    const size_t ch = (size_t)ci;
    const EvRec<double> rec = reinterpret_cast<const EvRec<double>*>(a.ev)[(size_t)row_ev[o] * a.n_off + o];
    double sf[P1], sfm;
    bool ok = SY::scales(a.params, a.n_vox, v, sf, sfm);
    double v0[N], big = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) v0[i] = a.m0[(size_t)v * N + i];
    SY::turn(v0, rec.c, rec.s);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        v0[i] = v0[i] / SY::scale_of(sf, sfm, i);
        big = fmax(big, fabs(v0[i]));
    }
    ok = ok && big <= kSymLargest;
    if constexpr (kTan) {
        // a derivative along a fraction divides by its scale
        for (int p = 0; p < n_tan; ++p) {
            const int fr = a.field_row[p];
            if ((fr >= L::CF && fr < L::CF + NC) || fr == L::MF)
                ok = ok && a.params[(size_t)fr * a.n_vox + v] >= kSymLeastFraction;
        }
    }
    for (int node = 0; node < a.n_nodes && ok; ++node) {
        ChainConst<NC, D0> cc;
        C0::load_const(a, v, node, cc);
        Dn<double, 3> g3 = dconst<double, 3>(0.0);
        if (cc.mt_on && cc.ls != 0 && rec.w1 != 0.0) {
            const D0 offmt = (rec.wf - cc.dw0) - cc.dwmt;
            if constexpr (kTan) {
                Dn<double, 3> off3 = dconst<double, 3>(offmt.v), t23 = dconst<double, 3>(cc.t2mt.v),
                              w03 = dconst<double, 3>(cc.w0sl.v);
                off3.d[0] = t23.d[1] = w03.d[2] = 1.0;
                g3 = cc.ls == 1 ? lorentzian<double, 3>(off3, t23) : super_lorentzian<double, 3>(off3, t23, w03);
            } else {
                g3.v = (cc.ls == 1 ? lorentzian<double, 0>(offmt, cc.t2mt)
                                   : super_lorentzian<double, 0>(offmt, cc.t2mt, cc.w0sl)).v;
            }
        }
        StepCoef<NC, D0> sc;
        C0::event_coef(cc, rec, D0{g3.v}, sc);
        const double nu = rec.dt * C0::coef_norm(sc, cc);
        const int s = nu > tt.dense_theta ? (int)ceil(log2(nu / tt.dense_theta)) : 0;
        if (!(nu < INFINITY) || s > 200) {     // the general path flags these
            ok = false;
            break;
        }
        const double h = ldexp(rec.dt, -s);
        typename SY::Gen g;
        SY::gen(cc, sc, rec.w1 * cc.relb1.v, sf, sfm, h, g);
        typename SY::Mat T, H;
        double phi[N], hr[N];
        if constexpr (kTan) SY::expm_frechet(g, s, ldexp(1.0, -s), v0, tt, T, phi, H, hr);
        else SY::expm(g, s, tt, T, phi);
        const double wgt = a.n_nodes > 1 ? a.w[node] : 1.0;
        double z = phi[Z0];
#pragma unroll
        for (int j = 0; j < N; ++j) z = fma(T.at(Z0, j), v0[j], z);
        z += v0[Z0];
        a.out[ch] = (node ? a.out[ch] : 0.0) + wgt * z;
        if (a.work) {
            atomicAdd(a.work + 1, (unsigned long long)((N + 1) * tt.dense_m));
            atomicAdd(a.work + 2, (unsigned long long)s);
        }
        if constexpr (kTan) {
#pragma unroll 1
            for (int p = 0; p < n_tan; ++p) {
                ChainConst<NC, D1> cp;
                C1::load_const(a, v, node, cp, p);
                D1 gm = dconst<double, 1>(g3.v);
                if (cp.mt_on && cp.ls != 0 && rec.w1 != 0.0) {
                    const D1 offmt = (rec.wf - cp.dw0) - cp.dwmt;
                    gm.d[0] = fma(g3.d[0], offmt.d[0], fma(g3.d[1], cp.t2mt.d[0], g3.d[2] * cp.w0sl.d[0]));
                }
                EvRec<double> rx = rec;
                rx.c = 1.0;
                rx.s = 0.0;
                StepCoef<NC, D1> sp;
                C1::event_coef(cp, rx, gm, sp);
                const double dw = sp.w1x.d[0];
                // tr(dA H) over the generator's entries, (i, j) against (j, i)
                double x = -sp.Rw2.d[0] * (H.at(X0, X0) + H.at(Y0, Y0));
                x = fma(-sp.Rw1.d[0], H.at(Z0, Z0), x);
                x = fma(sp.offw.d[0], H.at(Y0, X0) - H.at(X0, Y0), x);
                x = fma(dw, H.at(Z0, Y0) - H.at(Y0, Z0), x);
                x = fma(-sp.Rm1W.d[0], H.at(M0, M0), x);
                const double dfm = C1::field(a, L::MF, v, p).d[0], dsm = dfm / (2.0 * sfm);
                x = fma(fma(cp.kmt.d[0], sfm, cp.kmt.v * dsm), H.at(M0, Z0) + H.at(Z0, M0), x);
                // C: r1 d per pool
                double y = fma(cp.cw.d[0], hr[Z0], (cp.cm.d[0] / sfm - cp.cm.v * dsm / (sfm * sfm)) * hr[M0]);
                double dd[P1];                                // dd / d per pool
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    const int xi = X0 + 1 + i, yi = Y0 + 1 + i, zi = Z0 + 1 + i;
                    const double ds = C1::field(a, L::CF + i, v, p).d[0] / (2.0 * sf[i]);
                    dd[i] = ds / sf[i];
                    const double dk = fma(cp.k[i].d[0], sf[i], cp.k[i].v * ds);
                    x = fma(dk, (H.at(X0, xi) + H.at(xi, X0)) + (H.at(Y0, yi) + H.at(yi, Y0)) +
                                    (H.at(Z0, zi) + H.at(zi, Z0)), x);
                    x = fma(-sp.Rc2[i].d[0], H.at(xi, xi) + H.at(yi, yi), x);
                    x = fma(-sp.Rc1[i].d[0], H.at(zi, zi), x);
                    x = fma(sp.offc[i].d[0], H.at(xi, yi) - H.at(yi, xi), x);
                    x = fma(dw, H.at(zi, yi) - H.at(yi, zi), x);
                    y = fma(cp.cc[i].d[0] / sf[i] - cp.cc[i].v * dd[i] / sf[i], hr[zi], y);
                }
                double r = rec.dt * (x + y);
                // the start state's derivative, turned and scaled, and the scales'
                double dv[N];
#pragma unroll
                for (int i = 0; i < N; ++i) dv[i] = a.dm0 ? a.dm0[((size_t)p * a.n_vox + v) * N + i] : 0.0;
                SY::turn(dv, rec.c, rec.s);
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const int pool = i == M0 ? 0 : i % P1;
                    const double e = i == M0 ? dsm / sfm : (pool ? dd[pool > 0 ? pool - 1 : 0] : 0.0);
                    const double u = T.at(Z0, i) + (i == Z0 ? 1.0 : 0.0);
                    r = fma(u, dv[i] / SY::scale_of(sf, sfm, i) - v0[i] * e, r);
                }
                double* jp = a.jout + (size_t)p * nch + ch;
                *jp = (node ? *jp : 0.0) + wgt * r;
            }
        }
    }
    done[ch] = ok ? 1 : 0;
    if (!ok) atomicOr(a.left, 1);
}

}  // namespace bmc
