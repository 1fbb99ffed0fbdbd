// bmc_chain.cuh -- the chain kernel: one thread per (voxel, offset), the whole event table.
//
// Semantics follow BMC-JAX simulation/simulate.py:22-132 exactly:
//   * an event evolves the state only if dt > 1e-9 (simulate.py:51);
//   * GRADIENT and SPOILER zero the x and y entries of water and every CEST pool (simulate.py:55-72);
//   * last_M is the state after every event; after an ADC the running state returns to M0
//     (simulate.py:105-114); the result is last_M after the final event (simulate.py:128-132).
// The time step is exp([A C; 0 0] h)^s [M; 1]; see bmc_device.cuh for how it is evaluated.
#pragma once
#include <type_traits>

#include "bmc_device.cuh"
#include "bmc_tail32.cuh"

namespace bmc {

constexpr int kMaxNodes = 64;
constexpr int kMaxT = 8;
constexpr int kTaylorMMax = 40;

// Truncated-Taylor tables, filled by the host (bmc_capi.cu) for the precision in use:
// theta[m] = the largest ||X|| for which the degree-m tail bound stays under the tolerance.
struct TaylorTable {
    double theta[kTaylorMMax + 1];
    double inv_fact[kTaylorMMax + 1];   // 1 / k!
    double inv_k[kTaylorMMax + 1];      // 1 / k
    int m_max;             // short path: degree cap
    double dense_theta;    // dense path: ||X / 2^s|| <= dense_theta ...
    int dense_m;           // ... with this Horner degree
    double dense_switch;   // warps whose largest ||X|| exceeds this take the dense path
    // float64 kernels: for a chain of Taylor degree m, the terms from f32_from[m] on are below the
    // table's float32 threshold of the state (theta[m]^k / k! <= 1e-6 for BMC_F64, 0.3 for BMC_MIXED)
    // and are formed in float32 (> m: none)
    int f32_from[kTaylorMMax + 1];
    float inv_fact_f[kTaylorMMax + 1];  // 1 / k! in float32
};

// A row's unit of a shaped-pulse train (bmc_train.cuh): the reference pulse (first event, samples), the gap events
// it takes in, how many equal units are applied at each mark (run) and the events those cover (span). n = 0: the
// row has no train.
struct TrainRow {
    int first, n, gap, run;
    int span;
    int mirrored;              // the pulse's shape is its own mirror image
    double w_max;
};
constexpr int kTrainMark = 8;  // added to the type of a record where a unit begins
// a chain of a table that was looked over for trains: it has its propagator, its row has no train, or the row has one but
// the chain is beyond the propagator's bounds (it takes its events one by one)
constexpr int kTrained = 1, kPlain = 2, kRefused = 4, kEveryPart = 7;

struct ChainArgs {
    int n_vox, n_off, n_ev, n_fields;
    int mz;                    // state index written; < 0: whole state
    int reset_after_adc;
    int n_nodes;               // spread isochromats (1 = none)
    double u[kMaxNodes], w[kMaxNodes];
    const double* params;      // [n_fields][n_vox]
    const double* params_dir;  // [n_fields][n_vox] or null: the design direction of params (design kernel)
    const void* ev;            // EvRec<R>[n_ev][n_off]
    const double* m0;          // [n_vox][N]
    const double* sigma;       // [n_vox] spread width [Hz] or null
    // tangents handled by this launch: global tangent indices t0 .. t0 + NT - 1
    int t0;
    int n_tan;                 // tangents of the whole set (node_jout's layout)
    int field_row[kMaxT];
    const double* seed;        // [P][n_vox]
    const double* dm0;         // [P][n_vox][N] or null
    const int* active;         // [n_vox] or null: voxels with 0 are skipped
    const int* order;          // [n_vox * n_off] or null: the chain each thread takes, in launch order
    double* out;               // [n_vox][n_off] (mz >= 0) or [n_vox][n_off][N]
    double* jout;              // [P][n_vox][n_off] or null
    double* traj;              // [n_vox][n_off][n_ev][N] or null: the state after every event
    int* status;               // error flags (bit 0: non-finite norm)
    unsigned long long* work;  // null, or [5]: useful Taylor terms, dense Horner column products,
                               // dense squarings, Taylor terms executed (warp maximum), and of the
                               // useful Taylor terms those formed in float32
    // uneven batches (chain_kernel<..., true>): every voxel has its own event table
    long long n_chains;        // chains of the launch (canonical order: voxel-major, then row)
    const int2* chain_map;     // [n_chains]: (voxel, row of its table)
    const int* vox_table;      // [n_vox]: table of each voxel
    const long long* tab_base; // [n_tables]: first record of each table in `ev`
    const int* tab_noff;       // [n_tables]: rows (records per event) of each table
    const int* tab_nev;        // [n_tables]: events of each table
    // repeated blocks (propagator reuse): per row (a, L, r, 0), the r copies of the L events from event a
    // on are applied as one propagator; r < 2: none. Uniform tables: row o; uneven: tab_row0[t] + o.
    const int4* seg;           // null: no reuse
    const int* tab_row0;       // [n_tables]: first row of each table in `seg` (uneven batches)
    double dense_switch;       // > 0: the norm above which an event takes the dense path (else the table's)
    int cpw;                   // chains per warp: lanes from cpw on have none (chains_per_warp below)
    // Isochromats as chains of their own (chain kernel): node j of chain c is chain j * chains + c of the launch,
    // and its weighted results go to node_out [node][chains (x N)] and node_jout [node][P][chains]; node_sum_kernel
    // adds them in node order. Null node_out: every chain loops over its nodes.
    double* node_out;
    double* node_jout;
    int node_lo, node_hi;      // with a null node_out: the nodes of this launch (from 1 on added to the output)
    // Part of the launch order (uniform tables; chain_count 0: all): chains first_chain .. first_chain + chain_count
    long long first_chain, chain_count;
    // Shaped pulses (train null: none were looked for): the rows' trains, the propagators of those chains, applied at the
    // marked records, which of them have one, and the chains that this launch takes (kTrained, kPlain, kRefused)
    const TrainRow* train;     // [n_off]
    const double* prop;
    const unsigned char* prop_ok;
    int parts;
    const int* kinds;          // what the table and the chains so far have of the three (a launch without work ends)
    // adjoint passes: the chains that the thread kernel (bmc_sym.cuh) has taken, and whether it left any
    unsigned char* done;       // [n_vox * n_off] or null
    int* left;
    const int* live;           // null, or how many entries of `order` the pass takes (the active voxels' chains)
};

// Chains per warp of a launch: 32, or as many fewer as still leave the launch's warps resident at once. A launch
// of few chains is bound by the latency of one warp, which grows with its lanes: their dense events are taken a
// group of lanes at a time, one round after another, and their Taylor degrees differ. One spectrum of 61 chains (2 s
// CW, two pools and MT) took 292 us in the kernel with 32 chains per warp, 83 us with one. The chain kernel counts
// one block per SM as resident: its unrolled term loops stream from the instruction cache, and 714 chains (a fit of
// 100-sample trains) in 2 chains per warp on 90 blocks took 49.7 ms of tangent passes, in 1 per warp on 179 blocks, two
// on some SMs, 76.6 (32 per warp: 53.0). A power of two from `least` (the chains a warp's lane groups take at once) to
// `most`: 32, or 16 for the adjoint passes of up to kFewWaves waves of warps (adjoint_chains_per_warp), whose last wave
// is then less empty: 93,452 chains of four pools and MT (ten passes of each kind) took 21.0 ms of tangent and 9.9 ms of primal
// passes at 32, 20.1 and 8.9 at 16, 20.4 and 9.7 at 8 (2.5 waves); 292,800 such chains (7.7 waves) fit 1% faster at 32.
constexpr int kSMs = 148;
constexpr int kFewWaves = 4;
inline int chains_per_warp(long long chains, int blocks_per_sm, int warps, int least, int most = 32) {
    int c = most;
    const long long slots = (long long)kSMs * blocks_per_sm * warps;
    while (c > least && (chains + c / 2 - 1) / (c / 2) <= slots) c /= 2;
    return c;
}
inline int adjoint_chains_per_warp(long long chains, int blocks_per_sm, int warps, int least) {
    const bool few = chains <= 32ll * kSMs * blocks_per_sm * warps * kFewWaves;
    return chains_per_warp(chains, blocks_per_sm, warps, least, few ? 16 : 32);
}

template <int NC>
struct Layout {
    static constexpr int N = 3 * NC + 4;        // state size, reference layout
    static constexpr int NA = N + 1;            // augmented
    static constexpr int NF = 13 + 5 * NC;      // params rows
    // params rows (SimParams order, CEST fields expanded)
    static constexpr int WR1 = 0, WR2 = 1, WF = 2, CK = 3, CF = 3 + NC, CDW = 3 + 2 * NC, CR1 = 3 + 3 * NC,
                         CR2 = 3 + 4 * NC, MK = 3 + 5 * NC, MF = MK + 1, MDW = MK + 2, MR1 = MK + 3, MR2 = MK + 4,
                         MLS = MK + 5, B0 = MK + 6, GAM = MK + 7, B0I = MK + 8, RB1 = MK + 9;
    // reference state indices
    static constexpr int ixw = 0, iyw = NC + 1, izw = 2 * (NC + 1), izm = 3 * (NC + 1);
    static __device__ __forceinline__ int ixc(int i) { return 1 + i; }
    static __device__ __forceinline__ int iyc(int i) { return NC + 2 + i; }
    static __device__ __forceinline__ int izc(int i) { return 2 * NC + 3 + i; }
};

template <int NC, typename R, int NT>
struct Chain {
    using D = Dn<R, NT>;
    using L = Layout<NC>;
    static constexpr int N = L::N;
    static constexpr int NA = L::NA;

    // ---------------------------------------------------------------------------------------------
    // parameters -> per-chain constants (matrix.py:99-173), with tangents seeded per field row
    // ---------------------------------------------------------------------------------------------
    // tangents t0 .. t0 + NT - 1 of the launch's set (a.t0 in the chain kernel; the adjoint kernel seeds
    // one tangent per lane)
    static __device__ __forceinline__ D field(const ChainArgs& a, int row, int v, int t0) {
        D r = dconst<R, NT>(lift<R>(a.params, a.params_dir, (size_t)row * a.n_vox + v));
        if constexpr (NT > 0) {
#pragma unroll
            for (int t = 0; t < NT; ++t)
                if (a.field_row[t0 + t] == row) r.d[t] = R(a.seed[(size_t)(t0 + t) * a.n_vox + v]);
        }
        return r;
    }

    static __device__ void load_const(const ChainArgs& a, int v, int node, ChainConst<NC, D>& cc) {
        load_const(a, v, node, cc, a.t0);
    }

    static __device__ void load_const(const ChainArgs& a, int v, int node, ChainConst<NC, D>& cc, int t0) {
        const D r1w = field(a, L::WR1, v, t0), r2w = field(a, L::WR2, v, t0);
        const D b0 = field(a, L::B0, v, t0), gam = field(a, L::GAM, v, t0);
        D b0i = field(a, L::B0I, v, t0);
        const D larmor = R(1e6) * (gam * b0);
        if (a.n_nodes > 1 || a.sigma) {
            // isochromat `node`: b0_inhom + sigma u / (gamma b0 / 2 pi)   (spread.py:101-104)
            D sig = dconst<R, NT>(a.sigma ? R(a.sigma[v]) : R(0));
            if constexpr (NT > 0) {
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    if (a.field_row[t0 + t] == -2) sig.d[t] = R(a.seed[(size_t)(t0 + t) * a.n_vox + v]);
            }
            const D hzpp = R(1.0 / 6.283185307179586) * (gam * b0);
            b0i = b0i + (R(a.u[node]) * sig) / hzpp;
        }
        cc.dw0 = R(1e-6) * (larmor * b0i);
        D ksum = dconst<R, NT>(R(0));
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const D k = field(a, L::CK + i, v, t0), f = field(a, L::CF + i, v, t0);
            const D r1 = field(a, L::CR1 + i, v, t0), r2 = field(a, L::CR2 + i, v, t0);
            const D dw = field(a, L::CDW + i, v, t0);
            cc.k[i] = k;
            cc.kwc[i] = k * f;
            ksum = ksum + cc.kwc[i];
            cc.Rc2[i] = r2 + k;
            cc.Rc1[i] = r1 + k;
            cc.cc[i] = r1 * f;
            cc.offc0[i] = R(1e-6) * (dw * larmor);
        }
        const D kmt = field(a, L::MK, v, t0), fmt = field(a, L::MF, v, t0), r1mt = field(a, L::MR1, v, t0);
        const D r2mt = field(a, L::MR2, v, t0), dwmt = field(a, L::MDW, v, t0);
        cc.kmt = kmt;
        cc.kwmt = kmt * fmt;
        cc.Rm1 = r1mt + kmt;
        cc.cm = r1mt * fmt;
        cc.Rw2 = r2w + ksum;
        cc.Rw1 = (r1w + ksum) + cc.kwmt;
        cc.cw = r1w;
        cc.relb1 = field(a, L::RB1, v, t0);
        cc.dwmt = R(1e-6) * (dwmt * larmor);
        cc.t2mt = dconst<R, NT>(R(1)) / r2mt;
        cc.w0sl = R(1e-6) * larmor;
        int ls = (int)a.params[(size_t)L::MLS * a.n_vox + v];
        cc.ls = ls < 0 ? 0 : (ls > 2 ? 2 : ls);
        cc.mt_on = fmt.v > R(1e-9);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const double f = a.params[(size_t)(L::CF + i) * a.n_vox + v];
            cc.sf[i] = f > 1e-30 ? sqrt(f) : 1.0;
        }
        const double fm = a.params[(size_t)L::MF * a.n_vox + v];
        cc.sfm = fm > 1e-30 ? sqrt(fm) : 1.0;
    }

    // ---------------------------------------------------------------------------------------------
    // one event's coefficients (unscaled) and the infinity norm of its generator times dt
    // ---------------------------------------------------------------------------------------------
    static __device__ __forceinline__ void event_coef(const ChainConst<NC, D>& cc, const EvRec<R>& e, D g_mt,
                                                      StepCoef<NC, D>& sc) {
        const D offw = e.wf - cc.dw0;                                  // matrix.py:162
        const D w1 = e.w1 * cc.relb1;                                  // matrix.py:121
        sc.offw = offw;
        sc.w1x = e.c * w1;
        sc.w1y = e.s * w1;
        sc.Rw2 = cc.Rw2;
        sc.Rw1 = cc.Rw1;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            sc.k[i] = cc.k[i];
            sc.kwc[i] = cc.kwc[i];
            sc.Rc2[i] = cc.Rc2[i];
            sc.Rc1[i] = cc.Rc1[i];
            sc.offc[i] = cc.offc0[i] - offw;                           // matrix.py:166
        }
        sc.kmt = cc.kmt;
        sc.kwmt = cc.kwmt;
        sc.Rm1W = cc.Rm1 + (w1 * w1) * g_mt;                           // matrix.py:210, 283
    }

    // sqrt(a^2 + b^2) <= max + (sqrt(2) - 1) min, within 8.3%
    static __device__ __forceinline__ R hyp(R a, R b) { return fmax(a, b) + R(0.41421357) * fmin(a, b); }
    // sqrt(a^2 + b^2), rounded; the callers scale their result by (1 + kNormSlack) to keep a bound
    static __device__ __forceinline__ R blk(R a, R b) { return sqrt(fma(a, a, b * b)); }
    static constexpr double kNormSlack = std::is_same<R, float>::value ? 1e-6 : 1e-14;

    // An upper bound of ||D^-1 A D|| in the norm max_b ||v_b||_2 / d_b over blocks b = (x, y) pairs and
    // z entries, with d = sqrt(f) per pool. The similarity balances the exchange terms (detailed
    // balance: k f one way, k the other, so k sqrt(f) both ways) and each precession-relaxation block
    // counts sqrt(R^2 + w^2) instead of R + w (exactly in the part a chain keeps across events, through
    // the bound `hyp` for the RF term, which changes every event). Being an induced norm, it bounds
    // ||X^k|| and so the Taylor tail; the truncation error of water's entries stays below tol times
    // max(|M_w|, |M_c| / sqrt(f_c), 1).
    //
    // Every water and CEST row carries the RF term w1 once, so the bound is max(rows + w1, mt): `rows`
    // (those rows without w1) and the MT row's constant depend on the event's frequency, not on its RF
    // amplitude or phase, and a chain keeps them while its frequency stays the same (`NormBase`).
    struct NormBase {
        R rows;   // max over the water and CEST rows of their w1-free sums
        R mt_c;   // the MT row without |R1 + k + w1^2 g|
    };

    static __device__ __forceinline__ NormBase norm_base(const StepCoef<NC, D>& s, const ChainConst<NC, D>& cc) {
        // the constant column C enters through the augmented row: |C_i| / d_i
        R ex = R(0);
#pragma unroll
        for (int i = 0; i < NC; ++i) ex += fabs(s.k[i].v) * R(cc.sf[i]);
        const R km = fabs(s.kmt.v) * R(cc.sfm);
        R m = blk(s.Rw2.v, s.offw.v) + ex;
        m = fmax(m, fabs(s.Rw1.v) + ex + km + fabs(R(cc.cw.v)));
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const R b = fabs(s.k[i].v) * R(cc.sf[i]);
            m = fmax(m, blk(s.Rc2[i].v, s.offc[i].v) + b);
            m = fmax(m, fabs(s.Rc1[i].v) + b + fabs(R(cc.cc[i].v)) / R(cc.sf[i]));
        }
        return {m * R(1 + kNormSlack), (km + fabs(R(cc.cm.v)) / R(cc.sfm)) * R(1 + kNormSlack)};
    }

    static __device__ __forceinline__ R rf_norm(const NormBase& b, R w1x, R w1y, R Rm1W) {
        return fmax(b.rows + hyp(fabs(w1x), fabs(w1y)), fabs(Rm1W) + b.mt_c);
    }

    static __device__ __forceinline__ R coef_norm(const StepCoef<NC, D>& s, const ChainConst<NC, D>& cc) {
        return rf_norm(norm_base(s, cc), s.w1x.v, s.w1y.v, s.Rm1W.v);
    }

    // the RF entries of an event's coefficients, unscaled, computed as event_coef computes them
    static __device__ __forceinline__ void rf_coef(const ChainConst<NC, D>& cc, const EvRec<R>& e, D g_mt, D& w1x,
                                                   D& w1y, D& Rm1W) {
        const D w1 = e.w1 * cc.relb1;
        w1x = e.c * w1;
        w1y = e.s * w1;
        Rm1W = cc.Rm1 + (w1 * w1) * g_mt;
    }

    static __device__ __forceinline__ void scale_coef(StepCoef<NC, D>& s, R h) {
        s.Rw2 = h * s.Rw2; s.Rw1 = h * s.Rw1;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            s.k[i] = h * s.k[i]; s.kwc[i] = h * s.kwc[i]; s.Rc2[i] = h * s.Rc2[i];
            s.Rc1[i] = h * s.Rc1[i]; s.offc[i] = h * s.offc[i];
        }
        s.offw = h * s.offw; s.w1x = h * s.w1x; s.w1y = h * s.w1y;
        s.kmt = h * s.kmt; s.kwmt = h * s.kwmt; s.Rm1W = h * s.Rm1W;
    }

    // y = X v (+ C h when WithC): the sparse Bloch-McConnell operator (matrix.py:238-293)
    template <bool WithC>
    static __device__ __forceinline__ void matvec(const StepCoef<NC, D>& s, const State<NC, D>& v, State<NC, D>& y,
                                                  const ChainConst<NC, D>* cst = nullptr, R h = R(0)) {
        // water rows: own terms and the pools' exchange terms in two partial sums (shorter dependency
        // chains), pool rows: four terms each
        D xw = dfma(s.offw, v.yw, -(s.Rw2 * v.xw));
        xw = xw - s.w1y * v.zw;
        D yw = dfma(s.w1x, v.zw, -(s.Rw2 * v.yw));
        yw = yw - s.offw * v.xw;
        D zw = dfma(s.w1y, v.xw, -(s.Rw1 * v.zw));
        zw = zw - s.w1x * v.yw;
        D zm = dfma(s.kwmt, v.zw, -(s.Rm1W * v.zm));
        if constexpr (WithC) {                     // the constant column C h, rebuilt here: it is needed
            zw = dfma(cst->cw, dconst<R, NT>(h), zw);   // by the first term of a sub-step only
            zm = dfma(cst->cm, dconst<R, NT>(h), zm);
        }
        D px = dconst<R, NT>(R(0)), py = px, pz = s.kmt * v.zm;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            px = dfma(s.k[i], v.xc[i], px);
            py = dfma(s.k[i], v.yc[i], py);
            pz = dfma(s.k[i], v.zc[i], pz);
            D xc = dfma(s.kwc[i], v.xw, -(s.Rc2[i] * v.xc[i]));
            xc = xc - s.offc[i] * v.yc[i];
            xc = xc - s.w1y * v.zc[i];
            D yc = dfma(s.kwc[i], v.yw, -(s.Rc2[i] * v.yc[i]));
            yc = dfma(s.offc[i], v.xc[i], yc);
            yc = dfma(s.w1x, v.zc[i], yc);
            D zc = dfma(s.kwc[i], v.zw, -(s.Rc1[i] * v.zc[i]));
            zc = dfma(s.w1y, v.xc[i], zc);
            zc = zc - s.w1x * v.yc[i];
            if constexpr (WithC) zc = dfma(cst->cc[i], dconst<R, NT>(h), zc);
            y.xc[i] = xc;
            y.yc[i] = yc;
            y.zc[i] = zc;
        }
        y.xw = xw + px;
        y.yw = yw + py;
        y.zw = zw + pz;
        y.zm = zm;
    }

    static __device__ __forceinline__ void axpy_state(State<NC, D>& acc, const State<NC, D>& t) {
        acc.xw = acc.xw + t.xw; acc.yw = acc.yw + t.yw; acc.zw = acc.zw + t.zw; acc.zm = acc.zm + t.zm;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            acc.xc[i] = acc.xc[i] + t.xc[i]; acc.yc[i] = acc.yc[i] + t.yc[i]; acc.zc[i] = acc.zc[i] + t.zc[i];
        }
    }
    static __device__ __forceinline__ void scal_state(State<NC, D>& t, R a) {
        t.xw = a * t.xw; t.yw = a * t.yw; t.zw = a * t.zw; t.zm = a * t.zm;
#pragma unroll
        for (int i = 0; i < NC; ++i) { t.xc[i] = a * t.xc[i]; t.yc[i] = a * t.yc[i]; t.zc[i] = a * t.zc[i]; }
    }

    // acc += a * t, entry by entry
    static __device__ __forceinline__ void fma_state(State<NC, D>& acc, R a, const State<NC, D>& t) {
        acc.xw = dfma(dconst<R, NT>(a), t.xw, acc.xw); acc.yw = dfma(dconst<R, NT>(a), t.yw, acc.yw);
        acc.zw = dfma(dconst<R, NT>(a), t.zw, acc.zw); acc.zm = dfma(dconst<R, NT>(a), t.zm, acc.zm);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            acc.xc[i] = dfma(dconst<R, NT>(a), t.xc[i], acc.xc[i]);
            acc.yc[i] = dfma(dconst<R, NT>(a), t.yc[i], acc.yc[i]);
            acc.zc[i] = dfma(dconst<R, NT>(a), t.zc[i], acc.zc[i]);
        }
    }

    // exp(X)^s [M; 1] by s sub-steps of the degree-m Taylor polynomial, X = [A C; 0 0] h: the
    // unnormalised powers p_k = X^k [M; 1] are accumulated with weights 1/k!, so each term is one sparse
    // operator product and one fused multiply-add per state entry. The coefficients (scaled by h) are
    // formed at each sub-step, so that they are not held in registers across the rest of the event.
    // Every lane runs its own (ns, m): a chain's result never depends on which chains share its warp. Where the
    // lanes of a warp agree (cost-sorted warps mostly do) the loops do not diverge.
    //
    // In the float64 kernel without tangents, the terms of a chain from tt.f32_from[m] on (each below
    // 1e-6 of the state, in the balanced norm of coef_norm) are formed in float32 and summed in a float32
    // accumulator that is added to M once per sub-step: their rounding, a few units of 2^-24 of terms
    // below 1e-6, is at most ~2e-13 of the state per event, the order of the truncation tolerance.
    // The switch point is the chain's own too: the lanes leave the float64 loop at their own term and meet again
    // before the float32 loop, so a warp takes one pass per sub-step (its largest float64 count plus its largest
    // float32 count) however its switch points differ. Passing over the sub-step once per distinct switch point
    // instead cost a warp of 32 different offsets (one spectrum) up to ten passes: 1 voxel x 102 offsets x 4,041
    // events took 78.9 ms so, 22.1 ms in one pass (cost-sorted warps, 2,048 voxels: 90.5 against 92.8 ms).
    static __device__ __forceinline__ void taylor_apply(const ChainConst<NC, D>& cst, const EvRec<R>& rec, D g_mt,
                                                        R h, int ns, int m, State<NC, D>& M, const TaylorTable& tt) {
        constexpr bool kMixed = std::is_same<R, double>::value && NT == 0;
        const int k32 = kMixed ? tt.f32_from[m] : m + 1;
        // The terms are added to M as they are formed (later terms derive from `term`, not from M), so no
        // separate accumulator is held.
#pragma unroll 1
        for (int j = 0; j < ns; ++j) {
            StepCoef<NC, D> s;
            event_coef(cst, rec, g_mt, s);
            scale_coef(s, h);
            State<NC, D> term;
            matvec<true>(s, M, term, &cst, h);
            fma_state(M, R(1), term);
            int k = 2;
#pragma unroll 1
            for (; k <= m && k < k32; ++k) {
                State<NC, D> nt;
                matvec<false>(s, term, nt);
                term = nt;
                fma_state(M, R(tt.inv_fact[k]), term);
            }
            if constexpr (kMixed) {
                if (k <= m) {
                    // paired float32 instructions over the CEST pools (bmc_tail32.cuh)
                    using T32 = Tail32<NC>;
                    typename T32::Coef s32;
                    typename T32::St t32, a32;
                    T32::coef(s, s32);
                    T32::state(term, t32);
                    T32::zero(a32);
#pragma unroll 1
                    for (; k <= m; ++k) {
                        typename T32::St n32;
                        T32::matvec(s32, t32, n32);
                        t32 = n32;
                        T32::fma_acc(a32, tt.inv_fact_f[k], t32);
                    }
                    T32::add_to(M, a32);
                }
            }
        }
    }

    // Whether an event leaves the transverse entries at zero: no RF, and all of them (with their tangents) zero.
    static __device__ __forceinline__ bool longitudinal(const State<NC, D>& M) {
        auto zero = [](const D& x) {
            bool z = x.v == R(0);
            DN_LOOP(z = z && x.d[t] == R(0));
            return z;
        };
        bool z = zero(M.xw) && zero(M.yw);
#pragma unroll
        for (int i = 0; i < NC; ++i) z = z && zero(M.xc[i]) && zero(M.yc[i]);
        return z;
    }

    // exp(X) [M; 1] of a free event (no RF) whose transverse entries are all zero: they stay zero, and the z entries
    // (water, CEST pools, MT) evolve by their own (NC + 2) x (NC + 2) block, which one thread exponentiates for its
    // chain: the degree-m Horner recurrence of the block and of its constant column, then s squarings, the norm
    // without any precession in it. What is squared is F = exp - 1 (F <- F F + 2 F): the slow modes' entries keep
    // their digits, where squaring 1 + F doubles their error each time.
    // Recoveries and the delays behind a spoiler are such events. The dense path gives each of them a warp for ~11
    // Horner steps and ~13 squarings of the whole (N + 1) x (N + 1) matrix: 206,848 chains of four pools with one
    // 3 s recovery (and one propagator to apply) took 4.89 ms in the chain kernel so, 0.31 ms this way.
    static __device__ __noinline__ void z_event(const ChainConst<NC, D>& cc, R dt, State<NC, D>& M,
                                                const TaylorTable& tt) {
        constexpr int Z = NC + 2;
        // the infinity norm in the balanced scaling of norm_base
        R ex = R(0);
#pragma unroll
        for (int i = 0; i < NC; ++i) ex += fabs(cc.k[i].v) * R(cc.sf[i]);
        const R km = fabs(cc.kmt.v) * R(cc.sfm);
        R nu = fabs(cc.Rw1.v) + ex + km + fabs(cc.cw.v);
        nu = fmax(nu, fabs(cc.Rm1.v) + km + fabs(cc.cm.v) / R(cc.sfm));
#pragma unroll
        for (int i = 0; i < NC; ++i)
            nu = fmax(nu, fabs(cc.Rc1[i].v) + fabs(cc.k[i].v) * R(cc.sf[i]) + fabs(cc.cc[i].v) / R(cc.sf[i]));
        nu = nu * dt;
        const int s = nu > R(tt.dense_theta) ? (int)ceil(log2(double(nu) / tt.dense_theta)) : 0;
        const R h = R(ldexp(double(dt), -s));
        D T[Z][Z], phi[Z];                    // F: T[column][row]
        // Horner, column by column: v <- e + X v / k, without e at the end (the constant column: phi <- X [phi; 1] / k)
#pragma unroll
        for (int j = 0; j <= Z; ++j) {
            D v[Z];
#pragma unroll
            for (int i = 0; i < Z; ++i) v[i] = dconst<R, NT>(i == j ? R(1) : R(0));
#pragma unroll 1
            for (int k = tt.dense_m; k >= 1; --k) {
                const R ik = h * R(tt.inv_k[k]);
                D w = dfma(cc.kmt, v[Z - 1], -(cc.Rw1 * v[0]));
                D m = dfma(cc.kwmt, v[0], -(cc.Rm1 * v[Z - 1]));
                if (j == Z) {
                    w = w + cc.cw;
                    m = m + cc.cm;
                }
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    w = dfma(cc.k[i], v[1 + i], w);
                    D c = dfma(cc.kwc[i], v[0], -(cc.Rc1[i] * v[1 + i]));
                    if (j == Z) c = c + cc.cc[i];
                    v[1 + i] = ik * c;
                }
                v[0] = ik * w;
                v[Z - 1] = ik * m;
                if (j < Z && k > 1) v[j] = v[j] + R(1);
            }
#pragma unroll
            for (int i = 0; i < Z; ++i) (j < Z ? T[j < Z ? j : 0][i] : phi[i]) = v[i];
        }
#pragma unroll 1
        for (int q = 0; q < s; ++q) {
            D n[Z][Z];
#pragma unroll
            for (int i = 0; i < Z; ++i) {
                D p = phi[i] + phi[i];
#pragma unroll
                for (int l = 0; l < Z; ++l) p = dfma(T[l][i], phi[l], p);
                n[0][i] = p;                  // parked: phi is read by every row
            }
#pragma unroll
            for (int i = 0; i < Z; ++i) phi[i] = n[0][i];
#pragma unroll
            for (int j = 0; j < Z; ++j)
#pragma unroll
                for (int i = 0; i < Z; ++i) {
                    D x = T[j][i] + T[j][i];
#pragma unroll
                    for (int l = 0; l < Z; ++l) x = dfma(T[l][i], T[j][l], x);
                    n[j][i] = x;
                }
#pragma unroll
            for (int j = 0; j < Z; ++j)
#pragma unroll
                for (int i = 0; i < Z; ++i) T[j][i] = n[j][i];
        }
        D z[Z];
#pragma unroll
        for (int i = 0; i < Z; ++i) {
            D x = dfma(T[0][i], M.zw, phi[i]);
#pragma unroll
            for (int l = 0; l < NC; ++l) x = dfma(T[1 + l][i], M.zc[l], x);
            z[i] = dfma(T[Z - 1][i], M.zm, x);
        }
        M.zw = M.zw + z[0];
#pragma unroll
        for (int i = 0; i < NC; ++i) M.zc[i] = M.zc[i] + z[1 + i];
        M.zm = M.zm + z[Z - 1];
    }

    static __device__ __forceinline__ void spoil(State<NC, D>& M) {
        const D z = dconst<R, NT>(R(0));
        M.xw = z; M.yw = z;
#pragma unroll
        for (int i = 0; i < NC; ++i) { M.xc[i] = z; M.yc[i] = z; }
    }

    static __device__ __forceinline__ D& at(State<NC, D>& M, int ref_index) {
        // reference index -> member (used only outside hot loops)
        if (ref_index == L::ixw) return M.xw;
        if (ref_index == L::iyw) return M.yw;
        if (ref_index == L::izw) return M.zw;
        if (ref_index == L::izm) return M.zm;
        if (ref_index <= NC) return M.xc[ref_index - 1];
        if (ref_index <= 2 * NC + 1) return M.yc[ref_index - NC - 2];
        return M.zc[ref_index - 2 * NC - 3];
    }

    static __device__ void load_m0(const ChainArgs& a, int v, State<NC, D>& M) {
        const double* m0 = a.m0 + (size_t)v * N;
#pragma unroll
        for (int q = 0; q < N; ++q) {
            D x = dconst<R, NT>(R(m0[q]));
            if constexpr (NT > 0) {
                if (a.dm0) {
#pragma unroll
                    for (int t = 0; t < NT; ++t) x.d[t] = R(a.dm0[((size_t)(a.t0 + t) * a.n_vox + v) * N + q]);
                }
            }
            at(M, q) = x;
        }
    }
};

}  // namespace bmc
