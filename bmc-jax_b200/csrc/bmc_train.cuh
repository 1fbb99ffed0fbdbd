// bmc_train.cuh -- propagators of shaped pulses: a pulse that a row repeats is propagated once per chain.
//
// A pulsed saturation train repeats one shaped pulse: n RF events of one duration h, frequency and phase whose
// amplitudes follow the shape (200 samples, 20 pulses in the tables met most). The chain kernel takes every event
// of every repeat through the Taylor action, n x repeats times ~20 operator products. Here the pulse's propagator
//     P = E_n ... E_1,   E_k = exp([A(w_k) C; 0 0] h)
// is formed once per chain and applied at each repeat (chain kernel).
//
// * The events of one pulse differ in their RF amplitude alone, so all E_k are values of one matrix function E(w). In
//   the frame turned by the pulse's phase the RF couples y to z only, so the entries between {x, y} and {z} are odd in
//   w and the others even: with u = (w / w_max)^2, E's even entries and its odd entries over w are entire functions
//   of u. They are interpolated in u through NQ Chebyshev nodes of [0, 1]: exact exponentials (scaling and squaring) at
//   the nodes, their divided differences, and per sample the Newton form, NQ - 1 fused multiply-adds an entry.
//   The error is at most 2 / 4^NQ times the order-NQ term of the series in u, which falls like
//   (w h)^(2 NQ) / (2 NQ)!: NQ is 4 or 6, the chain's own choice (interp_nodes), and a chain beyond the bound is left
//   to the chain kernel.
// * P is a chain of dense N x N products: a warp per chain, on the FP64 tensor cores (mma.sync m8n8k4). P stays in
//   registers as the left operand: the accumulator layout of one product is the A operand of the next when the k
//   index of step e of a tile is read as its columns 2 t + e, so P <- P E_k needs no shuffle; E_k is evaluated
//   straight into the B layout from the E_q in shared memory.
// * The constant column: phi <- phi + P e_k before each product, every lane summing its own columns; the lanes' parts
//   are added once at the end.
// * A shape that is its own mirror image costs half: E_1 ... E_m (the second half) is the first half's product with its
//   order reversed, and every E_k is its own transpose up to signs and the pools' fractions (G E^T G^-1 = E, G = diag(+-f),
//   detailed balance; bmc_sym.cuh), so Phi_2 = G Phi_1^T G^-1. Only the second half's constant column needs its own
//   recurrence, a matrix-vector product per sample.
// * Equal events between the repeats (gaps, spoilers) belong to the unit too; units that follow one another with the
//   same phase are one propagator P^repeats.
#pragma once
#include "bmc_adjoint.cuh"

namespace bmc {

constexpr int kTrainMinSamples = 8;      // a shaped pulse has at least this many samples ...
constexpr int kTrainMaxSamples = 1024;   // ... and at most this many (its weights are kept per row)
constexpr int kTrainMaxPulses = 1024;    // pulses of a row that are looked at
constexpr int kTrainMaxGap = 4;          // events between two pulses that a unit takes in
constexpr double kTrainTol = 2e-15;      // interpolation error per event
constexpr double kTrainMirror = 9e-16;   // 8 x 2^-53: two samples this close (over the largest) mirror each other

// the table's side of a propagator launch; the chains' side (ChainArgs: train, prop, prop_ok, first_chain,
// chain_count) is the chain kernel's too
struct TrainArgs {
    const double* rho;         // [rows][max_samples]: the reference pulse's amplitudes over its largest
    int max_samples;
    double* prop;              // [chains of the launch][mats][N][NS]: P's rows, phi last, then the derivatives'
    int mats;                  // 1 + the launch's tangents
    unsigned char* ok;         // [chains of the launch]: the propagator was formed
    int* kinds;                // kTrained and kPlain by the rows, kRefused by the chains (ChainArgs::kinds)
};

// From when on a pulse's propagator pays: uses x (samples, and kTrainGapEvents for a gap's delays) >= fixed + sample x samples, in
// Taylor actions of one event: the cost of a propagator's exponentials at the nodes, and of its products and interpolation
// for one sample (kTrainSkewed times that without the mirror image). Measured by pool count on 51,712 chains (25,856 with a
// tangent), pulses of 10, 30 and 100 samples (0.5 ms, 1 uT) with and without a 5 ms gap, 2 to 8 uses, against the Taylor
// action before there were propagators, its lanes in step (now up to twice as fast). With four pools and a gap, propagator /
// that in ms: 4 x 10 samples 2.31 / 1.61, 8 x 10 2.44 / 3.12, 4 x 30 2.59 / 3.15, 2 x 100 3.55 / 4.26; with two pools 4 x 10 1.72 /
// 1.20, 8 x 10 1.77 / 2.26. The line knows the table alone, so that a chain's result does not depend on how many others the
// call has: twice as many chains move it up by a quarter, an eighth of them down by half, and one spectrum gains from two
// uses on (four pools, 2 x 10 samples: 0.08 ms against 0.28).
constexpr double kTrainGapEvents = 5.0, kTrainSkewed = 1.75;
struct TrainCost {
    double fixed, sample, skewed;
};
template <int NC>
constexpr TrainCost train_cost(bool tangents) {
    constexpr double fixed[2][6] = {{110, 44, 78, 77, 88, 150}, {52, 43, 75, 59, 54, 93}};
    constexpr double sample[2][6] = {{1.4, 0.42, 1.0, 0.95, 0.75, 2.2}, {2.0, 0.78, 2.55, 1.1, 1.0, 2.8}};
    return {fixed[tangents][NC], sample[tangents][NC], sample[tangents][NC] * (tangents ? 1.0 : kTrainSkewed)};
}
// the fewest events that a table with a train has (a pulse of kTrainMinSamples and its gap)
template <int NC>
constexpr int train_min_events(bool tangents) {
    return (int)(train_cost<NC>(tangents).fixed * kTrainMinSamples / (kTrainMinSamples + kTrainGapEvents));
}

// Chebyshev nodes of (0, 1), ascending: sin^2(pi (2 q + 1) / (4 n))
template <int NQ>
__device__ __forceinline__ constexpr double train_node(int q) {
    constexpr double c4[4] = {0.03806023374435663, 0.3086582838174551, 0.6913417161825449, 0.9619397662556434};
    constexpr double c6[6] = {0.01703708685546585, 0.14644660940672624, 0.37059047744873963,
                              0.6294095225512604,  0.8535533905932737,  0.9829629131445341};
    return NQ == 4 ? c4[q] : c6[q];
}

// ------------------------------------------------------------------------------------------------
// the trains of a table: one block per row
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool train_same_pulse(const EvRec<double>& x, const EvRec<double>& y) {
    return x.dt == y.dt && x.wf == y.wf && x.c == y.c && x.s == y.s;
}

constexpr int kTrainScanThreads = 256;

// Finds each row's pulses (runs of RF events of one duration, frequency and phase), takes the middle one as the
// reference, and keeps those with its samples; marks the units' first records and writes the reference pulse's
// relative amplitudes. A row whose repeated block (seg) saves more events has no train; a row with one keeps its
// block for the chains that have no propagator.
static __global__ void __launch_bounds__(kTrainScanThreads)
train_scan_kernel(EvRec<double>* __restrict__ ev, int n_ev, int stride, const TrainCost cost, const int4* __restrict__ seg,
                  TrainRow* __restrict__ rows, double* __restrict__ rho, int max_samples, int* __restrict__ kinds) {
    __shared__ int starts[kTrainMaxPulses], ends[kTrainMaxPulses];
    __shared__ unsigned char match[kTrainMaxPulses];
    __shared__ int n_start, n_end, warp_n[kTrainScanThreads / 32][2], flags[3];
    __shared__ double wmax_s;
    EvRec<double>* row = ev + blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    TrainRow out{0, 0, 0, 0, 0, 0, 0.0};
    if (tid == 0) n_start = n_end = 0;
    __syncthreads();
    auto is_rf = [&](const EvRec<double>& r) { return (int)r.type == EV_RF && r.dt > 1e-9; };
    for (int base = 0; base < n_ev; base += kTrainScanThreads) {
        const int e = base + tid;
        bool st = false, en = false;
        if (e < n_ev) {
            const EvRec<double> r = row[(size_t)e * stride];
            if (is_rf(r)) {
                st = en = true;
                if (e > 0) {
                    const EvRec<double> p = row[(size_t)(e - 1) * stride];
                    st = !(is_rf(p) && train_same_pulse(p, r));
                }
                if (e + 1 < n_ev) {
                    const EvRec<double> q = row[(size_t)(e + 1) * stride];
                    en = !(is_rf(q) && train_same_pulse(r, q));
                }
            }
        }
        const unsigned bs = __ballot_sync(kFull, st), be = __ballot_sync(kFull, en);
        if (lane == 0) {
            warp_n[warp][0] = __popc(bs);
            warp_n[warp][1] = __popc(be);
        }
        __syncthreads();
        int os = n_start, oe = n_end;
        for (int w = 0; w < warp; ++w) {
            os += warp_n[w][0];
            oe += warp_n[w][1];
        }
        const unsigned below = (1u << lane) - 1u;
        os += __popc(bs & below);
        oe += __popc(be & below);
        if (st && os < kTrainMaxPulses) starts[os] = e;
        if (en && oe < kTrainMaxPulses) ends[oe] = e;
        __syncthreads();
        if (tid == kTrainScanThreads - 1) {
            n_start = os + (st ? 1 : 0);
            n_end = oe + (en ? 1 : 0);
        }
        __syncthreads();
    }
    const int np = n_start;
    if (np >= 2 && np <= kTrainMaxPulses && np == n_end) {     // the same in every thread of the block
        const int ref = (np - 1) / 2, r0 = starts[ref], n = ends[ref] - r0 + 1;
        if (n >= kTrainMinSamples && n <= max_samples) {
            for (int p = tid; p < np; p += kTrainScanThreads) match[p] = ends[p] - starts[p] + 1 == n;
            if (tid < 3) flags[tid] = 1;
            __syncthreads();
            for (long long i = tid; i < (long long)np * n; i += kTrainScanThreads) {
                const int p = (int)(i / n), k = (int)(i % n);
                const EvRec<double> x = row[(size_t)(r0 + k) * stride];
                if (match[p]) {
                    const EvRec<double> y = row[(size_t)(starts[p] + k) * stride];
                    if (!(x.w1 == y.w1 && x.dt == y.dt && x.wf == y.wf)) match[p] = 0;
                }
            }
            __syncthreads();
            // the gap after the reference, and whether every unit has it
            const int ng = ref + 1 < np ? starts[ref + 1] - ends[ref] - 1 : 0;
            const bool gap_fits = ng >= 1 && ng <= kTrainMaxGap;
            for (int p = tid; p < np; p += kTrainScanThreads) {
                if (!match[p]) continue;
                bool same = gap_fits && ends[p] + ng < n_ev;
                for (int j = 0; same && j < ng; ++j) {
                    const EvRec<double> x = row[(size_t)(ends[ref] + 1 + j) * stride];
                    const EvRec<double> y = row[(size_t)(ends[p] + 1 + j) * stride];
                    const int type = (int)x.type;
                    same = same_rec(x, y) && type != EV_RF && type != EV_ADC && x.w1 == 0.0;
                }
                if (!same) atomicAnd(&flags[0], 0);
            }
            __syncthreads();
            const int gap = flags[0] ? ng : 0;
            // one run of equal units?
            for (int p = tid; p < np; p += kTrainScanThreads) {
                if (!match[p] || p + 1 >= np) continue;
                const EvRec<double> x = row[(size_t)starts[p] * stride], y = row[(size_t)starts[p + 1] * stride];
                bool next = match[p + 1] && starts[p + 1] == starts[p] + n + gap && x.c == y.c && x.s == y.s;
                if (!next)      // the last one of the run: fine if no other matches follow
                    for (int q = p + 1; q < np && !next; ++q)
                        if (match[q]) atomicAnd(&flags[1], 0);
            }
            if (warp == 0) {
                double m = 0.0;
                for (int k = lane; k < n; k += 32) m = fmax(m, fabs(row[(size_t)(r0 + k) * stride].w1));
                m = warp_max(m);
                if (lane == 0) wmax_s = m;
            }
            __syncthreads();
            // mirrored within the rounding of a shape that was computed sample by sample
            for (int k = tid; k < n / 2; k += kTrainScanThreads)
                if (!(fabs(row[(size_t)(r0 + k) * stride].w1 - row[(size_t)(r0 + n - 1 - k) * stride].w1) <=
                      kTrainMirror * wmax_s))
                    atomicAnd(&flags[2], 0);
            __syncthreads();
            int uses = 0, first_match = -1;
            for (int p = 0; p < np; ++p)
                if (match[p]) {
                    if (first_match < 0) first_match = p;
                    ++uses;
                }
            const int run = flags[1] ? uses : 1, unit = n + gap;
            const int4 blk = seg[blockIdx.x];
            const long long block_saves = blk.z >= 2 ? (long long)(blk.z - 1) * blk.y : 0;
            const double wm = wmax_s;
            const bool pays = uses >= 2 && uses * (n + (gap > 0 ? kTrainGapEvents : 0.0)) >=
                                               cost.fixed + n * (flags[2] ? cost.sample : cost.skewed);
            if (pays && wm > 0.0 && wm < INFINITY && (long long)(uses - 1) * n > block_saves) {
                out = TrainRow{r0, n, gap, run, run * unit, flags[2], wm};
                for (int p = tid; p < np; p += kTrainScanThreads)
                    if (match[p] && (run == 1 || p == first_match)) {
                        EvRec<double>& m = row[(size_t)starts[p] * stride];
                        m.type = m.type + double(kTrainMark);
                    }
                for (int k = tid; k < n; k += kTrainScanThreads)
                    rho[(size_t)blockIdx.x * max_samples + k] = row[(size_t)(r0 + k) * stride].w1 / wm;
            }
        }
    }
    if (tid == 0) {
        rows[blockIdx.x] = out;
        atomicOr(kinds, out.n > 0 ? kTrained : kPlain);
    }
}

// ------------------------------------------------------------------------------------------------
// the propagators: one warp per chain
// ------------------------------------------------------------------------------------------------
template <int NC, int NT>
struct TrainCoef {
    using D = Dn<double, NT>;
    static constexpr int NCA = NC > 0 ? NC : 1;
    D Rw2, Rw1, offw, k[NCA], kwc[NCA], Rc2[NCA], Rc1[NCA], offc[NCA], kmt, kwmt, cw, cm, cc[NCA];
    D w1[TrainShape<NC>::kSlots], Rm[TrainShape<NC>::kSlots];   // per matrix: the RF amplitude and the MT rate
};

// NT = 1: index 0 the values, 1 their derivatives along the launch's tangent
template <int NC, int NT>
struct alignas(16) TrainSmem {
    using S = TrainShape<NC>;
    double T[1 + NT][S::kSlots][S::TS];          // column-major, padded with zeros
    double phi[1 + NT][S::kSlots][8 * S::NT];
    double gv[8 * S::NT];                        // G by state entry, signed (1 in the padding)
    TrainCoef<NC, NT> coef;
};

// the MT lineshape summed by the warp: lane l takes the terms l, l + 32, ... of the 101-term sum
template <int NT>
__device__ __forceinline__ Dn<double, NT> warp_sl_direct(Dn<double, NT> delta, Dn<double, NT> t2, int lane) {
    using D = Dn<double, NT>;
    D acc = dconst<double, NT>(0.0);
    const D dt2 = delta * t2;
    for (int i = lane; i <= 100; i += 32) {
        const double u = 0.01 * double(i);
        double q = fabs(3.0 * u * u - 1.0);
        q = q > 1e-6 ? q : 1e-6;
        const double iq = 1.0 / q;
        const D arg = iq * dt2;
        acc = acc + iq * dexp(-2.0 * (arg * arg));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc.v += __shfl_xor_sync(kFull, acc.v, o);
        DN_LOOP(acc.d[t] += __shfl_xor_sync(kFull, acc.d[t], o));
    }
    return (0.7978845608028654 * 3.141592653589793 * 0.01) * (t2 * acc);
}

// super_lorentzian of bmc_device.cuh by the whole warp (all lanes hold the same arguments). The bridge's support
// points lie symmetrically about 0 and the sum depends on the square of its argument, so two sums serve the four.
template <int NT>
__device__ __forceinline__ Dn<double, NT> warp_super_lorentzian(Dn<double, NT> delta, Dn<double, NT> t2,
                                                                Dn<double, NT> w0, int lane) {
    using D = Dn<double, NT>;
    if (fabs(delta.v) >= w0.v) return warp_sl_direct<NT>(delta, t2, lane);
    const D p1 = -w0 - 100.0, p2 = w0 + 100.0;
    const D y0 = warp_sl_direct<NT>(w0 + 300.0, t2, lane), y1 = warp_sl_direct<NT>(p2, t2, lane);
    const D d0 = 30.0 * (y1 - y0), d1 = -d0;
    const D c = dabs((delta - p1 + 1.0) / (p2 - p1 + 1.0));
    const D c2 = c * c, c3 = c2 * c;
    return (2.0 * c3 - 3.0 * c2 + 1.0) * y1 + (3.0 * c2 - 2.0 * c3) * y1 + (c3 - 2.0 * c2 + c) * d0 + (c3 - c2) * d1;
}

// DT: tangents carried along (0, or 1: the derivative along one of the launch's tangents beside every value)
template <int NC, int DT>
struct Train {
    using D = Dn<double, DT>;
    using C = Chain<NC, double, DT>;
    using S = State<NC, D>;
    using SH = TrainShape<NC>;
    using SM = TrainSmem<NC, DT>;
    static constexpr int N = SH::N, NT = SH::NT, LD = SH::LD, NA = N + 1, ND = 1 + DT;
    static constexpr int Z0 = 2 * (NC + 1);                   // the first z entry

    // value (0) or derivative (1) of a dual
    static __device__ __forceinline__ double& part(D& x, int d) {
        if constexpr (DT > 0) return d ? x.d[0] : x.v;
        else return x.v;
    }

    // Interpolation nodes for a pulse of theta = |w_max| h and x = w_max^2 g h (the MT saturation's exponent): the
    // smallest of 4 and 6 whose bound 2 / 4^n sum_j theta^2j / (2j)! x^(n-j) / (n-j)! meets the tolerance; 0: neither.
    static __device__ __forceinline__ int interp_nodes(double theta, double x) {
        for (int n = 4; n <= 6; n += 2) {
            double sum = 0.0, a = 1.0;                        // a = theta^2j / (2j)!
            for (int j = 0; j <= n; ++j) {
                double b = 1.0;                               // x^(n-j) / (n-j)!
                for (int i = 1; i <= n - j; ++i) b *= x / i;
                sum += a * b;
                a *= theta * theta / ((2 * j + 1.0) * (2 * j + 2.0));
            }
            if (2.0 * sum <= kTrainTol * double(1ll << (2 * n))) return n;
        }
        return 0;
    }

    // y = X x + C c with the RF along x of the turned frame (matrix `q` of the coefficients)
    static __device__ __forceinline__ void op(const TrainCoef<NC, DT>& f, int q, const S& v, double c, S& y) {
        const D w = f.w1[q];
        D px = dconst<double, DT>(0.0), py = px, pz = dfma(f.kmt, v.zm, c * f.cw);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            px = dfma(f.k[i], v.xc[i], px);
            py = dfma(f.k[i], v.yc[i], py);
            pz = dfma(f.k[i], v.zc[i], pz);
            y.xc[i] = dfma(f.kwc[i], v.xw, -dfma(f.Rc2[i], v.xc[i], f.offc[i] * v.yc[i]));
            y.yc[i] = dfma(f.kwc[i], v.yw, dfma(f.offc[i], v.xc[i], dfma(w, v.zc[i], -(f.Rc2[i] * v.yc[i]))));
            y.zc[i] = dfma(f.kwc[i], v.zw, c * f.cc[i] - dfma(f.Rc1[i], v.zc[i], w * v.yc[i]));
        }
        y.xw = dfma(f.offw, v.yw, px - f.Rw2 * v.xw);
        y.yw = dfma(w, v.zw, py - dfma(f.Rw2, v.yw, f.offw * v.xw));
        y.zw = pz - dfma(w, v.yw, f.Rw1 * v.zw);
        y.zm = dfma(f.kwmt, v.zw, c * f.cm - f.Rm[q] * v.zm);
    }

    // The coefficients of one event times h, for matrices that differ in w1 and Rm (written by the caller).
    static __device__ __forceinline__ void put_coef(TrainCoef<NC, DT>& f, const StepCoef<NC, D>& s,
                                                    const ChainConst<NC, D>& cc, double h) {
        f.Rw2 = h * s.Rw2; f.Rw1 = h * s.Rw1; f.offw = h * s.offw;
        f.kmt = h * s.kmt; f.kwmt = h * s.kwmt; f.cw = h * cc.cw; f.cm = h * cc.cm;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            f.k[i] = h * s.k[i]; f.kwc[i] = h * s.kwc[i]; f.Rc2[i] = h * s.Rc2[i]; f.Rc1[i] = h * s.Rc1[i];
            f.offc[i] = h * s.offc[i]; f.cc[i] = h * cc.cc[i];
        }
    }

    // T[0 .. n) and phi[0 .. n) <- the exponentials of the n matrices of the coefficients: every column a task of its
    // own (the degree-m Horner recurrence), then s squarings of each matrix by the warp
    static __device__ void exponentials(SM* sm, int lane, int n, int s, const TaylorTable& tt) {
        for (int task = lane; task < n * NA; task += 32) {
            const int q = task / NA, col = task % NA;
            const double caug = col == N ? 1.0 : 0.0;
            S v;
#pragma unroll
            for (int i = 0; i < N; ++i) C::at(v, i) = dconst<double, DT>(i == col ? 1.0 : 0.0);
#pragma unroll 1
            for (int k = tt.dense_m; k >= 1; --k) {
                S y;
                op(sm->coef, q, v, caug, y);
                const double ik = tt.inv_k[k];
#pragma unroll
                for (int i = 0; i < N; ++i) C::at(v, i) = ik * C::at(y, i) + (i == col && k > 1 ? 1.0 : 0.0);
            }
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                double* out = col < N ? sm->T[d][q] + col * LD : sm->phi[d][q];
#pragma unroll
                for (int i = 0; i < N; ++i) out[i] = part(C::at(v, i), d);
            }
        }
        __syncwarp();
        for (int q = 0; q < n; ++q) {
            for (int j = 0; j < s; ++j) square(sm, q, lane);
            if (lane < N) sm->T[0][q][lane * LD + lane] += 1.0;
        }
        __syncwarp();
    }

    // F <- F F + 2 F, phi <- F phi + 2 phi of slot q (and their derivatives), F = exp - 1: the slow modes' entries keep
    // their digits, where squaring 1 + F doubles their error each time
    static __device__ __forceinline__ void square(SM* sm, int q, int lane) {
        const int g = lane >> 2, t = lane & 3;
        double c[ND][NT][NT][2];
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J < NT; ++J) c[d][I][J][0] = c[d][I][J][1] = 0.0;
#pragma unroll
        for (int K = 0; K < 2 * NT; ++K) {
            double a[ND][NT], b[ND][NT];
#pragma unroll
            for (int d = 0; d < ND; ++d)
#pragma unroll
                for (int I = 0; I < NT; ++I) {
                    // F + 2 as the left operand gives F F + 2 F (and F dF + 2 dF)
                    a[d][I] = sm->T[d][q][(4 * K + t) * LD + 8 * I + g] + (d == 0 && 8 * I + g == 4 * K + t ? 2.0 : 0.0);
                    b[d][I] = sm->T[d][q][(8 * I + g) * LD + 4 * K + t];
                }
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J < NT; ++J) {
                    dmma(c[0][I][J][0], c[0][I][J][1], a[0][I], b[0][J]);
                    if constexpr (DT > 0) {
                        dmma(c[DT][I][J][0], c[DT][I][J][1], a[0][I], b[DT][J]);
                        dmma(c[DT][I][J][0], c[DT][I][J][1], a[DT][I], b[0][J]);
                    }
                }
        }
        double p[ND];
        if (lane < N) {
#pragma unroll
            for (int d = 0; d < ND; ++d) p[d] = 2.0 * sm->phi[d][q][lane];
#pragma unroll
            for (int l = 0; l < N; ++l) {
                const double x = sm->T[0][q][l * LD + lane], y = sm->phi[0][q][l];
                p[0] = fma(x, y, p[0]);
                if constexpr (DT > 0)
                    p[DT] = fma(x, sm->phi[DT][q][l], fma(sm->T[DT][q][l * LD + lane], y, p[DT]));
            }
        }
        __syncwarp();
#pragma unroll
        for (int d = 0; d < ND; ++d) {
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J < NT; ++J)
#pragma unroll
                    for (int e = 0; e < 2; ++e) sm->T[d][q][(8 * J + 2 * t + e) * LD + 8 * I + g] = c[d][I][J][e];
            if (lane < N) sm->phi[d][q][lane] = p[d];
        }
        __syncwarp();
    }

    // the running propagator: lane (g, t) holds P[8 I + g][8 J + 2 t + e] and its part of phi's rows
    struct Run {
        double P[ND][NT][NT][2];
        double f[ND][NT];
    };

    static __device__ __forceinline__ void identity(Run& r, int lane) {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                r.f[d][I] = 0.0;
#pragma unroll
                for (int J = 0; J < NT; ++J)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        r.P[d][I][J][e] = d == 0 && 8 * I + g == 8 * J + 2 * t + e ? 1.0 : 0.0;
            }
    }

    // a lane's part of E in the B layout and of its constant column: E[8 K + 2 t + (x, y)][8 J + g], v[8 K + 2 t + ..]
    struct Op {
        double2 E[ND][NT][NT], v[ND][NT];
    };

    static __device__ __forceinline__ double2 lds2(const double* p) {
        double2 x;      // volatile: not moved out of the sample loop, whose registers it would take
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                     : "=d"(x.x), "=d"(x.y)
                     : "r"((unsigned)__cvta_generic_to_shared(p)));
        return x;
    }

    // matrix slot `q` as it is
    static __device__ __forceinline__ void load(const SM* sm, int q, Op& o, int lane) {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int K = 0; K < NT; ++K) {
                o.v[d][K] = lds2(sm->phi[d][q] + 8 * K + 2 * t);
#pragma unroll
                for (int J = 0; J < NT; ++J) o.E[d][K][J] = lds2(sm->T[d][q] + (8 * J + g) * LD + 8 * K + 2 * t);
            }
    }

    // The interpolant at w = rho w_max: Newton's form over the divided differences in the slots (the values' in
    // registers where they fit: H, kHeld of the slots), then the entries odd in the amplitude times rho.
    template <int NQ, int kHeld>
    static __device__ __forceinline__ void eval(const SM* sm, const double2 (&H)[kHeld > 0 ? kHeld : 1][NT][NT],
                                                double rho, Op& o, int lane) {
        const int g = lane >> 2, t = lane & 3;
        const double u = rho * rho;
        double d[NQ - 1];
#pragma unroll
        for (int q = 0; q < NQ - 1; ++q) d[q] = u - train_node<NQ>(q);
#pragma unroll
        for (int K = 0; K < NT; ++K) {
            const int row = 8 * K + 2 * t;                    // this lane's rows: row, row + 1
            const double o0 = row >= Z0 ? 1.0 : rho, o1 = row + 1 >= Z0 ? 1.0 : rho;   // v's and E[., z]'s factor
            const double p0 = row >= Z0 ? rho : 1.0, p1 = row + 1 >= Z0 ? rho : 1.0;   // E[., x and y]'s factor
#pragma unroll
            for (int k = 0; k < ND; ++k) {
                double2 v = lds2(sm->phi[k][NQ - 1] + row);
#pragma unroll
                for (int q = NQ - 2; q >= 0; --q) {
                    const double2 x = lds2(sm->phi[k][q] + row);
                    v.x = fma(v.x, d[q], x.x);
                    v.y = fma(v.y, d[q], x.y);
                }
                o.v[k][K] = make_double2(v.x * o0, v.y * o1);
#pragma unroll
                for (int J = 0; J < NT; ++J) {
                    const bool z = 8 * J + g >= Z0;
                    double2 E;
#pragma unroll
                    for (int q = NQ - 1; q >= 0; --q) {
                        const double2 x = k == 0 && q < kHeld ? H[q < kHeld ? q : 0][K][J]
                                                              : lds2(sm->T[k][q] + (8 * J + g) * LD + row);
                        if (q == NQ - 1) {
                            E = x;
                        } else {
                            E.x = fma(E.x, d[q], x.x);
                            E.y = fma(E.y, d[q], x.y);
                        }
                    }
                    o.E[k][K][J] = make_double2(E.x * (z ? o0 : p0), E.y * (z ? o1 : p1));
                }
            }
        }
    }

    // phi <- phi + P v, P <- P E (and the derivatives)
    static __device__ __forceinline__ void apply(Run& r, const Op& o) {
        double c[ND][NT][NT][2];
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J < NT; ++J) c[d][I][J][0] = c[d][I][J][1] = 0.0;
#pragma unroll
        for (int K = 0; K < NT; ++K) {
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int J = 0; J < NT; ++J)
#pragma unroll
                    for (int I = 0; I < NT; ++I) {
                        const double E = e ? o.E[0][K][J].y : o.E[0][K][J].x;
                        dmma(c[0][I][J][0], c[0][I][J][1], r.P[0][I][K][e], E);
                        if constexpr (DT > 0) {
                            dmma(c[DT][I][J][0], c[DT][I][J][1], r.P[DT][I][K][e], E);
                            dmma(c[DT][I][J][0], c[DT][I][J][1], r.P[0][I][K][e],
                                 e ? o.E[DT][K][J].y : o.E[DT][K][J].x);
                        }
                    }
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                const double2 v = o.v[0][K];
                r.f[0][I] = fma(r.P[0][I][K][0], v.x, fma(r.P[0][I][K][1], v.y, r.f[0][I]));
                if constexpr (DT > 0) {
                    const double2 w = o.v[DT][K];
                    double x = fma(r.P[DT][I][K][0], v.x, fma(r.P[DT][I][K][1], v.y, r.f[DT][I]));
                    r.f[DT][I] = fma(r.P[0][I][K][0], w.x, fma(r.P[0][I][K][1], w.y, x));
                }
            }
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J < NT; ++J) {
                    r.P[d][I][J][0] = c[d][I][J][0];
                    r.P[d][I][J][1] = c[d][I][J][1];
                }
    }

    static __device__ __forceinline__ void step(const SM* sm, Run& r, int lane) {
        Op o;
        load(sm, 0, o, lane);
        apply(r, o);
    }

    // phi's rows summed over the lanes that hold parts of them; the sum is left in the t = 0 lane, zero in the others
    static __device__ __forceinline__ void sum_phi(Run& r, int lane) {
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                double x = r.f[d][I];
                x += __shfl_xor_sync(kFull, x, 1);
                x += __shfl_xor_sync(kFull, x, 2);
                r.f[d][I] = (lane & 3) == 0 ? x : 0.0;
            }
    }

    // (P, phi) into matrix slot `q`, in the layout `step` reads (phi summed)
    static __device__ __forceinline__ void put(SM* sm, int q, Run& r, int lane) {
        const int g = lane >> 2, t = lane & 3;
        sum_phi(r, lane);
        __syncwarp();
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int I = 0; I < NT; ++I) {
#pragma unroll
                for (int J = 0; J < NT; ++J)
#pragma unroll
                    for (int e = 0; e < 2; ++e) sm->T[d][q][(8 * J + 2 * t + e) * LD + 8 * I + g] = r.P[d][I][J][e];
                if (t == 0) sm->phi[d][q][8 * I + g] = r.f[d][I];
            }
        __syncwarp();
    }

    // The pools' G = diag(+-f) by state entry: its magnitude (1 for water, and for a pool without exchange)
    static __device__ __forceinline__ double balance(const double* params, int n_vox, int v, int i, bool& ok) {
        using L = Layout<NC>;
        double f = 1.0, k = 0.0;
        if (i == N - 1) {
            f = params[(size_t)L::MF * n_vox + v];
            k = params[(size_t)L::MK * n_vox + v];
        } else if (i < N - 1 && i % (NC + 1) != 0) {
            const int p = i % (NC + 1) - 1;
            f = params[(size_t)(L::CF + p) * n_vox + v];
            k = params[(size_t)(L::CK + p) * n_vox + v];
        }
        if (f > 1e-20) return f;
        ok = ok && k == 0.0;
        return 1.0;
    }

    // A mirrored pulse from its first half: r <- Phi_2 (E_c) Phi_1 with its constant column. `gv` holds G by state entry
    // in shared memory (signed; slot 1 is free until the end of the sweep only for its own product).
    template <int NQ>
    static __device__ __forceinline__ void mirrored(SM* sm, Run& r, const double* __restrict__ rho, int n,
                                                    const double* gv, int lane) {
        static_assert(DT == 0, "the propagators' derivatives take the whole pulse");
        constexpr int kHeld = NT == 1 ? NQ : (NT == 2 && NQ == 4 ? 4 : 0);
        const int g = lane >> 2, t = lane & 3, m = n / 2;
        double2 H[kHeld > 0 ? kHeld : 1][NT][NT];
#pragma unroll
        for (int q = 0; q < kHeld; ++q)
#pragma unroll
            for (int K = 0; K < NT; ++K)
#pragma unroll
                for (int J = 0; J < NT; ++J) H[q][K][J] = lds2(sm->T[0][q] + (8 * J + g) * LD + 8 * K + 2 * t);
        // psi = G^-1 phi_2: psi <- G^-1 v + E^T psi, from the middle out (rows 8 K + 2 t + (x, y) in this lane)
        double2 ig[NT], psi[NT];
#pragma unroll
        for (int K = 0; K < NT; ++K) {
            ig[K] = make_double2(1.0 / gv[8 * K + 2 * t], 1.0 / gv[8 * K + 2 * t + 1]);
            psi[K] = make_double2(0.0, 0.0);
        }
        Op cur;
        eval<NQ, kHeld>(sm, H, rho[m - 1], cur, lane);
        double next = rho[m > 1 ? m - 2 : 0];
#pragma unroll 1
        for (int k = m - 1; k >= 0; --k) {
            const double after = rho[k > 2 ? k - 2 : 0];
            Op nx;
            eval<NQ, kHeld>(sm, H, next, nx, lane);
            apply(r, cur);
            double x[NT];
#pragma unroll
            for (int J = 0; J < NT; ++J) {
                x[J] = 0.0;
#pragma unroll
                for (int K = 0; K < NT; ++K)
                    x[J] = fma(cur.E[0][K][J].x, psi[K].x, fma(cur.E[0][K][J].y, psi[K].y, x[J]));
                x[J] += __shfl_xor_sync(kFull, x[J], 1);
                x[J] += __shfl_xor_sync(kFull, x[J], 2);      // entry 8 J + g
            }
#pragma unroll
            for (int K = 0; K < NT; ++K) {
                psi[K].x = fma(cur.v[0][K].x, ig[K].x, __shfl_sync(kFull, x[K], 8 * t));
                psi[K].y = fma(cur.v[0][K].y, ig[K].y, __shfl_sync(kFull, x[K], 8 * t + 4));
            }
            cur = nx;
            next = after;
        }
        Op mid;
        if (n & 1) eval<NQ, kHeld>(sm, H, rho[m], mid, lane);
        // Phi_1 and phi_1 into slot 1 (the differences are no longer needed), Phi_2 and phi_2 into the registers
        __syncwarp();
        put(sm, 1, r, lane);
        if (g == 0) {
#pragma unroll
            for (int K = 0; K < NT; ++K) {
                sm->phi[0][0][8 * K + 2 * t] = psi[K].x * gv[8 * K + 2 * t];
                sm->phi[0][0][8 * K + 2 * t + 1] = psi[K].y * gv[8 * K + 2 * t + 1];
            }
        }
        __syncwarp();
#pragma unroll
        for (int I = 0; I < NT; ++I) {
            const int row = 8 * I + g;
            r.f[0][I] = t == 0 ? sm->phi[0][0][row] : 0.0;
#pragma unroll
            for (int J = 0; J < NT; ++J)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = 8 * J + 2 * t + e;
                    r.P[0][I][J][e] = sm->T[0][1][row * LD + col] * (gv[row] / gv[col]);
                }
        }
        if (n & 1) apply(r, mid);
        Op first;
        load(sm, 1, first, lane);
        apply(r, first);
    }

    // The samples of the pulse, from the last to the first; the next sample's matrix is evaluated beside the products
    // with this one's, so that the vector and the tensor FP64 pipes work together.
    template <int NQ>
    static __device__ __forceinline__ void samples(const SM* sm, Run& r, const double* __restrict__ rho, int n, int lane) {
        // 64 registers at most
        constexpr int kHeld = DT > 0 ? 0 : (NT == 1 ? NQ : (NT == 2 && NQ == 4 ? 4 : 0));
        const int g = lane >> 2, t = lane & 3;
        double2 H[kHeld > 0 ? kHeld : 1][NT][NT];
#pragma unroll
        for (int q = 0; q < kHeld; ++q)
#pragma unroll
            for (int K = 0; K < NT; ++K)
#pragma unroll
                for (int J = 0; J < NT; ++J) H[q][K][J] = lds2(sm->T[0][q] + (8 * J + g) * LD + 8 * K + 2 * t);
        Op cur;
        eval<NQ, kHeld>(sm, H, rho[n - 1], cur, lane);
        double next = rho[n > 1 ? n - 2 : 0];
#pragma unroll 1
        for (int k = n - 1; k >= 0; --k) {
            const double after = rho[k > 2 ? k - 2 : 0];
            Op nx;
            eval<NQ, kHeld>(sm, H, next, nx, lane);
            apply(r, cur);
            cur = nx;
            next = after;
        }
    }

    // the slots' values at the nodes to divided differences, the odd entries taken over w / w_max first
    template <int NQ>
    static __device__ __forceinline__ void differences(SM* sm, int lane) {
        __syncwarp();
        for (int i = lane; i < ND * N * NA; i += 32) {
            const int d = i / (N * NA), col = i % (N * NA) / N, rw = i % N;
            const bool odd = (rw >= Z0) != (col >= Z0);
            double x[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                x[q] = col < N ? sm->T[d][q][col * LD + rw] : sm->phi[d][q][rw];
                if (odd) x[q] *= 1.0 / sqrt(train_node<NQ>(q));
            }
#pragma unroll
            for (int k = 1; k < NQ; ++k)
#pragma unroll
                for (int q = NQ - 1; q >= k; --q)
                    x[q] = (x[q] - x[q - 1]) * (1.0 / (train_node<NQ>(q) - train_node<NQ>(q - k)));
#pragma unroll
            for (int q = 0; q < NQ; ++q) (col < N ? sm->T[d][q][col * LD + rw] : sm->phi[d][q][rw]) = x[q];
        }
        __syncwarp();
    }

    // squarings for a norm, or -1 where the general path has to deal with it (not finite, or beyond the cap)
    static __device__ __forceinline__ int squarings(double nu, const TaylorTable& tt) {
        if (!(nu < INFINITY)) return -1;
        const int s = nu > tt.dense_theta ? (int)ceil(log2(nu / tt.dense_theta)) : 0;
        return s > 200 ? -1 : s;
    }
};

// Bound by the FP64 pipes, tensor and vector taking turns: 1.86 ms for 19,493 chains of 200 samples with four pools
// (dmma pipe 31% active, DFMA pipe 31%; 2.63 ms where the shape is not its own mirror image), where the Taylor action
// of every event took 31.6 ms.
// DT = 1: blockIdx.y is the tangent of the launch whose derivative the block forms, behind the values (tangent 0's
// blocks write the values too). One tangent costs three times a propagator; the Taylor action of every event with dual
// numbers took 12.6 ms for the three tangents of 714 chains (one pool, 10 pulses of 100 samples), this 0.53 ms.
template <int NC, int DT>
__global__ void __launch_bounds__(32 * TrainShape<NC>::warps(DT), TrainShape<NC>::blocks(DT))
train_kernel(const ChainArgs a, const TrainArgs tr, const __grid_constant__ TaylorTable tt) {
    using TR = Train<NC, DT>;
    using SH = TrainShape<NC>;
    using D = Dn<double, DT>;
    using C = Chain<NC, double, DT>;
    constexpr int N = SH::N, NT = SH::NT, Z0 = TR::Z0, ND = TR::ND;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    TrainSmem<NC, DT>* sm = reinterpret_cast<TrainSmem<NC, DT>*>(smem_raw) + warp;
    const long long pos = (long long)blockIdx.x * SH::warps(DT) + warp;
    if (pos >= a.chain_count || !(*tr.kinds & kTrained)) return;
    const long long nch = (long long)a.n_vox * a.n_off;
    long long ci = a.first_chain + pos;
    const int node = a.node_out ? (int)(ci / nch) : a.node_lo;
    if (a.node_out) ci -= node * nch;
    if (a.order) ci = a.order[ci];
    const int v = (int)(ci / a.n_off), o = (int)(ci % a.n_off);
    if (a.active && a.active[v] == 0) return;
    const TrainRow row = a.train[o];
    if (row.n == 0) return;                                   // no record of the row is marked
    const EvRec<double>* __restrict__ ev = reinterpret_cast<const EvRec<double>*>(a.ev) + o;

    for (int i = lane; i < ND * SH::kSlots * SH::TS; i += 32) (&sm->T[0][0][0])[i] = 0.0;
    for (int i = lane; i < ND * SH::kSlots * 8 * NT; i += 32) (&sm->phi[0][0][0])[i] = 0.0;
    ChainConst<NC, D> cc;
    C::load_const(a, v, node, cc, a.t0 + (int)blockIdx.y);
    const bool mt = cc.mt_on && cc.ls != 0;
    typename TR::Run r;
    TR::identity(r, lane);
    bool ok = true;
    if (ok) {
        // the pulse's matrix function at its nodes
        EvRec<double> rec = ev[(size_t)row.first * a.n_off];
        rec.w1 = row.w_max;
        rec.c = 1.0;
        rec.s = 0.0;
        D g = dconst<double, DT>(0.0);
        if (mt) {
            const D offmt = (rec.wf - cc.dw0) - cc.dwmt;
            g = cc.ls == 1 ? lorentzian<double, DT>(offmt, cc.t2mt)
                           : warp_super_lorentzian<DT>(offmt, cc.t2mt, cc.w0sl, lane);
        }
        StepCoef<NC, D> sc;
        C::event_coef(cc, rec, g, sc);
        const D w1 = sc.w1x;
        const int s = TR::squarings(rec.dt * C::coef_norm(sc, cc), tt);
        const int nq = s < 0 ? 0 : TR::interp_nodes(fabs(w1.v) * rec.dt, fabs(w1.v * w1.v * g.v) * rec.dt);
        ok = nq > 0;
        if (ok) {
            const double h = ldexp(rec.dt, -s);
            __syncwarp();
            if (lane == 0) TR::put_coef(sm->coef, sc, cc, h);
            if (lane < nq) {
                double u = 0.0;
#pragma unroll
                for (int q = 0; q < 6; ++q)
                    if (q == lane) u = nq == 4 ? train_node<4>(q < 4 ? q : 0) : train_node<6>(q);
                sm->coef.w1[lane] = (h * sqrt(u)) * w1;
                sm->coef.Rm[lane] = h * dfma(u * (w1 * w1), g, cc.Rm1);
            }
            __syncwarp();
            TR::exponentials(sm, lane, nq, s, tt);
            const double* rho = tr.rho + (size_t)o * tr.max_samples;
            bool half = false;
            if constexpr (DT == 0) {
                if (row.mirrored) {
                    half = true;
                    if (lane < 8 * NT) {
                        const double f = lane < N ? TR::balance(a.params, a.n_vox, v, lane, half) : 1.0;
                        sm->gv[lane] = lane >= NC + 1 && lane < 2 * (NC + 1) ? -f : f;
                    }
                    half = __all_sync(kFull, half);
                }
            }
            if (nq == 4) TR::template differences<4>(sm, lane);
            else TR::template differences<6>(sm, lane);
            if constexpr (DT == 0) {
                if (half) {
                    if (nq == 4) TR::template mirrored<4>(sm, r, rho, row.n, sm->gv, lane);
                    else TR::template mirrored<6>(sm, r, rho, row.n, sm->gv, lane);
                }
            }
            if (!half) {
                if (nq == 4) TR::template samples<4>(sm, r, rho, row.n, lane);
                else TR::template samples<6>(sm, r, rho, row.n, lane);
            }
        }
    }
    if (ok && row.gap > 0) {
        // the pulse waits in slot 1 for the events behind it
        __syncwarp();
        TR::put(sm, 1, r, lane);
        TR::identity(r, lane);
    }
    // the events after the pulse, from the last on: P <- P S E (S: a spoiler zeroes the transverse entries)
    for (int j = row.gap - 1; j >= 0 && ok; --j) {
        const EvRec<double> rec = ev[(size_t)(row.first + row.n + j) * a.n_off];
        const int type = (int)rec.type;
        if (type == EV_GRADIENT || type == EV_SPOILER) {
#pragma unroll
            for (int J = 0; J < NT; ++J)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    if (8 * J + 2 * (lane & 3) + e < Z0)
#pragma unroll
                        for (int I = 0; I < NT; ++I)
#pragma unroll
                            for (int d = 0; d < ND; ++d) r.P[d][I][J][e] = 0.0;
        }
        if (!(rec.dt > 1e-9)) continue;
        StepCoef<NC, D> sc;
        C::event_coef(cc, rec, dconst<double, DT>(0.0), sc);
        const int s = TR::squarings(rec.dt * C::coef_norm(sc, cc), tt);
        if (s < 0) {
            ok = false;
            break;
        }
        const double h = ldexp(rec.dt, -s);
        __syncwarp();
        if (lane == 0) {
            TR::put_coef(sm->coef, sc, cc, h);
            sm->coef.w1[0] = dconst<double, DT>(0.0);
            sm->coef.Rm[0] = h * sc.Rm1W;
        }
        __syncwarp();
        TR::exponentials(sm, lane, 1, s, tt);
        TR::step(sm, r, lane);
    }
    if (ok) {
        if (row.gap > 0) {
            typename TR::Op pulse;
            TR::load(sm, 1, pulse, lane);
            TR::apply(r, pulse);
        }
        // equal units in a row: P^run, by squaring and multiplying from the leading bit on
        if (row.run > 1) {
            __syncwarp();
            TR::put(sm, 1, r, lane);
            const int top = 31 - __clz(row.run);
            for (int b = top - 1; b >= 0; --b) {
                TR::put(sm, 0, r, lane);
                TR::step(sm, r, lane);
                if ((row.run >> b) & 1) {
                    // P^(2k + 1) = P^2k P: the multiplicand is in slot 1
                    __syncwarp();
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        for (int i = lane; i < SH::TS; i += 32) sm->T[d][0][i] = sm->T[d][1][i];
                        for (int i = lane; i < 8 * NT; i += 32) sm->phi[d][0][i] = sm->phi[d][1][i];
                    }
                    __syncwarp();
                    TR::step(sm, r, lane);
                }
            }
        }
        TR::sum_phi(r, lane);
        const int gg = lane >> 2, t = lane & 3;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            if (d == 0 && blockIdx.y != 0) continue;
            double* out = tr.prop + ((size_t)pos * tr.mats + (d ? 1 + blockIdx.y : 0)) * (N * SH::NS);
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                const int rw = 8 * I + gg;
                if (rw < N) {
#pragma unroll
                    for (int J = 0; J < NT; ++J)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (8 * J + 2 * t + e < N) out[rw * SH::NS + 8 * J + 2 * t + e] = r.P[d][I][J][e];
                    if (t == 0) out[rw * SH::NS + N] = r.f[d][I];
                }
            }
        }
    }
    if (lane == 0 && blockIdx.y == 0) {
        tr.ok[pos] = ok ? 1 : 0;
        if (!ok) atomicOr(tr.kinds, kRefused);
    }
}

}  // namespace bmc
