// bmc_impl.cu -- the entry points of one pool count (Impl<BMC_NC>): every launch of a call, and the
// device-side Levenberg-Marquardt loop. Compiled once per pool count with -DBMC_NC=0 .. 5 (build.py), so that
// the instantiations build in parallel.
#include <cuda_runtime.h>

#include <type_traits>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>

#include "bmc_host.h"
#include "bmc_lm.cuh"
#include "bmc_adjoint.cuh"
#include "bmc_adjoint_block.cuh"
#include "bmc_design.cuh"
#include "bmc_train.cuh"

#ifndef BMC_NC
#error "compile with -DBMC_NC=<CEST pools>"
#endif

namespace bmc {
namespace {

template <typename R>
bmc_status prep_events(const bmc_problem* pr, const bmc_events* ev, EvRec<R>* out, cudaStream_t st) {
    const size_t n = (size_t)pr->n_offsets * pr->n_events;
    if (n == 0) return BMC_OK;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    prep_events_kernel<R><<<blocks, 256, 0, st>>>(pr->n_offsets, pr->n_events, ev->d_type, ev->d_dt, ev->d_rf_amp,
                                                  ev->d_rf_phase, ev->d_rf_freq, out);
    CUDA_TRY(cudaGetLastError());
    return BMC_OK;
}

template <int NC, typename R, int NT, bool U, bool COUNT>
bmc_status launch_chain_impl(ChainArgs a, const TaylorTable* tt, cudaStream_t st) {
    constexpr int kWarps = ChainLaunch<NC, NT>::kWarps;
    const size_t smem = kWarps * sizeof(DenseSmem<NC, typename DenseReal<R>::type, NT>) +
                        32 * kWarps * sizeof(ChainConst<NC, Dn<R, NT>>);
    // the attribute once per device and instantiation: later calls then only enqueue work (which keeps
    // them capturable in a CUDA graph). Atomic: calls on several devices may come from several threads.
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !((configured.load(std::memory_order_acquire) >> dev) & 1ull)) {
        CUDA_TRY(cudaFuncSetAttribute(chain_kernel<NC, R, NT, U, COUNT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_acq_rel);
    }
    long long nch = (U ? a.n_chains : (long long)a.n_vox * a.n_off) * (a.node_out ? a.n_nodes : 1);
    if (a.chain_count) nch = a.chain_count;
    a.cpw = chains_per_warp(nch, 1, kWarps, 1);
    const long long blocks = (nch + kWarps * a.cpw - 1) / (kWarps * a.cpw);
    if (blocks > 0x7fffffffLL) return fail(BMC_ERR_INVALID, "%lld chains exceed one launch", nch);
    if (blocks == 0) return BMC_OK;
    TaylorTable th;
    if (bmc_status s = host_table_of(tt, &th); s != BMC_OK) return s;
    chain_kernel<NC, R, NT, U, COUNT><<<(unsigned)blocks, kWarps * 32, smem, st>>>(a, th);
    CUDA_TRY(cudaGetLastError());
    return BMC_OK;
}

// the counting instantiation only where a.work asks for counts (the uneven plans never do)
template <int NC, typename R, int NT, bool U = false>
bmc_status launch_chain(const ChainArgs& a, const TaylorTable* tt, cudaStream_t st) {
    if constexpr (!U) {
        if (a.work) return launch_chain_impl<NC, R, NT, U, true>(a, tt, st);
    } else {
        if (a.work) return fail(BMC_ERR_UNSUPPORTED, "work counts of an uneven plan");
    }
    return launch_chain_impl<NC, R, NT, U, false>(a, tt, st);
}

template <int NC, bool kTan = true>
bmc_status launch_adjoint(ChainArgs a, const int* row_ev, int n_tan, const TaylorTable* tt, cudaStream_t st) {
    const size_t smem = kAdjWarps * AdjGroup<NC>::G * sizeof(AdjSlot<NC>);
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !((configured.load(std::memory_order_acquire) >> dev) & 1ull)) {
        CUDA_TRY(cudaFuncSetAttribute(adjoint_kernel<NC, kTan>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_acq_rel);
    }
    const long long nch = (long long)a.n_vox * a.n_off;   // (a device-side a.live bounds the pass itself)
    if constexpr (Sym<NC>::kFits) {
        // a thread per chain (the chains that it leaves are then the group kernel's); it reads water's z
        if (a.done && a.mz == Layout<NC>::izw && nch > 0) {
            TaylorTable th;
            if (bmc_status s = host_table_of(tt, &th); s != BMC_OK) return s;
            CUDA_TRY(cudaMemsetAsync(a.left, 0, sizeof(int), st));
            sym_kernel<NC, kTan><<<(unsigned)((nch + 127) / 128), 128, 0, st>>>(a, row_ev, n_tan, th, a.done);
            CUDA_TRY(cudaGetLastError());
        } else {
            a.done = nullptr;
        }
    }
    a.cpw = adjoint_chains_per_warp(nch, kTan ? 2 : BMC_ADJ_PRIMAL_BLOCKS, kAdjWarps, AdjGroup<NC>::G);
    const long long blocks = (nch + kAdjWarps * a.cpw - 1) / (kAdjWarps * a.cpw);
    if (blocks > 0x7fffffffLL) return fail(BMC_ERR_INVALID, "%lld chains exceed one launch", nch);
    if (blocks == 0) return BMC_OK;
    TaylorTable th;
    if (bmc_status s = host_table_of(tt, &th); s != BMC_OK) return s;
    adjoint_kernel<NC, kTan><<<(unsigned)blocks, kAdjWarps * 32, smem, st>>>(a, row_ev, n_tan, th);
    CUDA_TRY(cudaGetLastError());
    return BMC_OK;
}

template <int NC, bool kTan = true>
bmc_status launch_adjoint_block(ChainArgs a, const int4* blk, int n_tan, const TaylorTable* tt, cudaStream_t st) {
    const size_t smem = kAdjBlkWarps * DenseGroup<NC>::G * sizeof(AdjBlkSlot<NC, kTan>);
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !((configured.load(std::memory_order_acquire) >> dev) & 1ull)) {
        CUDA_TRY(cudaFuncSetAttribute(adjoint_block_kernel<NC, kTan>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_acq_rel);
    }
    // one round per warp: the rounds of a warp run one after another whatever its lanes hold, so short warps only
    // balance the launch better (192 voxels, 1 to 5 pools: 129 ms per joint fit with 32 chains per warp, 38 with as
    // many as the resident warps leave, 35 with one round)
    a.cpw = DenseGroup<NC>::G;
    const long long blocks = (a.n_chains + kAdjBlkWarps * a.cpw - 1) / (kAdjBlkWarps * a.cpw);
    if (blocks > 0x7fffffffLL) return fail(BMC_ERR_INVALID, "%lld chains exceed one launch", a.n_chains);
    if (blocks == 0) return BMC_OK;
    TaylorTable th;
    if (bmc_status s = host_table_of(tt, &th); s != BMC_OK) return s;
    adjoint_block_kernel<NC, kTan><<<(unsigned)blocks, kAdjBlkWarps * 32, smem, st>>>(a, blk, n_tan, th);
    CUDA_TRY(cudaGetLastError());
    return BMC_OK;
}

// Whether the nodes of a spread run as chains of their own (ChainArgs::node_out): where the chains alone fill less
// than half of the resident lanes, and the nodes' results take at most 256 MB. 101 chains of 16 nodes (five pools, 20
// pulses of 100 samples) took 1.37 s in 4 warps.
bool split_nodes(long long chains, const bmc_spread* sp, size_t values) {
    return sp && sp->n_nodes > 1 && chains < (long long)kSMs * BMC_FWD_MIN_BLOCKS * 4 * 16 &&
           values * sp->n_nodes * sizeof(double) <= (size_t(256) << 20);
}

template <typename R>
bmc_status sum_nodes(const ChainArgs& a, long long n, const double* part, double* out, cudaStream_t st) {
    node_sum_kernel<std::is_same<R, double>::value><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a, part, n, out);
    CUDA_TRY(cudaGetLastError());
    return BMC_OK;
}

// Order the chains by estimated cost: `order` and the sort's scratch are carved from `cv`.
template <int NC, typename R>
bmc_status order_chains(ChainArgs& a, Carve& cv, cudaStream_t st) {
    const long long nch = (long long)a.n_vox * a.n_off;
    if (nch < 2 * 128 || a.n_ev == 0) return BMC_OK;
    float* k_in = cv.take<float>(nch);
    float* k_out = cv.take<float>(nch);
    int* i_in = cv.take<int>(nch);
    int* i_out = cv.take<int>(nch);
    size_t tmp = 0;
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp, k_in, k_out, i_in, i_out, (int)nch, 0, 32, st));
    void* t = cv.take<char>(tmp);
    cost_kernel<NC, R><<<(unsigned)((nch + 127) / 128), 128, 0, st>>>(a, k_in, i_in);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(t, tmp, k_in, k_out, i_in, i_out, (int)nch, 0, 32, st));
    a.order = i_out;
    return BMC_OK;
}

// whether a chain's voxel is active
struct ActiveChain {
    const int* active;
    int n_off;
    __device__ __forceinline__ bool operator()(int chain) const { return active[chain / n_off] != 0; }
};

// The active voxels' chains in launch order, into `list`, their number into *count: an adjoint pass over a part of the
// voxels (a fit's tangents after rejected steps) then fills its warps. 2,048 voxels x 244 rows,
// 30 iterations of two values: 21.4 ms of tangent passes without, 8.1 ms with it (0.2 ms of selection).
size_t live_bytes(long long nch) {
    size_t tmp = 0;
    cub::DeviceSelect::If(nullptr, tmp, (const int*)nullptr, (int*)nullptr, (int*)nullptr, (int)nch, ActiveChain{});
    return align256(sizeof(int) * nch) + align256(tmp) + 512;
}
bmc_status live_chains(ChainArgs& a, int* list, int* count, void* tmp, size_t tmp_bytes, cudaStream_t st) {
    const int nch = (int)((long long)a.n_vox * a.n_off);
    CUDA_TRY(cub::DeviceSelect::If(tmp, tmp_bytes, a.order, list, count, nch, ActiveChain{a.active, a.n_off}, st));
    a.order = list;
    a.live = count;
    return BMC_OK;
}

// tangents per launch, by pool count (register budget of the dual-number state)
template <int NC>
constexpr int tangents_per_pass() { return NC <= 1 ? 2 : 1; }

// Shaped-pulse trains of a call: the rows' units and amplitudes, and the propagators (with those of `tangents`
// derivatives) of `chunk` chains at a time: whole waves of the chain kernel that applies them, as many as kTrainBytes
// hold and at least one (131 MB with four pools, 115 with five; 175 and 230 with a tangent), or waves of train_kernel's
// warps where fewer fit. A call of at most a chunk takes every chain in one launch. A larger one takes, chunk by chunk, the
// chains that have a propagator, and all others (rows without a train, chains whose propagator is refused) in launches over
// the whole order, for chunk by chunk each launch ends in a partly empty wave. 16,384 voxels x 101 rows, everything in
// chunks of 131,072 / now: 64 pulses without a train, four pools 19.6 / 17.3 ms; 20 block pulses, four pools 83 / 72; ten,
// five pools, in bmc_simulate_noalloc's static scratch (11,000 chains a chunk) 321 / 103. 4,096 voxels x 101 rows of 20
// shaped pulses: 28.6 / 28.6.
constexpr size_t kTrainBytes = size_t(160) << 20;
constexpr long long kTrainWindow = 1ll << 22;        // chains whose flags are kept at once
template <int NC>
struct Trains {
    int max_samples = 0, mats = 1;
    long long chunk = 0, window = 0;
    TrainArgs tr{};
    const TaylorTable* tt64 = nullptr;   // the float64 table, which the propagators are formed with

    // whether the table can have trains
    static bool wanted(const bmc_problem* pr, bool tangents) { return pr->n_events >= train_min_events<NC>(tangents); }

    size_t per_chain() const { return sizeof(double) * mats * TrainShape<NC>::N * TrainShape<NC>::NS; }
    size_t fixed_bytes(const bmc_problem* pr, int tangents) {
        max_samples = std::min(pr->n_events, kTrainMaxSamples);
        mats = 1 + tangents;
        return align256(sizeof(TrainRow) * pr->n_offsets) +
               align256(sizeof(double) * (size_t)max_samples * pr->n_offsets) + 1024;
    }
    // the scratch for `chains` chains, the propagators (and the chains' flags) in at most `most` bytes
    size_t bytes(const bmc_problem* pr, long long chains, int tangents, size_t most = ~size_t(0) >> 1) {
        const size_t fixed = fixed_bytes(pr, tangents);
        window = std::min(chains, kTrainWindow);
        // a wave of the chain kernel, more of them up to kTrainBytes; where not one fits, waves of train_kernel's warps
        const long long full = 128ll * kSMs * (tangents ? ChainLaunch<NC, 1>::kMinBlocks : ChainLaunch<NC, 0>::kMinBlocks);
        constexpr long long wave = (long long)TrainShape<NC>::warps(0) * TrainShape<NC>::blocks(0) * kSMs;
        const long long fit = (long long)((most - align256(window)) / per_chain());
        chunk = std::max<long long>(1, kTrainBytes / (full * per_chain())) * full;
        if (chunk > fit) chunk = fit >= full ? fit - fit % full : (fit >= wave ? fit - fit % wave : fit);
        chunk = std::min(chunk, window);
        return fixed + align256(chunk * per_chain()) + align256(window);
    }
    // carves the scratch, finds the rows' trains and marks the records `rec` (a.ev's)
    bmc_status scan(ChainArgs& a, EvRec<double>* rec, Carve& cv, cudaStream_t st) {
        TrainRow* rows = cv.take<TrainRow>(a.n_off);
        double* rho = cv.take<double>((size_t)max_samples * a.n_off);
        tr.rho = rho;
        tr.max_samples = max_samples;
        tr.prop = cv.take<double>((size_t)chunk * per_chain() / sizeof(double));
        tr.ok = cv.take<unsigned char>(window);
        tr.kinds = cv.take<int>(1);
        CUDA_TRY(cudaMemsetAsync(tr.kinds, 0, sizeof(int), st));
        train_scan_kernel<<<a.n_off, kTrainScanThreads, 0, st>>>(rec, a.n_ev, a.n_off, train_cost<NC>(mats > 1), a.seg, rows,
                                                                 rho, max_samples, tr.kinds);
        CUDA_TRY(cudaGetLastError());
        a.train = rows;
        a.prop = tr.prop;
        a.kinds = tr.kinds;
        return BMC_OK;
    }

    template <int DT>
    bmc_status form(const ChainArgs& a, unsigned char* ok, int tangents, cudaStream_t st) const {
        constexpr int kWarps = TrainShape<NC>::warps(DT);
        const size_t smem = kWarps * sizeof(TrainSmem<NC, DT>);
        static std::atomic<unsigned long long> configured{0};
        int dev = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        if (dev >= 64 || !((configured.load(std::memory_order_acquire) >> dev) & 1ull)) {
            CUDA_TRY(cudaFuncSetAttribute(train_kernel<NC, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            if (dev < 64) configured.fetch_or(1ull << dev, std::memory_order_acq_rel);
        }
        TaylorTable th;
        if (bmc_status s = host_table_of(tt64, &th); s != BMC_OK) return s;
        TrainArgs t = tr;
        t.mats = 1 + tangents;
        t.ok = ok;
        const dim3 grid((unsigned)((a.chain_count + kWarps - 1) / kWarps), DT ? tangents : 1);
        train_kernel<NC, DT><<<grid, 32 * kWarps, smem, st>>>(a, t, th);
        CUDA_TRY(cudaGetLastError());
        return BMC_OK;
    }

    // One pass over every chain with NT tangents. Per node where the nodes do not run as chains of their own: a chain's
    // nodes are added in their order.
    template <int NT>
    bmc_status pass(ChainArgs a, const TaylorTable* tt, cudaStream_t st) const {
        const long long all = (long long)a.n_vox * a.n_off * (a.node_out ? a.n_nodes : 1);
        const int nodes = a.node_out ? 1 : a.n_nodes;
        bmc_status s = BMC_OK;
        auto of_node = [&](int j) {
            if (a.node_out) return;
            a.node_lo = j;
            a.node_hi = j + 1;
        };
        auto with_propagators = [&](unsigned char* ok) {
            a.prop_ok = ok;
            const bmc_status e = form<(NT > 0 ? 1 : 0)>(a, ok, NT, st);
            return e != BMC_OK ? e : launch_chain<NC, double, NT>(a, tt, st);
        };
        if (all <= chunk) {
            a.parts = kEveryPart;
            a.chain_count = all;
            for (int j = 0; j < nodes; ++j) {
                of_node(j);
                if ((s = with_propagators(tr.ok)) != BMC_OK) return s;
            }
            return BMC_OK;
        }
        // the rows without a train: all nodes of a chain in one launch, or (one node) beside the refused chains
        a.parts = kPlain;
        if (nodes > 1 && (s = launch_chain<NC, double, NT>(a, tt, st)) != BMC_OK) return s;
        for (long long lo = 0; lo < all; lo += window) {
            const long long end = std::min(all, lo + window);
            for (int j = 0; j < nodes; ++j) {
                of_node(j);
                a.parts = kTrained;
                for (a.first_chain = lo; a.first_chain < end; a.first_chain += chunk) {
                    a.chain_count = std::min(chunk, end - a.first_chain);
                    if ((s = with_propagators(tr.ok + (a.first_chain - lo))) != BMC_OK) return s;
                }
                a.parts = kRefused | (nodes > 1 ? 0 : kPlain);
                a.first_chain = lo;
                a.chain_count = end - lo;
                a.prop_ok = tr.ok;
                if ((s = launch_chain<NC, double, NT>(a, tt, st)) != BMC_OK) return s;
            }
        }
        return BMC_OK;
    }
};

// every tangent, tangents_per_pass at a time; `trains`: the table's trains (null: none looked for)
template <int NC, bool U = false>
bmc_status run_tangents(ChainArgs a, int P, const TaylorTable* tt, cudaStream_t st, const Trains<NC>* trains = nullptr) {
    constexpr int TP = tangents_per_pass<NC>(), TP2 = TP >= 2 ? 2 : 1;
    a.n_tan = P;
    for (int t0 = 0; t0 < P; t0 += TP) {
        a.t0 = t0;
        const bool two = P - t0 >= 2 && TP >= 2;
        bmc_status s = BMC_OK;
        if constexpr (!U) {
            if (trains) {
                s = two ? trains->template pass<TP2>(a, tt, st) : trains->template pass<1>(a, tt, st);
                if (s != BMC_OK) return s;
                continue;
            }
        }
        s = two ? launch_chain<NC, double, TP2, U>(a, tt, st) : launch_chain<NC, double, 1, U>(a, tt, st);
        if (s != BMC_OK) return s;
    }
    if (a.node_out) {
        const long long nch = (long long)a.n_vox * a.n_off;
        bmc_status s = sum_nodes<double>(a, nch, a.node_out, a.out, st);
        return s != BMC_OK ? s : sum_nodes<double>(a, nch * P, a.node_jout, a.jout, st);
    }
    return BMC_OK;
}

// a primal pass, its nodes summed where they ran as chains of their own
template <int NC, typename R>
bmc_status run_primal(const ChainArgs& a, const TaylorTable* tt, cudaStream_t st, const Trains<NC>* trains = nullptr) {
    bmc_status s = BMC_OK;
    if constexpr (std::is_same<R, double>::value) {
        s = trains ? trains->template pass<0>(a, tt, st) : launch_chain<NC, R, 0>(a, tt, st);
    } else {
        s = launch_chain<NC, R, 0>(a, tt, st);
    }
    if (s != BMC_OK || !a.node_out) return s;
    return sum_nodes<R>(a, (long long)a.n_vox * a.n_off * (a.mz >= 0 ? 1 : Layout<NC>::N), a.node_out, a.out, st);
}

}  // namespace

// one simulation (or tangent set) of an uneven batch: chains sorted by estimated cost, outputs
// in canonical chain order (voxel-major, then table row)
template <int NC>
bmc_status Impl<NC>::uneven(const UnevenPlan& pl, const double* params, const double* m0, const bmc_spread* sp,
                         const bmc_tangents* tg, const int32_t* active, double* z, double* jz, cudaStream_t st) {
    const TaylorTable* tt = nullptr;
    bmc_status s = tables(BMC_F64, &tt);
    if (s != BMC_OK) return s;
    ChainArgs a{};
    a.n_vox = pl.n_vox; a.n_off = 1; a.n_ev = 0; a.n_fields = Layout<NC>::NF;
    a.mz = pl.mz; a.reset_after_adc = pl.reset;
    if ((s = fill_spread(a, sp)) != BMC_OK) return s;
    a.params = params; a.m0 = m0; a.out = z; a.jout = jz;
    a.ev = pl.rec;
    a.n_chains = pl.n_chains; a.chain_map = pl.chain_map; a.vox_table = pl.vox_table;
    a.tab_base = pl.tab_base; a.tab_noff = pl.tab_noff; a.tab_nev = pl.tab_nev;
    a.seg = pl.seg; a.tab_row0 = pl.tab_row0; a.active = active; a.dense_switch = pl.dense_switch;
    Carve cv(pl.scratch);
    a.status = cv.take<int>(1);
    CUDA_TRY(cudaMemsetAsync(a.status, 0, sizeof(int), st));
    // the plan's passes go to the block kernel where its rows qualify (forward mode keeps the chain kernel). Its warps
    // take a round of chains each, neighbours of one voxel: the cost sort would only delay them.
    const bool adj = pl.adj_ok && g_tangent_mode.load(std::memory_order_relaxed) == BMC_TANGENTS_AUTO;
    const long long nch = pl.n_chains;
    if (nch >= 2 * 128 && !adj) {
        float* k_in = cv.take<float>(nch);
        float* k_out = cv.take<float>(nch);
        int* i_in = cv.take<int>(nch);
        int* i_out = cv.take<int>(nch);
        size_t tmp = 0;
        CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp, k_in, k_out, i_in, i_out, (int)nch, 0, 32, st));
        void* t = cv.take<char>(tmp);
        if (cv.used > pl.scratch_bytes) return fail(BMC_ERR_INVALID, "uneven plan: scratch too small");
        cost_kernel<NC, double, true><<<(unsigned)((nch + 127) / 128), 128, 0, st>>>(a, k_in, i_in);
        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cub::DeviceRadixSort::SortPairs(t, tmp, k_in, k_out, i_in, i_out, (int)nch, 0, 32, st));
        a.order = i_out;
    }
    if (!tg) return adj ? launch_adjoint_block<NC, false>(a, pl.adj_blk, 0, tt, st)
                        : launch_chain<NC, double, 0, true>(a, tt, st);
    for (int t = 0; t < tg->n_tangents; ++t) a.field_row[t] = tg->field_row[t];
    a.seed = tg->d_seed;
    a.dm0 = tg->d_dm0;
    if (adj && tg->n_tangents >= 2) return launch_adjoint_block<NC, true>(a, pl.adj_blk, tg->n_tangents, tt, st);
    return run_tangents<NC, true>(a, tg->n_tangents, tt, st);
}

template <int NC>
bmc_status Impl<NC>::simulate(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                           const bmc_spread* sp, double* out, cudaStream_t st, unsigned long long* work) {
    const TaylorTable* tt = nullptr;
    bmc_status s = tables(pr->precision, &tt);
    if (s != BMC_OK) return s;
    const size_t nrec = (size_t)pr->n_offsets * pr->n_events;
    void* ws = nullptr;
    const size_t recb = pr->precision == BMC_F32 ? sizeof(EvRec<float>) : sizeof(EvRec<double>);
    const long long nch = (long long)pr->n_voxels * pr->n_offsets;
    const size_t per_node = (size_t)nch * (pr->mz_loc >= 0 ? 1 : Layout<NC>::N);
    bool split = split_nodes(nch, sp, per_node);
    const size_t part = split ? per_node * sp->n_nodes : 0;
    Trains<NC> tn;
    // the counting calls integrate event by event: their counts are the work of that
    bool trains = pr->precision != BMC_F32 && !work && Trains<NC>::wanted(pr, false);
    const size_t least = align256(nrec * recb) + 256 + align256(sizeof(int4) * pr->n_offsets) + order_bytes(nch);
    const size_t nodes = least + align256(part * sizeof(double));
    int taken = 0;
    if ((s = workspace({nodes + (trains ? tn.bytes(pr, split ? nch * sp->n_nodes : nch, 0) : 0), nodes, least}, st, &ws,
                       &taken)) != BMC_OK)
        return s;
    trains = trains && taken < 1;
    split = split && taken < 2;
    Carve cv(ws);
    ChainArgs a{};
    a.n_vox = pr->n_voxels; a.n_off = pr->n_offsets; a.n_ev = pr->n_events; a.n_fields = Layout<NC>::NF;
    a.mz = pr->mz_loc; a.reset_after_adc = pr->reset_after_adc;
    if ((s = fill_spread(a, sp)) != BMC_OK) return s;
    a.params = params; a.m0 = m0; a.out = out; a.work = work;
    a.status = cv.take<int>(1);
    CUDA_TRY(cudaMemsetAsync(a.status, 0, sizeof(int), st));
    if (split) a.node_out = cv.take<double>(part);
    if (pr->precision == BMC_F32) {
        EvRec<float>* rec = cv.take<EvRec<float>>(nrec);
        if ((s = prep_events<float>(pr, ev, rec, st)) != BMC_OK) return s;
        a.ev = rec;
        if ((s = order_chains<NC, float>(a, cv, st)) != BMC_OK) return s;
        return run_primal<NC, float>(a, tt, st);
    }
    EvRec<double>* rec = cv.take<EvRec<double>>(nrec);
    if ((s = prep_events<double>(pr, ev, rec, st)) != BMC_OK) return s;
    a.ev = rec;
    a.seg = cv.take<int4>(pr->n_offsets);
    if ((s = scan_blocks(rec, pr->n_offsets, pr->n_events, pr->n_offsets, const_cast<int4*>(a.seg), st)) != BMC_OK)
        return s;
    if ((s = order_chains<NC, double>(a, cv, st)) != BMC_OK) return s;
    if (!trains) return run_primal<NC, double>(a, tt, st);
    if ((s = tables(BMC_F64, &tn.tt64)) != BMC_OK || (s = tn.scan(a, rec, cv, st)) != BMC_OK) return s;
    return run_primal<NC, double>(a, tt, st, &tn);
}

template <int NC>
bmc_status Impl<NC>::trajectory(const bmc_problem* pr, const double* params, const bmc_events* ev,
                             const double* m0, double* traj, cudaStream_t st) {
    const TaylorTable* tt = nullptr;
    bmc_status s = tables(BMC_F64, &tt);
    if (s != BMC_OK) return s;
    const size_t nrec = (size_t)pr->n_offsets * pr->n_events;
    void* ws = nullptr;
    if ((s = workspace(align256(nrec * sizeof(EvRec<double>)) + 256 + align256(sizeof(double) * pr->n_voxels * pr->n_offsets), st, &ws)) != BMC_OK) return s;
    Carve cv(ws);
    ChainArgs a{};
    a.n_vox = pr->n_voxels; a.n_off = pr->n_offsets; a.n_ev = pr->n_events; a.n_fields = Layout<NC>::NF;
    a.mz = Layout<NC>::izw; a.reset_after_adc = pr->reset_after_adc;
    fill_spread(a, nullptr);
    a.params = params; a.m0 = m0; a.traj = traj;
    a.status = cv.take<int>(1);
    a.out = cv.take<double>((size_t)pr->n_voxels * pr->n_offsets);
    CUDA_TRY(cudaMemsetAsync(a.status, 0, sizeof(int), st));
    EvRec<double>* rec = cv.take<EvRec<double>>(nrec);
    if ((s = prep_events<double>(pr, ev, rec, st)) != BMC_OK) return s;
    a.ev = rec;
    return launch_chain<NC, double, 0>(a, tt, st);
}

template <int NC>
bmc_status Impl<NC>::jvp(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                      const bmc_spread* sp, const bmc_tangents* tg, double* z, double* jz, cudaStream_t st,
                      unsigned long long* work) {
    const TaylorTable* tt = nullptr;
    bmc_status s = tables(BMC_F64, &tt);
    if (s != BMC_OK) return s;
    const size_t nrec = (size_t)pr->n_offsets * pr->n_events;
    void* ws = nullptr;
    const long long nch = (long long)pr->n_voxels * pr->n_offsets;
    const size_t per_node = (size_t)nch * (1 + tg->n_tangents);
    bool split = split_nodes(nch, sp, per_node);
    const size_t part = split ? (size_t)nch * sp->n_nodes : 0;
    Trains<NC> tn;
    bool trains = !work && Trains<NC>::wanted(pr, true);               // counting calls: event by event
    const size_t train_bytes = trains ? tn.bytes(pr, split ? nch * sp->n_nodes : nch, tangents_per_pass<NC>()) : 0;
    const size_t least = align256(nrec * sizeof(EvRec<double>)) + 256 + align256(sizeof(int4) * pr->n_offsets) +
                         align256(sizeof(int) * pr->n_offsets) + 1024 + order_bytes(nch) + align256(nch);
    const size_t nodes = least + align256(part * (1 + tg->n_tangents) * sizeof(double)) + 512;
    int taken = 0;
    if ((s = workspace({nodes + train_bytes, nodes, least}, st, &ws, &taken)) != BMC_OK) return s;
    trains = trains && taken < 1;
    split = split && taken < 2;
    Carve cv(ws);
    ChainArgs a{};
    a.n_vox = pr->n_voxels; a.n_off = pr->n_offsets; a.n_ev = pr->n_events; a.n_fields = Layout<NC>::NF;
    a.mz = pr->mz_loc; a.reset_after_adc = pr->reset_after_adc;
    if ((s = fill_spread(a, sp)) != BMC_OK) return s;
    a.params = params; a.m0 = m0; a.out = z; a.jout = jz; a.work = work;
    for (int t = 0; t < tg->n_tangents; ++t) a.field_row[t] = tg->field_row[t];
    a.seed = tg->d_seed; a.dm0 = tg->d_dm0;
    a.status = cv.take<int>(1);
    CUDA_TRY(cudaMemsetAsync(a.status, 0, sizeof(int), st));
    EvRec<double>* rec = cv.take<EvRec<double>>(nrec);
    if ((s = prep_events<double>(pr, ev, rec, st)) != BMC_OK) return s;
    a.ev = rec;
    a.seg = cv.take<int4>(pr->n_offsets);
    if ((s = scan_blocks(rec, pr->n_offsets, pr->n_events, pr->n_offsets, const_cast<int4*>(a.seg), st)) != BMC_OK)
        return s;
    int* row_ev = cv.take<int>(pr->n_offsets);
    int* flag = cv.take<int>(1);
    bool adj = false;
    if ((s = use_adjoint(rec, pr, tg->n_tangents, row_ev, flag, st, &adj)) != BMC_OK) return s;
    if ((s = order_chains<NC, double>(a, cv, st)) != BMC_OK) return s;
    if (adj) {
        if (Sym<NC>::kFits) {
            a.left = cv.take<int>(1);
            a.done = cv.take<unsigned char>(nch);
        }
        return launch_adjoint<NC>(a, row_ev, tg->n_tangents, tt, st);
    }
    if (split) {
        a.node_out = cv.take<double>(part);
        a.node_jout = cv.take<double>(part * tg->n_tangents);
    }
    if (!trains) return run_tangents<NC>(a, tg->n_tangents, tt, st);
    tn.tt64 = tt;
    if ((s = tn.scan(a, rec, cv, st)) != BMC_OK) return s;
    return run_tangents<NC>(a, tg->n_tangents, tt, st, &tn);
}

// Z, its tangents and the derivatives of both along one design direction (design_kernel): one launch
// per tangent, the direction's records prepared beside the table's
template <int NC>
bmc_status Impl<NC>::design(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                         const double* params_dir, const bmc_events* ev_dir, const double* m0_dir,
                         const bmc_tangents* tg, double* z, double* jz, double* dz, double* djz, cudaStream_t st) {
    const TaylorTable* tt = nullptr;
    bmc_status s = tables(BMC_F64, &tt);
    if (s != BMC_OK) return s;
    const size_t nrec = (size_t)pr->n_offsets * pr->n_events;
    const long long nch = (long long)pr->n_voxels * pr->n_offsets;
    constexpr int N = Layout<NC>::N;
    const size_t mats = (size_t)nch * (2 * N * N + N);           // Phi, its square, psi per chain
    void* ws = nullptr;
    if ((s = workspace(2 * align256(nrec * sizeof(EvRec<double>)) + 256 + align256(mats * sizeof(Dn<HD, 1>)),
                       st, &ws)) != BMC_OK)
        return s;
    Carve cv(ws);
    ChainArgs a{};
    a.n_vox = pr->n_voxels; a.n_off = pr->n_offsets; a.n_ev = pr->n_events; a.n_fields = Layout<NC>::NF;
    a.mz = pr->mz_loc; a.reset_after_adc = pr->reset_after_adc;
    if ((s = fill_spread(a, nullptr)) != BMC_OK) return s;
    a.params = params; a.params_dir = params_dir; a.m0 = m0; a.out = z; a.jout = jz;
    for (int t = 0; t < tg->n_tangents; ++t) a.field_row[t] = tg->field_row[t];
    a.seed = tg->d_seed;
    a.status = cv.take<int>(1);
    CUDA_TRY(cudaMemsetAsync(a.status, 0, sizeof(int), st));
    EvRec<double>* rec = cv.take<EvRec<double>>(nrec);
    if ((s = prep_events<double>(pr, ev, rec, st)) != BMC_OK) return s;
    a.ev = rec;
    DesignArgs d{};
    if (ev_dir && nrec > 0) {
        EvRec<double>* dr = cv.take<EvRec<double>>(nrec);
        const int blocks = (int)std::min<size_t>((nrec + 255) / 256, 148 * 16);
        prep_dir_kernel<<<blocks, 256, 0, st>>>(pr->n_offsets, pr->n_events, ev->d_rf_phase, ev_dir->d_dt,
                                               ev_dir->d_rf_amp, ev_dir->d_rf_phase, ev_dir->d_rf_freq, dr);
        CUDA_TRY(cudaGetLastError());
        d.ev_dir = dr;
    }
    d.m0_dir = m0_dir; d.dz = dz; d.djz = djz;
    d.scratch = reinterpret_cast<double*>(cv.take<Dn<HD, 1>>(mats));
    const long long blocks = (nch + 127) / 128;
    if (blocks > 0x7fffffffLL) return fail(BMC_ERR_INVALID, "%lld chains exceed one launch", nch);
    for (int t = 0; t < tg->n_tangents; ++t) {
        a.t0 = t;
        design_kernel<NC, 1><<<(unsigned)blocks, 128, 0, st>>>(a, d, tt);
        CUDA_TRY(cudaGetLastError());
    }
    return BMC_OK;
}

template <int NC>
bmc_status Impl<NC>::lm(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                     const bmc_spread* sp, const bmc_fit_spec* fs, const double* zm, const double* x0,
                     double* x_out, double* cost_traj, double* x_traj, cudaStream_t st) {
    const TaylorTable* tt = nullptr;
    bmc_status s = tables(BMC_F64, &tt);
    if (s != BMC_OK) return s;
    const int nv = pr->n_voxels, no = pr->n_offsets, P = fs->n_params;
    constexpr int NF = Layout<NC>::NF, N = Layout<NC>::N;
    const size_t nrec = (size_t)no * pr->n_events;
    bool split = split_nodes((long long)nv * no, sp, (size_t)nv * no * (1 + P));
    const size_t part = split ? (size_t)nv * no * sp->n_nodes : 0;
    Trains<NC> tn;
    bool trains = Trains<NC>::wanted(pr, true);
    const size_t least = align256(nrec * sizeof(EvRec<double>)) + 2 * align256(sizeof(double) * NF * nv) +
                         2 * align256(sizeof(double) * N * nv) + 2 * align256(sizeof(double) * nv) +
                         align256(sizeof(double) * P * nv) + align256(sizeof(double) * P * nv * N) +
                         2 * align256(sizeof(double) * nv * no) + align256(sizeof(double) * P * nv * no) +
                         2 * align256(sizeof(double) * nv * P) + 2 * align256(sizeof(double) * nv) +
                         align256(sizeof(int) * nv) + align256(sizeof(int4) * no) + 4096 +
                         align256(sizeof(int) * no) + 1024 + order_bytes((long long)nv * no) + align256((size_t)nv * no) +
                         live_bytes((long long)nv * no);
    const size_t nodes = least + align256(part * (1 + P) * sizeof(double)) + 512;
    void* ws = nullptr;
    int taken = 0;
    if ((s = workspace({nodes + (trains ? tn.bytes(pr, (long long)nv * no * (split ? sp->n_nodes : 1), tangents_per_pass<NC>())
                                        : 0), nodes, least}, st, &ws, &taken)) != BMC_OK)
        return s;
    trains = trains && taken < 1;
    split = split && taken < 2;
    Carve cv(ws);
    EvRec<double>* rec = cv.take<EvRec<double>>(nrec);
    double* px = cv.take<double>((size_t)NF * nv);
    double* pt = cv.take<double>((size_t)NF * nv);
    double* m0x = cv.take<double>((size_t)N * nv);
    double* m0t = cv.take<double>((size_t)N * nv);
    double* sgx = cv.take<double>(nv);
    double* sgt = cv.take<double>(nv);
    double* seed = cv.take<double>((size_t)P * nv);
    double* dm0 = cv.take<double>((size_t)P * nv * N);
    double* z = cv.take<double>((size_t)nv * no);
    double* zt = cv.take<double>((size_t)nv * no);
    double* J = cv.take<double>((size_t)P * nv * no);
    double* x = cv.take<double>((size_t)nv * P);
    double* xt = cv.take<double>((size_t)nv * P);
    double* lam = cv.take<double>(nv);
    double* cost = cv.take<double>(nv);
    int* need = cv.take<int>(nv);
    int4* seg = cv.take<int4>(no);
    int* status = cv.take<int>(1);
    int* row_ev = cv.take<int>(no);
    int* flag = cv.take<int>(1);
    if ((s = prep_events<double>(pr, ev, rec, st)) != BMC_OK) return s;
    CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), st));
    CUDA_TRY(cudaMemcpyAsync(x, x0, sizeof(double) * nv * P, cudaMemcpyDeviceToDevice, st));
    std::vector<double> hl(nv, fs->lam0);
    std::vector<int> hn(nv, 1);
    CUDA_TRY(cudaMemcpyAsync(lam, hl.data(), sizeof(double) * nv, cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemcpyAsync(need, hn.data(), sizeof(int) * nv, cudaMemcpyHostToDevice, st));

    SlotSpec ss{};
    ss.P = P;
    bool has_m = false;
    for (int p = 0; p < P; ++p) {
        ss.field_row[p] = fs->field_row[p]; ss.mode[p] = fs->mode[p]; ss.scale[p] = fs->scale[p];
        ss.lo[p] = fs->lo[p]; ss.hi[p] = fs->hi[p];
        has_m = has_m || fs->field_row[p] == BMC_SLOT_M_START;
    }
    ChainArgs a{};
    a.n_vox = nv; a.n_off = no; a.n_ev = pr->n_events; a.n_fields = NF;
    a.mz = pr->mz_loc; a.reset_after_adc = pr->reset_after_adc;
    if ((s = fill_spread(a, sp)) != BMC_OK) return s;
    const double* sig0 = sp ? sp->d_sigma_hz : nullptr;
    a.ev = rec; a.status = status; a.seg = seg;
    if ((s = scan_blocks(rec, no, pr->n_events, no, seg, st)) != BMC_OK) return s;
    bool adj = false;
    if ((s = use_adjoint(rec, pr, P, row_ev, flag, st, &adj)) != BMC_OK) return s;
    a.params = params; a.m0 = m0;
    if ((s = order_chains<NC, double>(a, cv, st)) != BMC_OK) return s;
    if (split && !adj) {
        a.node_out = cv.take<double>(part);
        a.node_jout = cv.take<double>(part * P);
    }
    if (adj && Sym<NC>::kFits) {
        a.left = cv.take<int>(1);
        a.done = cv.take<unsigned char>((size_t)nv * no);
    }
    int *live_list = nullptr, *live_count = nullptr;
    void* live_tmp = nullptr;
    size_t live_tmp_bytes = 0;
    if (adj && a.order) {
        const int nch = nv * no;
        CUDA_TRY(cub::DeviceSelect::If(nullptr, live_tmp_bytes, a.order, live_list, live_count, nch, ActiveChain{}, st));
        live_list = cv.take<int>(nch);
        live_count = cv.take<int>(1);
        live_tmp = cv.take<char>(live_tmp_bytes);
    }
    const TaylorTable* ttf = nullptr;
    if ((s = tables(kTableFit, &ttf)) != BMC_OK) return s;
    const Trains<NC>* tp = trains && !adj ? &tn : nullptr;
    tn.tt64 = tt;
    if (tp && (s = tn.scan(a, rec, cv, st)) != BMC_OK) return s;
    for (int p = 0; p < P; ++p) a.field_row[p] = fs->field_row[p] == BMC_SLOT_M_START ? BMC_SEED_NONE : fs->field_row[p];
    const int vb = (nv + 127) / 128, wb = (nv + 3) / 4;
    for (int it = 0; it < fs->n_iter; ++it) {
        // residual and Jacobian at x, for the voxels whose x moved
        lm_params_kernel<NC><<<vb, 128, 0, st>>>(nv, ss, params, m0, sig0, x, fs->d_free, px, m0x,
                                                  sp ? sgx : nullptr, seed, has_m ? dm0 : nullptr);
        CUDA_TRY(cudaGetLastError());
        ChainArgs aj = a;
        aj.params = px; aj.m0 = m0x; aj.sigma = sp ? sgx : nullptr; aj.seed = seed; aj.dm0 = has_m ? dm0 : nullptr;
        aj.active = need; aj.out = z; aj.jout = J;
        if (live_list && it > 0 &&
            (s = live_chains(aj, live_list, live_count, live_tmp, live_tmp_bytes, st)) != BMC_OK)
            return s;
        if ((s = adj ? launch_adjoint<NC>(aj, row_ev, P, tt, st) : run_tangents<NC>(aj, P, tt, st, tp)) != BMC_OK)
            return s;
        lm_solve_kernel<<<wb, 128, 0, st>>>(nv, no, fs->n_points_skip, it, ss, z, zm, J, fs->d_free, x, lam, cost, xt);
        CUDA_TRY(cudaGetLastError());
        // the trial point
        lm_params_kernel<NC><<<vb, 128, 0, st>>>(nv, ss, params, m0, sig0, xt, fs->d_free, pt, m0t,
                                                  sp ? sgt : nullptr, nullptr, nullptr);
        CUDA_TRY(cudaGetLastError());
        ChainArgs at = a;
        at.params = pt; at.m0 = m0t; at.sigma = sp ? sgt : nullptr; at.out = zt;
        // the trial point's Z: with the adjoint tangents, the same dense layout without H
        if ((s = adj ? launch_adjoint<NC, false>(at, row_ev, 0, tt, st) : run_primal<NC, double>(at, ttf, st, tp)) !=
            BMC_OK)
            return s;
        lm_accept_kernel<<<wb, 128, 0, st>>>(nv, no, fs->n_points_skip, P, it, fs->n_iter, zt, zm, cost, xt, x,
                                             lam, need, cost_traj, x_traj);
        CUDA_TRY(cudaGetLastError());
    }
    CUDA_TRY(cudaMemcpyAsync(x_out, x, sizeof(double) * nv * P, cudaMemcpyDeviceToDevice, st));
    return BMC_OK;
}

namespace {

template <int NC, typename R>
bmc_status run_noalloc(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                       const bmc_spread* sp, double* out, const NoAllocScratch& ws, const TaylorTable* tt,
                       cudaStream_t st) {
    ChainArgs a{};
    a.n_vox = pr->n_voxels; a.n_off = pr->n_offsets; a.n_ev = pr->n_events; a.n_fields = Layout<NC>::NF;
    a.mz = pr->mz_loc; a.reset_after_adc = pr->reset_after_adc;
    bmc_status s = fill_spread(a, sp);
    if (s != BMC_OK) return s;
    a.params = params; a.m0 = m0; a.out = out;
    a.status = ws.status;
    CUDA_TRY(cudaMemsetAsync(a.status, 0, sizeof(int), st));          // must start at zero each call
    EvRec<R>* rec = static_cast<EvRec<R>*>(ws.rec);
    if ((s = prep_events<R>(pr, ev, rec, st)) != BMC_OK) return s;   // overwrites the previous call's
    a.ev = rec;
    if constexpr (std::is_same<R, double>::value) {
        if ((s = scan_blocks(rec, pr->n_offsets, pr->n_events, pr->n_offsets, ws.seg, st)) != BMC_OK) return s;
        a.seg = ws.seg;
        Trains<NC> tn;
        if (Trains<NC>::wanted(pr, false)) {
            // as many chains at a time as the static array holds (its size covers every table's amplitudes)
            tn.bytes(pr, (long long)pr->n_voxels * pr->n_offsets, 0, ws.train_bytes - tn.fixed_bytes(pr, 0));
            tn.tt64 = ws.tt64;
            Carve cv(ws.train);
            if ((s = tn.scan(a, rec, cv, st)) != BMC_OK) return s;
            return run_primal<NC, double>(a, tt, st, &tn);
        }
    }
    return launch_chain<NC, R, 0>(a, tt, st);
}

}  // namespace

template <int NC>
bmc_status Impl<NC>::noalloc(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                             const bmc_spread* sp, double* out, const NoAllocScratch& ws, const TaylorTable* tt,
                             cudaStream_t st) {
    return pr->precision == BMC_F32 ? run_noalloc<NC, float>(pr, params, ev, m0, sp, out, ws, tt, st)
                                    : run_noalloc<NC, double>(pr, params, ev, m0, sp, out, ws, tt, st);
}

template struct Impl<BMC_NC>;

}  // namespace bmc
