// bmc_host.h -- what the host side's translation units share: errors, tables, workspaces, launch plans, and the
// declarations of the per-pool-count entry points (Impl<NC>, instantiated once per pool count in bmc_impl.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <initializer_list>

#include "../../include/bmc_b200.h"

#include "bmc_chain.cuh"

namespace bmc {

// sets the calling thread's message and returns `s`
bmc_status fail(bmc_status s, const char* fmt, ...);

#define CUDA_TRY(expr)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (expr);                                                                \
        if (e_ != cudaSuccess) return fail(BMC_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

// The Taylor tables: one per precision (BMC_F64, BMC_F32, BMC_MIXED), and for the primal passes of a fit the float64
// one without a float32 tail, as the tangent kernels have none: the tail's rounding (~1e-13 in Z) differs between the
// costs that a fit compares, and near a minimum a step lowers the cost by less.
constexpr int kTableFit = 3, kTables = 4;
bmc_status tables(int precision, const TaylorTable** out);
bmc_status host_table_of(const TaylorTable* tt, TaylorTable* out);
// the first of the sizes (each at most the one before) that the stream's workspace has or can be grown to; *taken: which
bmc_status workspace(std::initializer_list<size_t> sizes, cudaStream_t st, void** out, int* taken);
inline bmc_status workspace(size_t bytes, cudaStream_t st, void** out) {
    int taken;
    return workspace({bytes}, st, out, &taken);
}
bmc_status fill_spread(ChainArgs& a, const bmc_spread* sp);
bmc_status scan_blocks(const EvRec<double>* rec, int n_rows, int n_ev, int stride, int4* seg, cudaStream_t st);
bmc_status use_adjoint(const EvRec<double>* rec, const bmc_problem* pr, int n_tan, int* row_ev, int* flag,
                       cudaStream_t st, bool* ok);
size_t order_bytes(long long nch);

// Tangent mode (bmc_set_tangent_mode): BMC_TANGENTS_AUTO takes the adjoint kernel where it applies.
extern std::atomic<int> g_tangent_mode;

struct Carve {
    char* p;
    size_t used = 0;
    explicit Carve(void* base) : p((char*)base) {}
    template <typename T>
    T* take(size_t n) {
        used = (used + 255) & ~size_t(255);
        T* r = (T*)(p + used);
        used += n * sizeof(T);
        return r;
    }
};
inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// An uneven batch: voxels with their own event tables, one pool count. Owns its device buffers
// (preprocessed records of every table, the chain map, the sort scratch); built by bmc_uneven_create.
struct UnevenPlan {
    int dev = 0, n_cest = 0, n_vox = 0, mz = 0, reset = 1, n_tables = 0;
    long long n_chains = 0, n_rec = 0;
    EvRec<double>* rec = nullptr;
    int2* chain_map = nullptr;
    int* vox_table = nullptr;
    long long* tab_base = nullptr;
    int* tab_noff = nullptr;
    int* tab_nev = nullptr;
    int4* seg = nullptr;       // the repeated block of every row of every table
    int* tab_row0 = nullptr;   // first row of each table in seg
    double dense_switch = 0.0; // > 0: the dense path's norm threshold for this plan (bmc_uneven_set_dense_switch)
    int4* adj_blk = nullptr;   // per row: the block the adjoint block kernel takes (adjoint_block_rows_kernel)
    int adj_ok = 0;            // every row of every table qualifies: tangents go through that kernel
    void* scratch = nullptr;   // sort keys and indices, cub scratch, status word
    size_t scratch_bytes = 0;
};

// the scratch of a call without allocation (bmc_simulate_noalloc), in the library's static array
struct NoAllocScratch {
    int* status;
    int4* seg;      // every row's repeated block
    void* rec;      // the event records
    void* train;    // rows, amplitudes and propagators of shaped pulses
    size_t train_bytes;
    const TaylorTable* tt64;   // the float64 table, which the propagators are formed with
};

// Everything that is compiled per pool count.
template <int NC>
struct Impl {
    static bmc_status uneven(const UnevenPlan& pl, const double* params, const double* m0, const bmc_spread* sp,
                             const bmc_tangents* tg, const int32_t* active, double* z, double* jz, cudaStream_t st);
    static bmc_status simulate(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                               const bmc_spread* sp, double* out, cudaStream_t st, unsigned long long* work = nullptr);
    static bmc_status trajectory(const bmc_problem* pr, const double* params, const bmc_events* ev,
                                 const double* m0, double* traj, cudaStream_t st);
    static bmc_status jvp(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                          const bmc_spread* sp, const bmc_tangents* tg, double* z, double* jz, cudaStream_t st,
                          unsigned long long* work = nullptr);
    static bmc_status design(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                             const double* params_dir, const bmc_events* ev_dir, const double* m0_dir,
                             const bmc_tangents* tg, double* z, double* jz, double* dz, double* djz, cudaStream_t st);
    static bmc_status lm(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                         const bmc_spread* sp, const bmc_fit_spec* fs, const double* zm, const double* x0,
                         double* x_out, double* cost_traj, double* x_traj, cudaStream_t st);
    static bmc_status noalloc(const bmc_problem* pr, const double* params, const bmc_events* ev, const double* m0,
                              const bmc_spread* sp, double* out, const NoAllocScratch& ws, const TaylorTable* tt,
                              cudaStream_t st);
};

}  // namespace bmc
