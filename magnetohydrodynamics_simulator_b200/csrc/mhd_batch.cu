// Host side of the batched C ABI (mhd_batch_* in include/mhd_b200.h): device memory plan of a
// batch of independent periodic simulations, the work-item lists of the batch kernels
// (mhd_batch.cuh), the launch sequence of one batched step, the CUDA-graph driver loop, the
// autotuner and per-instance diagnostics.
//
// Device memory: instance i owns 23 dense nx_i*ny_i FP64 planes (the same plan as a single
// context: S[6] state, T[6] predictor, A[6] accumulator, x, r[2], p[2]) plus its own StepCoeffs
// and DeviceStatus. The pool is plane-major: each of the 23 planes is one arena of all instances,
// instance i at the same zone offset in every arena, so a kernel reaches any plane of any instance
// from the arena bases (kernel parameters) and one offset. The descriptor array (BatchInst) is
// kept for even and odd steps, which differ only in the trading hydro planes of S and A.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "mhd_batch_solve.cuh"
#include "mhd_host_util.h"
#include "mhd_state_io.h"

using namespace mhd;

namespace {

constexpr int kBatchPlanes = 23;
constexpr int kQueues = 3;  // work counters: stage 1, stage 2, finalize

// Candidate decompositions the autotuner times: explicit-stage (rows per item, tail rows per
// item), solver rows (each with both decompositions).
constexpr int kStageCand[][2] = {{64, 0},   {128, 0},  {256, 0},  {128, 32}, {256, 32},
                                 {256, 64}, {512, 32}, {384, 32}, {192, 32}, {512, 64}};
// solver candidates (rows, order): even row ranges and fixed tiles of 32-256 rows, and tiles of a
// height chosen phase by phase (rows 0)
constexpr int kCgCand[][2] = {{32, 0}, {64, 0}, {128, 0}, {256, 0}, {32, 1}, {64, 1}, {128, 1}, {256, 1}, {0, 1}};

}  // namespace

struct mhd_batch {
    int count = 0;
    std::vector<mhd_params> prm;
    std::vector<size_t> ncell;
    size_t total_cells = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int device = 0;
    int num_sms = 0;
    double* pool = nullptr;
    StepCoeffs* coeffs = nullptr;    // [count]
    DeviceStatus* status = nullptr;  // [count]
    BatchInst* d_insts[2] = {nullptr, nullptr};
    std::vector<BatchInst> h_insts[2];
    int parity = 0;  // descriptor array of the next step
    ParamPlanes stage_base[2][2];  // [parity][stage - 1]: plane arenas of the explicit stages
    FinParams fin_base[2];         // [parity]: plane arenas of the finalize
    // work items of the explicit stages and of the finalize (the solver numbers its own)
    void* d_items_mem = nullptr;          // both lists in one allocation
    SweepItem* d_sweep_items = nullptr;  // explicit stages
    SweepItem* d_fin_items = nullptr;    // finalize
    size_t items_cap = 0;                // bytes
    int n_stage_items = 0;
    int n_fin_items = 0;
    int nchunks = 0;
    int stage_occ[2] = {0, 0}, fin_occ = 0, cg_occ = 0;
    int stage_grid[2] = {0, 0}, fin_grid = 0, cg_grid = 0;
    double* partials = nullptr;  // [2][CGB_MAX_INST][cg_occ * num_sms][4]
    CgSync* syncs = nullptr;     // [2 * nchunks] of k_cg_batch
    // solves (mhd_batch_solve.cuh), by chunk: instances that take a cluster, and all others
    struct SolveLists {
        std::vector<int> cluster, big;
        int cluster_off = 0, big_off = 0;  // in d_lists
    };
    std::vector<SolveLists> lists;
    int cluster_blocks = 0;
    size_t cluster_smem = 0;
    int solve_grid = 0;
    int* d_lists = nullptr;
    int* todo = nullptr;             // [count]
    BatchPlan* plans = nullptr;      // [CGB_MAX_INST]
    double* tile_partials = nullptr;
    CgSync* solve_syncs = nullptr;   // [nchunks] of k_solve_batch
    int* queues = nullptr;       // [kQueues]
    double* dt_dev = nullptr;    // [count] per-instance dt of mhd_batch_step
    double* divb_partial = nullptr;
    double* divb_out = nullptr;
    int divb_blocks = 0;
    DeviceStatus* host_status = nullptr;  // pinned [count]
    double* host_small = nullptr;         // pinned [8]
    std::vector<char> have_state;
    mhd_batch_tuning tuning{};
    double g = 0.0, d = 0.0;
    double timeout_s = 30.0;
    double* rec_dts = nullptr;       // [count][rec_cap]
    long long* rec_prods = nullptr;  // [count][rec_cap][2]
    int rec_cap = 0;
};

namespace {

mhd_status check_batch(mhd_batch* b) {
    if (!b) return MHD_ERR_INVALID_ARGUMENT;
    MHD_TRY(cudaSetDevice(b->device));
    return MHD_OK;
}

mhd_status check_index(mhd_batch* b, int index) {
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    return (index >= 0 && index < b->count) ? MHD_OK : MHD_ERR_INVALID_ARGUMENT;
}

bool all_states_set(const mhd_batch* b) {
    for (char h : b->have_state)
        if (!h) return false;
    return true;
}

int grid_for(int occ_blocks, int num_sms, int nitems, int warps_per_block) {
    const long long need = ((long long)nitems + warps_per_block - 1) / warps_per_block;
    return (int)std::max(1LL, std::min((long long)occ_blocks * num_sms, need));
}

// Smallest item height whose items (every 28-column strip cut into equal items of at most that
// many rows) number at most `waves` x `warps`, i.e. fill that many waves of the resident warps.
int balanced_rows(const mhd_batch* b, long long warps, int waves) {
    const long long slots = std::max(1LL, warps * waves);
    auto items_at = [&](int h) {
        long long n = 0;
        for (int i = 0; i < b->count; ++i)
            n += (long long)((b->prm[i].nx + SW_OUT - 1) / SW_OUT) * ((b->prm[i].ny + h - 1) / h);
        return n;
    };
    int lo = 1, hi = 1;
    for (int i = 0; i < b->count; ++i) hi = std::max(hi, b->prm[i].ny);
    if (items_at(hi) > slots) return hi;  // more strips than slots: whole strips
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (items_at(mid) <= slots) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}
int balanced_stage_rows(const mhd_batch* b, int waves) {
    return balanced_rows(b, (long long)std::min(b->stage_occ[0], b->stage_occ[1]) * b->num_sms * SW_WARPS,
                         waves);
}

// Items of at most `rows` rows (equal heights within a strip) over every strip, largest first.
void strip_items(const mhd_batch* b, int rows, int tail_rows, std::vector<SweepItem>& out) {
    for (int i = 0; i < b->count; ++i) {
        const int nx = b->prm[i].nx, ny = b->prm[i].ny;
        const int strips = (nx + SW_OUT - 1) / SW_OUT;
        const int big = std::min(rows, ny);
        const int tail_start = (tail_rows > 0) ? ny - big : ny;
        const int pieces = (tail_start + big - 1) / big;  // equal items over rows [0, tail_start)
        for (int sx = 0; sx < strips; ++sx) {
            for (int k = 0; k < pieces; ++k)
                out.push_back(SweepItem{i, sx, (int)((long long)k * tail_start / pieces),
                                        (int)((long long)(k + 1) * tail_start / pieces)});
            for (int r = tail_start; r < ny; r += tail_rows)
                out.push_back(SweepItem{i, sx, r, std::min(r + tail_rows, ny)});
        }
    }
    std::stable_sort(out.begin(), out.end(), [](const SweepItem& a, const SweepItem& c) {
        return (a.r1 - a.r0) > (c.r1 - c.r0);
    });
}

// Build the work-item lists and the descriptors' decomposition for tuning t, and upload both.
// Explicit stages: every 28-column strip of every instance is cut into equal items of at most
// stage_rows rows; with stage_tail_rows > 0 only the strip's first ny - min(stage_rows, ny) rows
// are, and the rest go in items of stage_tail_rows rows. Items run largest first (the kernels take
// them from a counter), so the small ones fill the end of the launch. Finalize: items that fill
// one wave of its resident warps (at least 16 rows), as a single context's finalize.
mhd_status apply_tuning(mhd_batch* b, const mhd_batch_tuning& t) {
    // cg_rows = 0: tiles whose height the solver chooses phase by phase (order 1 only)
    if (t.stage_rows < 1 || t.cg_rows < 0 || (t.cg_order != 0 && t.cg_order != 1) ||
        (t.cg_rows == 0 && t.cg_order != 1) || t.stage_tail_rows < 0)
        return MHD_ERR_INVALID_ARGUMENT;
    MHD_TRY(cudaStreamSynchronize(b->stream));  // in-flight steps still read the old lists
    std::vector<SweepItem> st_items, fin_items;
    strip_items(b, t.stage_rows, t.stage_tail_rows, st_items);
    strip_items(b, std::max(3, balanced_rows(b, (long long)b->fin_occ * b->num_sms * FS_WARPS, 1)), 0,
                fin_items);
    // solver: its grid covers the largest chunk at 8 or more rows per warp
    for (int p = 0; p < 2; ++p)
        for (int i = 0; i < b->count; ++i) b->h_insts[p][i].cg_strips_x = (b->prm[i].nx + CG_W - 1) / CG_W;
    long long max_chunk_rows = 0;
    for (int c = 0; c < b->nchunks; ++c) {
        const int i0 = c * CGB_MAX_INST, i1 = std::min(b->count, i0 + CGB_MAX_INST);
        long long n = 0;
        for (int i = i0; i < i1; ++i) n += (long long)((b->prm[i].nx + CG_W - 1) / CG_W) * b->prm[i].ny;
        max_chunk_rows = std::max(max_chunk_rows, n);
    }
    const int cg_warps = (int)std::min((max_chunk_rows + 7) / 8, (long long)1 << 30);
    b->n_stage_items = (int)st_items.size();
    b->n_fin_items = (int)fin_items.size();
    const size_t bytes = (st_items.size() + fin_items.size()) * sizeof(SweepItem);
    if (bytes > b->items_cap) {
        cudaFree(b->d_items_mem);
        b->d_items_mem = nullptr;
        b->items_cap = 0;
        MHD_TRY(cudaMalloc(&b->d_items_mem, bytes));
        b->items_cap = bytes;
    }
    b->d_sweep_items = static_cast<SweepItem*>(b->d_items_mem);
    b->d_fin_items = b->d_sweep_items + st_items.size();
    MHD_TRY(cudaMemcpy(b->d_sweep_items, st_items.data(), st_items.size() * sizeof(SweepItem),
                       cudaMemcpyHostToDevice));
    MHD_TRY(cudaMemcpy(b->d_fin_items, fin_items.data(), fin_items.size() * sizeof(SweepItem),
                       cudaMemcpyHostToDevice));
    for (int p = 0; p < 2; ++p)
        MHD_TRY(cudaMemcpy(b->d_insts[p], b->h_insts[p].data(), b->count * sizeof(BatchInst),
                           cudaMemcpyHostToDevice));
    b->stage_grid[0] = grid_for(b->stage_occ[0], b->num_sms, b->n_stage_items, SW_WARPS);
    b->stage_grid[1] = grid_for(b->stage_occ[1], b->num_sms, b->n_stage_items, SW_WARPS);
    b->fin_grid = grid_for(b->fin_occ, b->num_sms, b->n_fin_items, FS_WARPS);
    b->cg_grid = grid_for(b->cg_occ, b->num_sms, cg_warps, CGB_NW);
    b->tuning.stage_rows = t.stage_rows;
    b->tuning.cg_rows = t.cg_rows;
    b->tuning.cg_order = t.cg_order;
    b->tuning.stage_tail_rows = t.stage_tail_rows;
    return MHD_OK;
}

// Which instances' solves run in a cluster: those of at most CC's cells, in clusters of the fewest blocks that
// hold the largest of them, or of more while all clusters are resident at once. More than two waves of clusters
// take longer than the moment form: then the largest instances go there.
void plan_solves(mhd_batch* b) {
    std::vector<int> small;
    auto fits = [&](int i, int cs) { return cc_fits(b->prm[i].nx, b->prm[i].ny, cs); };
    for (int i = 0; i < b->count; ++i)
        if (fits(i, std::min(CC_MAX, b->prm[i].ny >= 8 ? 8 : (b->prm[i].ny >= 4 ? 4 : 1)))) small.push_back(i);
    std::stable_sort(small.begin(), small.end(), [&](int x, int y) { return b->ncell[x] > b->ncell[y]; });
    int cs = 0;
    while (!small.empty()) {
        cs = 1;
        auto all_fit = [&](int c) {
            for (int i : small)
                if (!fits(i, c)) return false;
            return true;
        };
        while (cs < CC_MAX && !all_fit(cs)) cs *= 2;
        if (all_fit(cs) && (long long)small.size() * cs <= 2LL * b->num_sms) break;
        small.erase(small.begin());
    }
    if (!small.empty()) {
        auto all_fit = [&](int c) {
            for (int i : small)
                if (!fits(i, c)) return false;
            return true;
        };
        while (cs < CC_MAX && (long long)small.size() * cs * 2 <= b->num_sms && all_fit(2 * cs)) cs *= 2;
    }
    b->cluster_blocks = cs;
    b->cluster_smem = 0;
    std::vector<char> in_cluster(b->count, 0);
    for (int i : small) {
        in_cluster[i] = 1;
        const int R = (b->prm[i].ny + cs - 1) / cs;
        b->cluster_smem = std::max(b->cluster_smem, (size_t)cc_smem_doubles(b->prm[i].nx, R) * sizeof(double));
    }
    b->lists.assign(b->nchunks, mhd_batch::SolveLists{});
    int off = 0;
    for (int c = 0; c < b->nchunks; ++c) {
        mhd_batch::SolveLists& L = b->lists[c];
        for (int i = c * CGB_MAX_INST; i < std::min(b->count, (c + 1) * CGB_MAX_INST); ++i)
            (in_cluster[i] ? L.cluster : L.big).push_back(i);
        L.cluster_off = off;
        off += (int)L.cluster.size();
        L.big_off = off;
        off += (int)L.big.size();
    }
}

mhd_status launch_cg_chunks(mhd_batch* b, const BatchInst* insts, int solve, bool record) {
    for (int c = 0; c < b->nchunks; ++c) {
        const mhd_batch::SolveLists& L = b->lists[c];
        if (!L.cluster.empty()) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)L.cluster.size() * b->cluster_blocks);
            cfg.blockDim = dim3(CC_NT);
            cfg.dynamicSmemBytes = b->cluster_smem;
            cfg.stream = b->stream;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = b->cluster_blocks;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            MHD_TRY(cudaLaunchKernelEx(&cfg, k_cluster_batch, insts, (const int*)(b->d_lists + L.cluster_off),
                                       b->cluster_blocks, solve, b->rec_cap, record ? b->rec_prods : nullptr,
                                       b->timeout_s));
        }
        if (L.big.empty()) continue;
        {
            SolveBatchArgs a{};
            a.insts = insts;
            a.list = b->d_lists + L.big_off;
            a.n = (int)L.big.size();
            a.solve = solve;
            a.partials = b->tile_partials;
            a.plans = b->plans;
            a.todo = b->todo;
            a.sync = b->solve_syncs + c;
            a.rec_stride = b->rec_cap;
            a.prods_rec = record ? b->rec_prods : nullptr;
            a.timeout_s = b->timeout_s;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(b->solve_grid);
            cfg.blockDim = dim3(CM_NT);
            cfg.dynamicSmemBytes = kCmSmemBytes;
            cfg.stream = b->stream;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            MHD_TRY(cudaLaunchKernelEx(&cfg, k_solve_batch, a));
        }
        CgBatchArgs a{};
        a.insts = insts;
        a.inst0 = c * CGB_MAX_INST;
        a.ninst = std::min(CGB_MAX_INST, b->count - a.inst0);
        a.order = b->tuning.cg_order;
        a.rows = b->tuning.cg_rows;
        a.partials = b->partials;
        a.sync = b->syncs + 2 * c + solve;
        a.todo = b->todo;
        a.solve_index = solve;
        a.rec_stride = b->rec_cap;
        a.prods_rec = record ? b->rec_prods : nullptr;
        a.timeout_s = b->timeout_s;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(b->cg_grid);
        cfg.blockDim = dim3(CGB_NT);
        cfg.dynamicSmemBytes = kCgbSmemBytes;
        cfg.stream = b->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        MHD_TRY(cudaLaunchKernelEx(&cfg, k_cg_batch, a));
    }
    return MHD_OK;
}

// One batched step with the descriptors of the current parity. dt_in: device array of per-instance
// dts or null (then dt_fixed for all; <= 0 selects the CFL step). run_mode: alpha rule of
// instances without a fixed coefficient (1: from dt, 2: the driver's rule). ev: 6 events around
// the kernels (stage 1, solve 0, stage 2, solve 1, finalize) or null.
mhd_status enqueue_step(mhd_batch* b, const double* dt_in, double dt_fixed, int run_mode,
                        double t_end, bool record, cudaEvent_t* ev) {
    const BatchInst* I = b->d_insts[b->parity];
    const int nthreads = std::max(std::max(b->count, 2 * b->nchunks), kQueues);
    k_batch_coeffs<<<(nthreads + 127) / 128, 128, 0, b->stream>>>(
        I, b->count, dt_in, dt_fixed, run_mode, t_end, b->g, b->d, record ? b->rec_dts : nullptr,
        b->rec_cap, b->queues, kQueues, b->syncs, 2 * b->nchunks);
    MHD_TRY(cudaGetLastError());
    if (ev) MHD_TRY(cudaEventRecord(ev[0], b->stream));
    k_stage_batch<1><<<b->stage_grid[0], 32 * SW_WARPS, sweep_smem_bytes(1), b->stream>>>(
        I, b->d_sweep_items, b->n_stage_items, b->queues, b->stage_base[b->parity][0]);
    MHD_TRY(cudaGetLastError());
    if (ev) MHD_TRY(cudaEventRecord(ev[1], b->stream));
    mhd_status s = launch_cg_chunks(b, I, 0, record);
    if (s != MHD_OK) return s;
    if (ev) MHD_TRY(cudaEventRecord(ev[2], b->stream));
    k_stage_batch<2><<<b->stage_grid[1], 32 * SW_WARPS, sweep_smem_bytes(2), b->stream>>>(
        I, b->d_sweep_items, b->n_stage_items, b->queues + 1, b->stage_base[b->parity][1]);
    MHD_TRY(cudaGetLastError());
    if (ev) MHD_TRY(cudaEventRecord(ev[3], b->stream));
    s = launch_cg_chunks(b, I, 1, record);
    if (s != MHD_OK) return s;
    if (ev) MHD_TRY(cudaEventRecord(ev[4], b->stream));
    k_finalize_batch<<<b->fin_grid, 32 * FS_WARPS, kFinSmemBytes, b->stream>>>(I, b->d_fin_items, b->n_fin_items,
                                                                   b->queues + 2, b->fin_base[b->parity]);
    MHD_TRY(cudaGetLastError());
    if (ev) MHD_TRY(cudaEventRecord(ev[5], b->stream));
    b->parity ^= 1;
    return MHD_OK;
}

mhd_status refresh_cfl(mhd_batch* b, int i) {
    const BatchInst& I = b->h_insts[b->parity][i];
    MHD_TRY(cudaMemsetAsync(&b->status[i].smax_bits, 0, sizeof(unsigned long long), b->stream));
    const int blocks = std::max(1, std::min((int)((b->ncell[i] + 255) / 256), b->num_sms * 8));
    CPlanes u;
    for (int k = 0; k < 6; ++k) u.f[k] = I.S[k];
    k_cfl_scan<<<blocks, 256, 0, b->stream>>>(I.D, u, b->status + i);
    MHD_TRY(cudaGetLastError());
    return MHD_OK;
}

mhd_status read_status(mhd_batch* b) {
    MHD_TRY(cudaMemcpyAsync(b->host_status, b->status, b->count * sizeof(DeviceStatus),
                            cudaMemcpyDeviceToHost, b->stream));
    MHD_TRY(cudaStreamSynchronize(b->stream));
    return MHD_OK;
}

mhd_status status_of(unsigned flags) {
    if (flags & kStatusTimeout) return MHD_ERR_TIMEOUT;
    if (flags & kStatusNonFinite) return MHD_ERR_NONFINITE;
    if (flags & kStatusCgNotConverged) return MHD_ERR_CG_NOT_CONVERGED;
    return MHD_OK;
}

int severity(mhd_status s) {
    switch (s) {
        case MHD_ERR_TIMEOUT: return 3;
        case MHD_ERR_NONFINITE: return 2;
        case MHD_ERR_CG_NOT_CONVERGED: return 1;
        default: return 0;
    }
}

}  // namespace

extern "C" {

mhd_status mhd_batch_create(const mhd_params* params, int count, void* stream, mhd_batch** out) {
    if (!params || !out || count < 1) return MHD_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    for (int i = 0; i < count; ++i) {
        const mhd_params& p = params[i];
        if (p.nx < 2 || p.ny < 2 || !(p.dx > 0) || !(p.dy > 0) || !(p.eta >= 0) ||
            (p.ct_mode != 0 && p.ct_mode != 1) || (long long)p.nx * p.ny > (1LL << 31))
            return MHD_ERR_INVALID_ARGUMENT;
    }
    if (!mhd_device_available()) return MHD_ERR_NO_DEVICE;
    mhd_batch* b = new (std::nothrow) mhd_batch();
    if (!b) return MHD_ERR_OUT_OF_MEMORY;
    auto fail = [&](mhd_status s) {
        mhd_batch_destroy(b);
        return s;
    };
    b->count = count;
    b->prm.assign(params, params + count);
    b->ncell.resize(count);
    b->have_state.assign(count, 0);
    b->g = (2.0 - sqrt(2.0)) / 2.0;     // solvers.hpp:41
    b->d = 1.0 - (1.0 / (2.0 * b->g));  // solvers.hpp:42
    b->timeout_s = 0.0;
    for (int i = 0; i < count; ++i) {
        mhd_params& p = b->prm[i];
        if (!(p.courant > 0)) p.courant = 0.5;
        if (!(p.safety > 0)) p.safety = 0.9;
        if (!(p.cg_timeout_s > 0)) p.cg_timeout_s = 30.0;
        b->timeout_s = std::max(b->timeout_s, p.cg_timeout_s);
        b->ncell[i] = (size_t)p.nx * (size_t)p.ny;
        b->total_cells += b->ncell[i];
    }
    b->nchunks = (count + CGB_MAX_INST - 1) / CGB_MAX_INST;
    if (cudaGetDevice(&b->device) != cudaSuccess) return fail(MHD_ERR_NO_DEVICE);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, b->device) != cudaSuccess) return fail(MHD_ERR_NO_DEVICE);
    b->num_sms = prop.multiProcessorCount;
    if (stream) {
        b->stream = (cudaStream_t)stream;
    } else {
        if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess)
            return fail(MHD_ERR_CUDA);
        b->own_stream = true;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->stage_occ[0], k_stage_batch<1>,
                                                      32 * SW_WARPS, sweep_smem_bytes(1)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->stage_occ[1], k_stage_batch<2>,
                                                      32 * SW_WARPS, sweep_smem_bytes(2)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->fin_occ, k_finalize_batch, 32 * FS_WARPS,
                                                      kFinSmemBytes) != cudaSuccess ||
        cudaFuncSetAttribute(k_cg_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kCgbSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->cg_occ, k_cg_batch, CGB_NT, kCgbSmemBytes) !=
            cudaSuccess ||
        b->stage_occ[0] < 1 || b->stage_occ[1] < 1 || b->fin_occ < 1 || b->cg_occ < 1) {
        cudaGetLastError();
        return fail(MHD_ERR_CUDA);
    }
    plan_solves(b);
    int solve_occ = 0;
    if (cudaFuncSetAttribute(k_solve_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCmSmemBytes) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_cluster_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(CC_SMEM_DOUBLES * sizeof(double))) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&solve_occ, k_solve_batch, CM_NT, kCmSmemBytes) != cudaSuccess ||
        solve_occ < 1) {
        cudaGetLastError();
        return fail(MHD_ERR_CUDA);
    }
    long long max_tiles = 1;  // of any chunk's passes, at the lowest tiles
    for (const mhd_batch::SolveLists& L : b->lists) {
        long long n = 0;
        for (int i : L.big)
            n += (long long)((b->prm[i].nx + cm_out(CM_MAXM, CM_C) - 1) / cm_out(CM_MAXM, CM_C)) *
                 ((b->prm[i].ny + kCmTileMinRows - 1) / kCmTileMinRows);
        max_tiles = std::max(max_tiles, n);
    }
    b->solve_grid = (int)std::min((long long)b->num_sms, (max_tiles + 3) / 4);
    b->cg_occ = std::min(b->cg_occ, std::max(1, mhd_host::env_int("MHD_B200_CG_BLOCKS_PER_SM", 1)));
    const size_t max_cg_grid = (size_t)b->cg_occ * b->num_sms;
    size_t max_cells = 0;
    for (size_t n : b->ncell) max_cells = std::max(max_cells, n);
    b->divb_blocks = std::max(1, std::min((int)((max_cells + 255) / 256), b->num_sms * 4));
    if (cudaMalloc(&b->pool, (size_t)kBatchPlanes * b->total_cells * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&b->coeffs, count * sizeof(StepCoeffs)) != cudaSuccess ||
        cudaMalloc(&b->status, count * sizeof(DeviceStatus)) != cudaSuccess ||
        cudaMalloc(&b->d_insts[0], count * sizeof(BatchInst)) != cudaSuccess ||
        cudaMalloc(&b->d_insts[1], count * sizeof(BatchInst)) != cudaSuccess ||
        cudaMalloc(&b->partials, 2 * (size_t)CGB_MAX_INST * max_cg_grid * 4 * sizeof(double)) !=
            cudaSuccess ||
        cudaMalloc(&b->syncs, 2 * (size_t)b->nchunks * sizeof(CgSync)) != cudaSuccess ||
        cudaMalloc(&b->d_lists, count * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&b->todo, count * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&b->plans, CGB_MAX_INST * sizeof(BatchPlan)) != cudaSuccess ||
        cudaMalloc(&b->tile_partials, (size_t)max_tiles * CM_NMU * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&b->solve_syncs, (size_t)b->nchunks * sizeof(CgSync)) != cudaSuccess ||
        cudaMalloc(&b->queues, kQueues * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&b->dt_dev, count * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&b->divb_partial, 2 * (size_t)b->divb_blocks * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&b->divb_out, 2 * sizeof(double)) != cudaSuccess ||
        cudaMallocHost(&b->host_status, count * sizeof(DeviceStatus)) != cudaSuccess ||
        cudaMallocHost(&b->host_small, 8 * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        return fail(MHD_ERR_OUT_OF_MEMORY);
    }
    // descriptors. The pool is plane-major: plane k (S 0-5, T 6-11, A 12-17, x, r0, r1, p0, p1)
    // is one arena of total_cells zones, with instance i at the same zone offset in every arena.
    for (int p = 0; p < 2; ++p) b->h_insts[p].assign(count, BatchInst{});
    const size_t tot = b->total_cells;
    size_t off = 0;
    for (int i = 0; i < count; ++i) {
        double* const q = b->pool + off;
        const mhd_params& p = b->prm[i];
        const size_t n = b->ncell[i];
        BatchInst I{};
        I.D.nx = p.nx;
        I.D.ny = p.ny;
        I.D.dx = p.dx;
        I.D.dy = p.dy;
        I.D.eta = p.eta;
        I.D.ct_mode = p.ct_mode;
        I.C = b->coeffs + i;
        I.st = b->status + i;
        I.off = (long long)off;
        for (int k = 0; k < 6; ++k) I.S[k] = q + (size_t)k * tot;
        for (int k = 0; k < 6; ++k) I.T[k] = q + (size_t)(6 + k) * tot;
        for (int k = 0; k < 6; ++k) I.A[k] = q + (size_t)(12 + k) * tot;
        I.x = q + 18 * tot;
        I.r[0] = q + 19 * tot;
        I.r[1] = q + 20 * tot;
        I.p[0] = q + 21 * tot;
        I.p[1] = q + 22 * tot;
        I.max_iters = p.cg_max_iters > 0 ? p.cg_max_iters : 2LL * (long long)n;
        I.tol = p.cg_tol > 0 ? p.cg_tol : 2.220446049250313e-16;
        I.alpha = 0.0;
        I.alpha_fixed = 0;
        I.hmin = std::min(p.dx, p.dy);
        I.courant = p.courant;
        I.safety = p.safety;
        b->h_insts[0][i] = I;
        for (int k = 0; k < 4; ++k) std::swap(I.S[k], I.A[k]);  // odd steps
        b->h_insts[1][i] = I;
        off += n;
    }
    // the arenas are instance 0's planes (offset 0)
    for (int p = 0; p < 2; ++p) {
        const BatchInst& I0 = b->h_insts[p][0];
        ParamPlanes& s1 = b->stage_base[p][0];
        ParamPlanes& s2 = b->stage_base[p][1];
        for (int k = 0; k < 6; ++k) {
            s1.in_.f[k] = I0.S[k];
            s1.a_.f[k] = I0.T[k];
            s1.b_.f[k] = I0.A[k];
            s2.in_.f[k] = I0.T[k];
            s2.a_.f[k] = nullptr;
            s2.b_.f[k] = I0.A[k];
        }
        s1.x_ = nullptr;
        s2.x_ = I0.x;
        FinParams& fp = b->fin_base[p];
        for (int k = 0; k < 6; ++k) fp.acc_.f[k] = I0.A[k];
        fp.x_ = I0.x;
        fp.bx_ = I0.S[4];
        fp.by_ = I0.S[5];
    }
    if (cudaMemsetAsync(b->status, 0, count * sizeof(DeviceStatus), b->stream) != cudaSuccess ||
        cudaMemsetAsync(b->coeffs, 0, count * sizeof(StepCoeffs), b->stream) != cudaSuccess ||
        cudaMemsetAsync(b->pool, 0, (size_t)kBatchPlanes * b->total_cells * sizeof(double),
                        b->stream) != cudaSuccess ||
        cudaMemsetAsync(b->syncs, 0, 2 * (size_t)b->nchunks * sizeof(CgSync), b->stream) !=
            cudaSuccess ||
        cudaMemsetAsync(b->solve_syncs, 0, (size_t)b->nchunks * sizeof(CgSync), b->stream) != cudaSuccess ||
        cudaMemsetAsync(b->todo, 0, count * sizeof(int), b->stream) != cudaSuccess)
        return fail(MHD_ERR_CUDA);
    for (const mhd_batch::SolveLists& L : b->lists) {
        if (cudaMemcpy(b->d_lists + L.cluster_off, L.cluster.data(), L.cluster.size() * sizeof(int),
                       cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(b->d_lists + L.big_off, L.big.data(), L.big.size() * sizeof(int), cudaMemcpyHostToDevice) !=
                cudaSuccess)
            return fail(MHD_ERR_CUDA);
    }
    mhd_batch_tuning t{};
    t.stage_rows = mhd_host::env_int("MHD_B200_BATCH_STAGE_ROWS", balanced_stage_rows(b, 2));
    t.stage_tail_rows = mhd_host::env_int("MHD_B200_BATCH_STAGE_TAIL_ROWS", 0);
    t.cg_rows = mhd_host::env_int("MHD_B200_BATCH_CG_ROWS", 128);
    t.cg_order = mhd_host::env_int("MHD_B200_BATCH_CG_ORDER", 0);
    const mhd_status s = apply_tuning(b, t);
    if (s != MHD_OK) return fail(s);
    *out = b;
    return MHD_OK;
}

mhd_status mhd_batch_destroy(mhd_batch* b) {
    if (!b) return MHD_ERR_INVALID_ARGUMENT;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    cudaFree(b->pool);
    cudaFree(b->coeffs);
    cudaFree(b->status);
    cudaFree(b->d_insts[0]);
    cudaFree(b->d_insts[1]);
    cudaFree(b->d_items_mem);
    cudaFree(b->partials);
    cudaFree(b->syncs);
    cudaFree(b->d_lists);
    cudaFree(b->todo);
    cudaFree(b->plans);
    cudaFree(b->tile_partials);
    cudaFree(b->solve_syncs);
    cudaFree(b->queues);
    cudaFree(b->dt_dev);
    cudaFree(b->divb_partial);
    cudaFree(b->divb_out);
    cudaFree(b->rec_dts);
    cudaFree(b->rec_prods);
    if (b->host_status) cudaFreeHost(b->host_status);
    if (b->host_small) cudaFreeHost(b->host_small);
    if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
    cudaGetLastError();
    delete b;
    return MHD_OK;
}

int mhd_batch_count(mhd_batch* b) { return b ? b->count : 0; }

void* mhd_batch_stream(mhd_batch* b) { return b ? (void*)b->stream : nullptr; }

int mhd_batch_launches_per_step(mhd_batch* b) {
    if (!b) return 0;
    int n = 4;  // coefficients, two stages, finalize; twice the chunks' solves
    for (const mhd_batch::SolveLists& L : b->lists) n += 2 * ((L.cluster.empty() ? 0 : 1) + (L.big.empty() ? 0 : 2));
    return n;
}

static mhd_status batch_copy_in(mhd_batch* b, int index, const double* const f[6],
                                cudaMemcpyKind kind) {
    mhd_status s = check_index(b, index);
    if (s != MHD_OK) return s;
    if (!f) return MHD_ERR_INVALID_ARGUMENT;
    for (int k = 0; k < 6; ++k)
        if (!f[k]) return MHD_ERR_INVALID_ARGUMENT;
    const BatchInst& I = b->h_insts[b->parity][index];
    if (kind == cudaMemcpyDeviceToDevice &&
        mhd_host::plain_state(f, I.S, b->ncell[index] * sizeof(double), b->device, false)) {
        b->have_state[index] = 1;
        return mhd_host::load_state(I.D, f, I.S, b->status + index, b->stream);
    }
    for (int k = 0; k < 6; ++k)
        MHD_TRY(cudaMemcpyAsync(I.S[k], f[k], b->ncell[index] * sizeof(double), kind, b->stream));
    b->have_state[index] = 1;
    return refresh_cfl(b, index);
}

static mhd_status batch_copy_out(mhd_batch* b, int index, double* const f[6], cudaMemcpyKind kind) {
    mhd_status s = check_index(b, index);
    if (s != MHD_OK) return s;
    if (!f) return MHD_ERR_INVALID_ARGUMENT;
    if (!b->have_state[index]) return MHD_ERR_NO_STATE;
    const BatchInst& I = b->h_insts[b->parity][index];
    if (kind == cudaMemcpyDeviceToDevice &&
        mhd_host::plain_state(f, I.S, b->ncell[index] * sizeof(double), b->device, true))
        return mhd_host::store_state(b->ncell[index], I.S, f, b->num_sms, b->stream);
    for (int k = 0; k < 6; ++k) {
        if (!f[k]) continue;
        MHD_TRY(cudaMemcpyAsync(f[k], I.S[k], b->ncell[index] * sizeof(double), kind, b->stream));
    }
    if (kind == cudaMemcpyDeviceToHost) MHD_TRY(cudaStreamSynchronize(b->stream));
    return MHD_OK;
}

mhd_status mhd_batch_set_state(mhd_batch* b, int index, const double* const f[6]) {
    return batch_copy_in(b, index, f, cudaMemcpyHostToDevice);
}
mhd_status mhd_batch_set_state_device(mhd_batch* b, int index, const double* const f[6]) {
    return batch_copy_in(b, index, f, cudaMemcpyDeviceToDevice);
}
mhd_status mhd_batch_get_state(mhd_batch* b, int index, double* const f[6]) {
    return batch_copy_out(b, index, f, cudaMemcpyDeviceToHost);
}
mhd_status mhd_batch_get_state_device(mhd_batch* b, int index, double* const f[6]) {
    return batch_copy_out(b, index, f, cudaMemcpyDeviceToDevice);
}

mhd_status mhd_batch_set_implicit_coefficient(mhd_batch* b, int index, double alpha) {
    mhd_status s = check_index(b, index);
    if (s != MHD_OK) return s;
    if (!(alpha >= 0) || !std::isfinite(alpha)) return MHD_ERR_INVALID_ARGUMENT;
    MHD_TRY(cudaStreamSynchronize(b->stream));  // in-flight steps read the descriptors
    for (int p = 0; p < 2; ++p) {
        b->h_insts[p][index].alpha = alpha;
        b->h_insts[p][index].alpha_fixed = 1;
        MHD_TRY(cudaMemcpy(b->d_insts[p] + index, &b->h_insts[p][index], sizeof(BatchInst),
                           cudaMemcpyHostToDevice));
    }
    return MHD_OK;
}

mhd_status mhd_batch_step(mhd_batch* b, const double* dts) {
    MHD_NVTX_RANGE("mhd_batch_step");
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    if (!all_states_set(b)) return MHD_ERR_NO_STATE;
    if (dts) {
        for (int i = 0; i < b->count; ++i)
            if (!std::isfinite(dts[i])) return MHD_ERR_INVALID_ARGUMENT;
        // pageable source: the call returns once the values are staged, so dts may be reused
        MHD_TRY(cudaMemcpyAsync(b->dt_dev, dts, b->count * sizeof(double), cudaMemcpyHostToDevice,
                                b->stream));
    }
    return enqueue_step(b, dts ? b->dt_dev : nullptr, 0.0, 1, 0.0, false, nullptr);
}

mhd_status mhd_batch_run(mhd_batch* b, int nsteps, double dt_fixed, double t_end, double* dts_out,
                         long long* prods_out) {
    MHD_NVTX_RANGE("mhd_batch_run");
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    if (!all_states_set(b)) return MHD_ERR_NO_STATE;
    if (nsteps < 0 || !std::isfinite(dt_fixed) || !std::isfinite(t_end)) return MHD_ERR_INVALID_ARGUMENT;
    if (nsteps == 0) return MHD_OK;
    if (nsteps > b->rec_cap) {
        MHD_TRY(cudaStreamSynchronize(b->stream));
        cudaFree(b->rec_dts);
        cudaFree(b->rec_prods);
        b->rec_dts = nullptr;
        b->rec_prods = nullptr;
        b->rec_cap = 0;
        MHD_TRY(cudaMalloc(&b->rec_dts, (size_t)b->count * nsteps * sizeof(double)));
        MHD_TRY(cudaMalloc(&b->rec_prods, (size_t)b->count * nsteps * 2 * sizeof(long long)));
        b->rec_cap = nsteps;
    }
    k_batch_driver_reset<<<(b->count + 127) / 128, 128, 0, b->stream>>>(b->d_insts[b->parity],
                                                                         b->count);
    MHD_TRY(cudaGetLastError());
    auto one_step = [&]() { return enqueue_step(b, nullptr, dt_fixed, 2, t_end, true, nullptr); };
    // Two consecutive steps (even and odd descriptors) form one CUDA graph, replayed nsteps/2 times.
    int done = 0;
    if (nsteps >= 4 && mhd_host::env_int("MHD_B200_NO_GRAPH", 0) == 0) {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        const int parity0 = b->parity;
        bool ok = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        if (ok) {
            const mhd_status r1 = one_step();
            const mhd_status r2 = (r1 == MHD_OK) ? one_step() : r1;
            ok = cudaStreamEndCapture(b->stream, &graph) == cudaSuccess && r1 == MHD_OK && r2 == MHD_OK;
            b->parity = parity0;  // the captured steps did not run
        }
        if (ok) ok = cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
        if (ok) {
            for (; done + 2 <= nsteps; done += 2) {
                if (cudaGraphLaunch(exec, b->stream) != cudaSuccess) {
                    ok = false;
                    break;
                }
            }
        }
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        if (!ok && done > 0) return MHD_ERR_CUDA;
    }
    for (; done < nsteps; ++done) {
        s = one_step();
        if (s != MHD_OK) return s;
    }
    if (dts_out)
        MHD_TRY(cudaMemcpy2DAsync(dts_out, (size_t)nsteps * sizeof(double), b->rec_dts,
                                  (size_t)b->rec_cap * sizeof(double), (size_t)nsteps * sizeof(double),
                                  b->count, cudaMemcpyDeviceToHost, b->stream));
    if (prods_out)
        MHD_TRY(cudaMemcpy2DAsync(prods_out, (size_t)nsteps * 2 * sizeof(long long), b->rec_prods,
                                  (size_t)b->rec_cap * 2 * sizeof(long long),
                                  (size_t)nsteps * 2 * sizeof(long long), b->count,
                                  cudaMemcpyDeviceToHost, b->stream));
    if (dts_out || prods_out) MHD_TRY(cudaStreamSynchronize(b->stream));
    return MHD_OK;
}

mhd_status mhd_batch_set_tuning(mhd_batch* b, const mhd_batch_tuning* t) {
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    if (!t) return MHD_ERR_INVALID_ARGUMENT;
    return apply_tuning(b, *t);
}

mhd_status mhd_batch_get_tuning(mhd_batch* b, mhd_batch_tuning* t) {
    if (!b || !t) return MHD_ERR_INVALID_ARGUMENT;
    *t = b->tuning;
    return MHD_OK;
}

// Autotuner: one CFL step of the current states per candidate, timed per kernel with events;
// the explicit-stage (row height, tail height) and the solver's (row height, dealing order) are chosen
// independently (they set disjoint kernels' decompositions). The solver's only sets k_cg_batch's: it stays as it is
// where the other forms settle every instance, so that a later solve's summation order does not hang on the noise of
// equal trials. States, device statuses, step coefficients and the descriptor parity are restored after every trial.
mhd_status mhd_batch_autotune(mhd_batch* b, mhd_batch_tuning* out) {
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    if (!all_states_set(b)) return MHD_ERR_NO_STATE;
    MHD_TRY(cudaStreamSynchronize(b->stream));
    const mhd_batch_tuning before = b->tuning;
    double* backup = nullptr;
    StepCoeffs* coeffs_bk = nullptr;
    DeviceStatus* status_bk = nullptr;
    cudaEvent_t ev[6] = {};
    struct Cleanup {
        double*& backup;
        StepCoeffs*& c;
        DeviceStatus*& st;
        cudaEvent_t* ev;
        ~Cleanup() {
            cudaFree(backup);
            cudaFree(c);
            cudaFree(st);
            for (int k = 0; k < 6; ++k)
                if (ev[k]) cudaEventDestroy(ev[k]);
        }
    } cleanup{backup, coeffs_bk, status_bk, ev};
    MHD_TRY(cudaMalloc(&backup, 6 * b->total_cells * sizeof(double)));
    MHD_TRY(cudaMalloc(&coeffs_bk, b->count * sizeof(StepCoeffs)));
    MHD_TRY(cudaMalloc(&status_bk, b->count * sizeof(DeviceStatus)));
    for (int k = 0; k < 6; ++k) MHD_TRY(cudaEventCreate(&ev[k]));
    const int parity0 = b->parity;
    auto planes_copy = [&](bool save) -> mhd_status {
        size_t off = 0;
        for (int i = 0; i < b->count; ++i) {
            const BatchInst& I = b->h_insts[parity0][i];
            for (int k = 0; k < 6; ++k) {
                double* bk = backup + off + (size_t)k * b->ncell[i];
                MHD_TRY(cudaMemcpyAsync(save ? bk : I.S[k], save ? I.S[k] : bk,
                                        b->ncell[i] * sizeof(double), cudaMemcpyDeviceToDevice,
                                        b->stream));
            }
            off += 6 * b->ncell[i];
        }
        MHD_TRY(cudaMemcpyAsync(save ? coeffs_bk : b->coeffs, save ? b->coeffs : coeffs_bk,
                                b->count * sizeof(StepCoeffs), cudaMemcpyDeviceToDevice, b->stream));
        MHD_TRY(cudaMemcpyAsync(save ? status_bk : b->status, save ? b->status : status_bk,
                                b->count * sizeof(DeviceStatus), cudaMemcpyDeviceToDevice, b->stream));
        // (a trial whose solve ran out of time: its status goes, so its barrier does)
        if (!save) MHD_TRY(cudaMemsetAsync(b->solve_syncs, 0, (size_t)b->nchunks * sizeof(CgSync), b->stream));
        b->parity = parity0;
        return MHD_OK;
    };
    if ((s = planes_copy(true)) != MHD_OK) return s;
    // explicit-stage candidates: the fixed list and items that fill 1-4 or 6 waves exactly
    std::vector<std::pair<int, int>> stage_cand;
    for (const auto& c : kStageCand) stage_cand.emplace_back(c[0], c[1]);
    for (int waves : {1, 2, 3, 4, 6}) stage_cand.emplace_back(balanced_stage_rows(b, waves), 0);
    const int nst = (int)stage_cand.size();
    constexpr int ncg = sizeof(kCgCand) / sizeof(kCgCand[0]);
    double best_stage = 1e300, best_cg = 1e300;
    int best_stage_rows = before.stage_rows, best_tail = before.stage_tail_rows;
    int best_cg_rows = before.cg_rows, best_order = before.cg_order;
    // trial -1 warms the kernels up; the others cover every explicit-stage candidate and, where it has work, every
    // solver candidate
    int ntrials = nst;
    bool solver = false;  // the step's second solve (the last to set todo) leaves an instance to k_cg_batch
    for (int trial = -1; trial < ntrials; ++trial) {
        mhd_batch_tuning t{};
        const int tk = std::max(trial, 0);
        t.stage_rows = stage_cand[tk % nst].first;
        t.stage_tail_rows = stage_cand[tk % nst].second;
        t.cg_rows = solver ? kCgCand[tk % ncg][0] : before.cg_rows;
        t.cg_order = solver ? kCgCand[tk % ncg][1] : before.cg_order;
        if ((s = apply_tuning(b, t)) != MHD_OK) return s;
        if ((s = enqueue_step(b, nullptr, 0.0, 1, 0.0, false, ev)) != MHD_OK) return s;
        MHD_TRY(cudaStreamSynchronize(b->stream));
        float ms[5];
        for (int k = 0; k < 5; ++k) MHD_TRY(cudaEventElapsedTime(&ms[k], ev[k], ev[k + 1]));
        if ((s = planes_copy(false)) != MHD_OK) return s;
        if (trial < 0) {
            std::vector<int> todo(b->count);
            MHD_TRY(cudaMemcpy(todo.data(), b->todo, b->count * sizeof(int), cudaMemcpyDeviceToHost));
            solver = std::any_of(todo.begin(), todo.end(), [](int v) { return v != 0; });
            if (solver) ntrials = std::max(nst, ncg);
            continue;
        }
        const double stage_ms = (double)ms[0] + ms[2] + ms[4];
        const double cg_ms = (double)ms[1] + ms[3];
        if (stage_ms < best_stage) {
            best_stage = stage_ms;
            best_stage_rows = t.stage_rows;
            best_tail = t.stage_tail_rows;
        }
        if (cg_ms < best_cg) {
            best_cg = cg_ms;
            best_cg_rows = t.cg_rows;
            best_order = t.cg_order;
        }
    }
    mhd_batch_tuning chosen{};
    chosen.stage_rows = best_stage_rows;
    chosen.stage_tail_rows = best_tail;
    chosen.cg_rows = best_cg_rows;
    chosen.cg_order = best_order;
    if ((s = apply_tuning(b, chosen)) != MHD_OK) return s;
    b->tuning.stage_ms = best_stage;
    b->tuning.cg_ms = best_cg;
    MHD_TRY(cudaStreamSynchronize(b->stream));
    if (out) *out = b->tuning;
    return MHD_OK;
}

mhd_status mhd_batch_synchronize(mhd_batch* b, mhd_status* per_instance) {
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    if ((s = read_status(b)) != MHD_OK) return s;
    mhd_status worst = MHD_OK;
    bool any = false;
    for (int i = 0; i < b->count; ++i) {
        const mhd_status si = status_of(b->host_status[i].flags);
        if (per_instance) per_instance[i] = si;
        if (severity(si) > severity(worst)) worst = si;
        any |= b->host_status[i].flags != 0;
    }
    if (any) {
        if (worst == MHD_ERR_TIMEOUT)
            MHD_TRY(cudaMemsetAsync(b->solve_syncs, 0, (size_t)b->nchunks * sizeof(CgSync), b->stream));
        for (int i = 0; i < b->count; ++i)
            if (b->host_status[i].flags)
                MHD_TRY(cudaMemsetAsync(&b->status[i].flags, 0, sizeof(unsigned int), b->stream));
        MHD_TRY(cudaStreamSynchronize(b->stream));
    }
    return worst;
}

mhd_status mhd_batch_last_cg_products(mhd_batch* b, long long* out) {
    mhd_status s = check_batch(b);
    if (s != MHD_OK) return s;
    if (!out) return MHD_ERR_INVALID_ARGUMENT;
    if ((s = read_status(b)) != MHD_OK) return s;
    for (int i = 0; i < b->count; ++i) {
        out[2 * i] = b->host_status[i].cg_products[0];
        out[2 * i + 1] = b->host_status[i].cg_products[1];
    }
    return MHD_OK;
}

mhd_status mhd_batch_cfl_dt(mhd_batch* b, int index, double* dt) {
    mhd_status s = check_index(b, index);
    if (s != MHD_OK) return s;
    if (!dt) return MHD_ERR_INVALID_ARGUMENT;
    if (!b->have_state[index]) return MHD_ERR_NO_STATE;
    MHD_TRY(cudaMemcpyAsync(b->host_small, &b->status[index].smax_bits, sizeof(unsigned long long),
                            cudaMemcpyDeviceToHost, b->stream));
    MHD_TRY(cudaStreamSynchronize(b->stream));
    double smaxv;
    memcpy(&smaxv, b->host_small, sizeof(double));
    const mhd_params& p = b->prm[index];
    const double h = std::min(p.dx, p.dy);  // diagnostics.hpp:52-86
    double dt_res = INFINITY;
    if (p.eta != 0.0) dt_res = h * h / (4.0 * p.eta);
    if (!(smaxv > 1e-8)) smaxv = std::max(smaxv, 1e-8);
    *dt = std::min(p.courant * h / smaxv, dt_res) * p.safety;
    return MHD_OK;
}

mhd_status mhd_batch_divb(mhd_batch* b, int index, double* rms, double* maxabs) {
    mhd_status s = check_index(b, index);
    if (s != MHD_OK) return s;
    if (!b->have_state[index]) return MHD_ERR_NO_STATE;
    const BatchInst& I = b->h_insts[b->parity][index];
    const int blocks = std::max(1, std::min((int)((b->ncell[index] + 255) / 256), b->divb_blocks));
    k_divb_partial<<<blocks, 256, 0, b->stream>>>(I.D, I.S[4], I.S[5], b->divb_partial);
    MHD_TRY(cudaGetLastError());
    k_divb_final<<<1, 32, 0, b->stream>>>(b->divb_partial, blocks, (long long)b->ncell[index],
                                          b->divb_out);
    MHD_TRY(cudaGetLastError());
    MHD_TRY(cudaMemcpyAsync(b->host_small, b->divb_out, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                            b->stream));
    MHD_TRY(cudaStreamSynchronize(b->stream));
    if (rms) *rms = b->host_small[0];
    if (maxabs) *maxabs = b->host_small[1];
    return MHD_OK;
}

}  // extern "C"
