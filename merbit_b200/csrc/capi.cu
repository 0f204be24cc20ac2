// C ABI: plan lifetime, SpMV dispatch, tuning, error reporting.
//
// The plan plays the part of the reference's per-call setup in Fun_Merbit
// (include/tile.cuh:563-615: offset build, TILE construction, y/z buffers),
// done once and reused: the partition for the chosen tile size and the
// carry slots stay resident in HBM across launches.
#include <algorithm>
#include <chrono>
#include <map>
#include <mutex>
#include <tuple>

#include "merbit_internal.cuh"

namespace merbit {

namespace {
thread_local std::string g_detail;
thread_local int g_last_cuda = 0;
thread_local bool g_no_memory = false;
}  // namespace

void set_error_detail(const std::string& s) { g_detail = s; }

int fail(int status, const std::string& detail) {
    g_detail = detail;
    g_no_memory = false;
    return status;
}

int cuda_fail(cudaError_t e, const char* where) {
    g_last_cuda = (int)e;
    g_no_memory = e == cudaErrorMemoryAllocation;
    g_detail = std::string(where) + ": " + cudaGetErrorString(e);
    // un-latch a non-sticky error so that a later launch check of this
    // thread does not report it again (a sticky error stays)
    cudaGetLastError();
    return MERBIT_ERR_CUDA;
}

bool out_of_memory() { return g_no_memory; }

namespace {

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// Gives the plan carry words for `tiles` tiles (both parity arrays start empty:
// all ones).  A smaller block is kept, words and epoch, until the plan is
// destroyed: a captured launch that holds its address stays valid.  The fill is
// ordered on s; callers synchronize s before a launch on another stream can use
// the words.
int grow_carry(merbit_plan_s* p, int tiles, cudaStream_t s) {
    if (tiles <= p->carry.slots) return MERBIT_OK;
    const bool first = p->carry.words == nullptr;  // takes the plan's own launch state
    const size_t bytes = sizeof(unsigned long long) * 4 * (size_t)tiles;
    SpmvCarry c;
    int st = dev_alloc(&c.words, bytes + (first ? 0 : sizeof(LaunchState)), s);
    if (st != MERBIT_OK) return st;
    c.slots = tiles;
    c.state = first ? p->state : reinterpret_cast<LaunchState*>(c.words + 4 * (size_t)tiles);
    cudaError_t e = cudaMemsetAsync(c.words, 0xFF, bytes, s);
    if (e == cudaSuccess && !first) {
        LaunchState init = {};
        init.epoch = 1u;
        e = cudaMemcpyAsync(c.state, &init, sizeof(init), cudaMemcpyHostToDevice, s);
    }
    if (e != cudaSuccess) {
        dev_free(c.words, s);
        return cuda_fail(e, "carry slots");
    }
    if (!first) p->old_carries.push_back(p->carry);
    p->carry = c;
    return MERBIT_OK;
}

}  // namespace

int plan_partition(merbit_plan_s* p, int tile_items, const Partition** out, cudaStream_t s) {
    for (auto& q : p->parts)
        if (q.tile_items == tile_items) {
            *out = &q;
            return MERBIT_OK;
        }
    Partition q;
    const int st = build_partition_async(p->row_ptr, p->nrow, p->nnz, tile_items, &q, s);
    if (st != MERBIT_OK) {
        dev_free(q.coords, s);
        return st;
    }
    p->parts.push_back(q);
    *out = &p->parts.back();
    return MERBIT_OK;
}

namespace {

// The partition of an SpMV configuration, with its largest rows-per-tile and
// carry words for its tiles.  (SpMM and batch launches take any rows per tile and
// bring words of their own, SpmmSlots: they need the coordinates alone.)
int spmv_partition(merbit_plan_s* p, int tile_items, const Partition** out, cudaStream_t s) {
    int st = plan_partition(p, tile_items, out, s);
    if (st != MERBIT_OK) return st;
    const bool rows = (*out)->max_rows < 0, words = (*out)->num_tiles > p->carry.slots;
    if (!rows && !words) return MERBIT_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    MERBIT_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone)  // before anything is queued
        return fail(MERBIT_ERR_INVALID,
                    "the stream is being captured and the plan has not run this configuration: "
                    "select it (or make its first product) before capture");
    int h_max = (*out)->max_rows;
    if (words) st = grow_carry(p, (*out)->num_tiles, s);
    if (st == MERBIT_OK && rows) {
        st = max_rows_async(**out, &p->scratch->max_rows, s);
        if (st == MERBIT_OK) {
            const cudaError_t e = cudaMemcpyAsync(&h_max, &p->scratch->max_rows, sizeof(int),
                                                  cudaMemcpyDeviceToHost, s);
            if (e != cudaSuccess) st = cuda_fail(e, "partition: max rows");
        }
    }
    const cudaError_t e = cudaStreamSynchronize(s);  // the partition, whatever failed
    if (st != MERBIT_OK) return st;
    if (e != cudaSuccess) return cuda_fail(e, "partition");
    const_cast<Partition*>(*out)->max_rows = h_max;
    return MERBIT_OK;
}

// Whether configuration idx can run this plan (builds its partition).
int plan_config_ok(merbit_plan_s* p, int idx, bool* ok, cudaStream_t s) {
    *ok = false;
    const SpmvConfig c = spmv_config(p->dtype, idx);
    if (!spmv_config_allowed(c, p->vec)) return MERBIT_OK;
    if (c.kind == 3) {  // row groups: no partition, any matrix
        *ok = true;
        return MERBIT_OK;
    }
    const Partition* part = nullptr;
    int st = spmv_partition(p, spmv_tile_items(c), &part, s);
    if (st != MERBIT_OK) return st;
    *ok = part->max_rows <= spmv_config_row_cap(c);
    return MERBIT_OK;
}

// The untuned choice for a matrix whose longest row is short: row groups, -1
// for the merge-path kernels.  Measured on B200 against the merge-path default
// (us; FP64 / FP32; longest row, mean):
//   27-point stencil 160^3 (27, 26.7)      250 / 177   against 503 / 411
//   5-point Laplacian 2048^2 (5, 5)        108 /  64   against 111 /  96
//   random rows of 3 and of 12             91 / 78 and 63 / 54   against 98 / 92, 89 / 74
//   random rows of 28, of 64, of 0 to 100  101 / 91, 118 / 113, 105 / 98
//                                          against 131 / 109, 163 / 128, 127 / 103
//   random rows of 2                       56 / 50   against 55 / 45 (not taken)
// Short rows (mean below 14, none above 32) go one per lane through shared
// memory, longer ones to 4 lanes, from a mean of 40 to 8: rows of 12 take 63
// us at one lane and 65 at 4, of 16 135 and 90; of 32 95 at 4 lanes and 93 at 8, of
// 64 85 and 72 (FP64).  Above 128 entries a row the rule leaves the matrix to
// the merge path, which balances any rows.
// A group of lanes waits for the longest row of its warp.  Where the longest is
// more than 2.5 times the mean, that is made up for only while the merge path's
// tiles do not fill the device: skew (longest / mean) times rows up to 4.2 million,
// twice that for 4-byte x when a row fills its 4 lanes (mean 3.75).  Row groups /
// merge path, us, FP64 and FP32 (rows of a, a fraction f of b):
//   rows       a, b, f           skew  FP64          FP32
//   2,000,000  3, 40, 0.01       11.9   66 /  65      64 /  51   not taken
//   2,000,000  0, 128, 0.1       10.0  201 / 164     193 / 148   not taken
//   500,000    3, 128, 0.01      30.0   31 /  25      26 /  29   not taken
//   500,000    6, 128, 0.02      15.2   39 /  35      31 /  40   FP32 alone
//   500,000    10, 128, 0.05      8.1   59 /  60      48 /  50   taken
//   200,000    2, 64, 0.03       16.7   12 /  13      11 /  13   taken
//   60,000     3, 128, 0.01      29.7   11 /  11       7 /  11   taken
// (Arrays off 16 bytes go to CTA tiles otherwise, which lose more.)
constexpr int kShortRows = 128;
int short_rows_choice(const merbit_plan_s* p) {
    if (p->max_row_len < 1 || p->max_row_len > kShortRows) return -1;
    const double rows = (double)std::max(p->nrow, 1);
    const double mean = (double)p->nnz / rows;
    if (mean < 2.5) return -1;
    const bool lane_per_row = mean < 14.0 && p->max_row_len <= 32;
    if (!lane_per_row && p->vec) {
        const double skew = (double)p->max_row_len / mean;
        const double most = p->dtype != MERBIT_F64 && mean >= 3.75 ? 8.5e6 : 4.2e6;
        if (skew > 2.5 && skew * rows > most) return -1;
    }
    const int lanes = lane_per_row ? 1 : mean < 40.0 ? 4 : 8;
    for (int i = 0, n = spmv_num_configs(p->dtype); i < n; ++i) {
        const SpmvConfig c = spmv_config(p->dtype, i);
        if (c.kind == 3 && c.ipt == lanes && !c.cg && (c.stg != 0) == lane_per_row) return i;
    }
    return -1;
}

// First usable configuration in table order; when the tiles of the first end
// more rows than its row_ptr window holds (runs of empty and one-entry rows, as
// in R-MAT graphs), the first whose window holds a tile of row ends.
int plan_pick_default(merbit_plan_s* p, cudaStream_t s) {
    const int n = spmv_num_configs(p->dtype);
    for (int pass = 0; pass < 2; ++pass)
        for (int i = 0; i < n; ++i) {
            const SpmvConfig c = spmv_config(p->dtype, i);
            const bool early = i == 0 || (c.kind == 1 && c.stg);
            if (early != (pass == 0)) continue;
            bool ok = false;
            int st = plan_config_ok(p, i, &ok, s);
            if (st != MERBIT_OK) return st;
            if (ok) {
                p->cfg = i;
                return MERBIT_OK;
            }
        }
    return fail(MERBIT_ERR_UNSUPPORTED, "no SpMV configuration fits this matrix");
}

// Grows the plan's residual partials to hold one word per CTA of any launch
// over `num_tiles` tiles (warp-tile kernel: at most 32 resident CTAs per SM;
// CTA-tile kernel: one CTA per tile).
int plan_partials(merbit_plan_s* p, int num_tiles, cudaStream_t s) {
    int sms = 0;
    MERBIT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device));
    const long long need = std::max<long long>(num_tiles, 32LL * std::max(sms, 1));
    if (need <= p->npartials) return MERBIT_OK;
    double* words = nullptr;
    int st = dev_alloc(&words, sizeof(double) * (size_t)need, s);
    if (st != MERBIT_OK) return st;
    if (p->partials) p->owned.push_back(p->partials);  // captured launches may hold it
    p->partials = words;
    p->npartials = need;
    return MERBIT_OK;
}

// y = alpha A x + beta z (z NULL: y); residual != NULL also writes
// *residual = sum_r |y[r] - x[r]| from the same launch.
int run_spmv(merbit_plan_s* p, int cfg, double alpha, const void* x, double beta, void* y,
             cudaStream_t s, const void* z = nullptr, double* residual = nullptr) {
    const SpmvConfig c = spmv_config(p->dtype, cfg);
    const Partition* part = nullptr;
    int st = MERBIT_OK;
    if (c.kind != 3) {
        st = spmv_partition(p, spmv_tile_items(c), &part, s);
        if (st != MERBIT_OK) return st;
    }
    if (residual) {
        st = plan_partials(p, part ? part->num_tiles : 0, s);
        if (st != MERBIT_OK) return st;
    }
    SpmvLaunch a;
    a.row_ptr = p->row_ptr;
    a.col = p->col;
    a.vals = p->vals;
    a.x = x;
    a.y = y;
    a.coords = part ? part->coords : nullptr;
    a.slots = p->carry.words;
    a.xch = p->carry.words + 2 * (size_t)p->carry.slots;
    a.nslots = p->carry.slots;
    a.state = part ? p->carry.state : p->state;  // row groups have no carries
    a.nrow = p->nrow;
    a.nnz = p->nnz;
    a.num_tiles = part ? part->num_tiles : 0;
    a.alpha = alpha;
    a.beta = beta;
    a.z = z;
    if (residual) {
        a.xres = x;
        a.partials = p->partials;
        a.residual = residual;
    }
    return spmv_launch(p->dtype, cfg, p->vec, a, s);
}

// Tuning cache: matrix signature -> config index.  The signature buckets
// (log2) the row count, the nonzero count, the density and the longest row,
// so that a configuration tuned on short, even rows (a stencil, where the
// row-group kernel wins) is never applied to a power-law matrix of the same
// size, whose long rows serialize that kernel.
struct Sig {
    int dtype, vec, nrow_bucket, nnz_bucket, density_bucket, maxrow_bucket;
    auto key() const {
        return std::tie(dtype, vec, nrow_bucket, nnz_bucket, density_bucket, maxrow_bucket);
    }
    bool operator<(const Sig& o) const { return key() < o.key(); }
    bool same_size(const Sig& o) const {
        return std::tie(dtype, vec, nrow_bucket, nnz_bucket, density_bucket) ==
               std::tie(o.dtype, o.vec, o.nrow_bucket, o.nnz_bucket, o.density_bucket);
    }
};
struct Tuned {
    int cfg;          // the configuration that won
    int max_row_len;  // longest row of the matrix it was tuned on
};
std::mutex g_tune_mu;
std::map<Sig, Tuned> g_tune;

int log2_bucket(double v) {
    int b = 0;
    while (v >= 2.0 && b < 62) {
        v *= 0.5;
        ++b;
    }
    return b;
}

Sig signature(const merbit_plan_s* p, int max_row_len) {
    Sig s;
    s.dtype = p->dtype;
    s.vec = p->vec;
    s.nrow_bucket = log2_bucket((double)p->nrow);
    s.nnz_bucket = log2_bucket((double)p->nnz);
    s.density_bucket = log2_bucket(4.0 * (double)p->nnz / (double)(p->nrow > 0 ? p->nrow : 1));
    s.maxrow_bucket = log2_bucket((double)(max_row_len > 0 ? max_row_len : 0) + 1.0);
    return s;
}

// Whether a cached choice may serve a plan whose longest row is
// max_row_len.  The row-group kernel gives each row to one lane group, so
// its time grows with the longest row: it is kept only for matrices whose
// longest row is at most twice the one it was tuned on.  Merge-path
// kernels balance any row lengths and are checked by their rows-per-tile
// cap instead.
bool cached_choice_fits(int dtype, const Tuned& t, int max_row_len) {
    if (spmv_config(dtype, t.cfg).kind != 3) return true;
    return (long long)max_row_len <= 2LL * std::max(t.max_row_len, 1);
}

// Batched k = 1 warp-tile kernel: the (variant, items per lane) the batch
// tuner chose for a matrix signature (same signature as the SpMV tuner's).
std::map<Sig, std::pair<int, int>> g_batch_ipt;

}  // namespace

int tune_cache_batch_ipt(const merbit_plan_s* p, int* variant) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    const Sig sg = signature(p, p->max_row_len);
    *variant = -1;
    auto it = g_batch_ipt.find(sg);
    if (it != g_batch_ipt.end()) {
        *variant = it->second.first;
        return it->second.second;
    }
    // a warp-tile SpMV configuration tuned for this signature suggests its
    // items per lane when the batch kernel has the same
    auto jt = g_tune.find(sg);
    if (jt != g_tune.end()) {
        const SpmvConfig c = spmv_config(p->dtype, jt->second.cfg);
        if (c.kind == 1)
            for (int i = 0; i < kNumBatchIpts; ++i)
                if (kBatchIpts[i] == c.ipt) return c.ipt;
    }
    return -1;
}

void tune_cache_store_batch_ipt(const merbit_plan_s* p, int variant, int ipt) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_batch_ipt[signature(p, p->max_row_len)] = {variant, ipt};
}

}  // namespace merbit

using namespace merbit;

extern "C" {

const char* merbit_status_string(int status) {
    switch (status) {
    case MERBIT_OK: return "MERBIT_OK";
    case MERBIT_ERR_INVALID: return "MERBIT_ERR_INVALID: invalid argument";
    case MERBIT_ERR_MATRIX: return "MERBIT_ERR_MATRIX: malformed CSR structure";
    case MERBIT_ERR_OVERFLOW: return "MERBIT_ERR_OVERFLOW: nrow+nnz exceeds the int32 range";
    case MERBIT_ERR_CUDA: return "MERBIT_ERR_CUDA: CUDA runtime error";
    case MERBIT_ERR_TIMEOUT: return "MERBIT_ERR_TIMEOUT: device-side carry wait ran out";
    case MERBIT_ERR_UNSUPPORTED: return "MERBIT_ERR_UNSUPPORTED: not implemented";
    default: return "MERBIT: unknown status";
    }
}

int merbit_last_cuda_error(void) { return g_last_cuda; }

const char* merbit_last_error_detail(void) { return g_detail.c_str(); }

int merbit_plan_create(merbit_plan* plan, int32_t nrow, int32_t ncol, int32_t nnz,
                       const int32_t* d_row_ptr, const int32_t* d_col_idx, const void* d_vals,
                       merbit_dtype dtype, uint32_t flags, void* stream) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "plan_create: plan is null");
    *plan = nullptr;
    if (nrow < 0 || ncol < 0 || nnz < 0) return fail(MERBIT_ERR_INVALID, "plan_create: negative size");
    if (dtype != MERBIT_F64 && dtype != MERBIT_F32 && dtype != MERBIT_BF16)
        return fail(MERBIT_ERR_INVALID, "plan_create: unknown dtype");
    if (!d_row_ptr) return fail(MERBIT_ERR_INVALID, "plan_create: row_ptr is null");
    if (nnz > 0 && (!d_col_idx || !d_vals))
        return fail(MERBIT_ERR_INVALID, "plan_create: col_idx/vals null with nnz > 0");
    if (nnz > 0 && ncol == 0) return fail(MERBIT_ERR_MATRIX, "plan_create: nnz > 0 with ncol == 0");
    if ((long long)nrow + nnz > (long long)INT_MAX - 64)
        return fail(MERBIT_ERR_OVERFLOW, "plan_create: nrow+nnz exceeds the int32 merge-path range");
    cudaStream_t s = (cudaStream_t)stream;
    auto* p = new merbit_plan_s();
    p->nrow = nrow;
    p->ncol = ncol;
    p->nnz = nnz;
    p->dtype = dtype;
    p->row_ptr = d_row_ptr;
    p->col = d_col_idx;
    p->vals = d_vals;
    p->vec = aligned16(d_col_idx) && aligned16(d_vals) && aligned16(d_row_ptr);
    cudaGetDevice(&p->device);
    // A provisional choice before the longest row is known: a cached
    // configuration of a matrix of the same size class (any longest-row
    // bucket; the exact signature decides after the read-back below).
    int provisional = -1;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        const Sig lo = signature(p, 0);
        for (auto it = g_tune.lower_bound(lo); it != g_tune.end() && it->first.same_size(lo); ++it)
            if (spmv_config(dtype, it->second.cfg).kind != 3) {
                provisional = it->second.cfg;
                break;
            }
    }
    // one allocation for the launch state and the build's readback words;
    // the whole build (validation, longest row, first partition, carry
    // slots) is queued on s and read back with one synchronization
    static_assert(sizeof(LaunchState) % alignof(PlanScratch) == 0, "scratch alignment");
    int st = dev_alloc(&p->state, sizeof(LaunchState) + sizeof(PlanScratch), s);
    if (st != MERBIT_OK) {
        delete p;
        return st;
    }
    p->scratch = reinterpret_cast<PlanScratch*>(p->state + 1);
    struct {
        LaunchState ls;
        PlanScratch sc;
    } init = {};
    static_assert(sizeof(init) == sizeof(LaunchState) + sizeof(PlanScratch), "state layout");
    init.ls.epoch = 1u;
    init.sc = PlanScratch{0, {INT_MAX, INT_MAX}, 0, 0, 0};
    cudaError_t e = cudaMemcpyAsync(p->state, &init, sizeof(init), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) {
        merbit_plan_destroy(p);
        return cuda_fail(e, "plan_create: init state");
    }
    const bool validate = !(flags & MERBIT_PLAN_SKIP_VALIDATE);
    st = validate_launch(d_row_ptr, d_col_idx, nrow, ncol, nnz, p->scratch, validate, s);
    // first candidate: the provisional cached configuration, else the
    // table's first entry the plan's alignment allows
    int first = -1;
    if (provisional >= 0 && spmv_config_allowed(spmv_config(dtype, provisional), p->vec))
        first = provisional;
    for (int i = 0, n = spmv_num_configs(dtype); first < 0 && i < n; ++i)
        if (spmv_config_allowed(spmv_config(dtype, i), p->vec)) first = i;
    const Partition* part = nullptr;
    if (st == MERBIT_OK && first >= 0 && spmv_config(dtype, first).kind != 3) {
        st = plan_partition(p, spmv_tile_items(spmv_config(dtype, first)), &part, s);
        if (st == MERBIT_OK) st = max_rows_async(*part, &p->scratch->max_rows, s);
        if (st == MERBIT_OK) st = grow_carry(p, part->num_tiles, s);
    }
    PlanScratch h = {};
    if (st == MERBIT_OK) {
        e = cudaMemcpyAsync(&h, p->scratch, sizeof(h), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) st = cuda_fail(e, "plan_create: readback");
    }
    if (st == MERBIT_OK && validate) st = validate_status(h);
    if (st == MERBIT_OK) {
        p->max_row_len = h.max_row_len;
        if (part) const_cast<Partition*>(part)->max_rows = h.max_rows;
        // the exact signature, longest row included
        int tuned = -1;
        {
            std::lock_guard<std::mutex> lk(g_tune_mu);
            auto it = g_tune.find(signature(p, p->max_row_len));
            if (it != g_tune.end() && cached_choice_fits(dtype, it->second, p->max_row_len))
                tuned = it->second.cfg;
        }
        bool ok = false;
        const int rule = tuned < 0 ? short_rows_choice(p) : -1;
        if (tuned >= 0) {
            st = plan_config_ok(p, tuned, &ok, s);  // reuses the partition built above
            if (st == MERBIT_OK && ok) p->cfg = tuned;
        } else if (rule >= 0) {
            p->cfg = rule;  // row groups take any matrix
            ok = true;
        } else {
            // no cached choice for this signature: the provisional one came
            // from another longest-row bucket, so it is not kept
            const bool from_cache = first == provisional && provisional >= 0;
            ok = !from_cache && first >= 0 &&
                 (!part || h.max_rows <= spmv_config_row_cap(spmv_config(dtype, first)));
            if (ok) p->cfg = first;
        }
        if (st == MERBIT_OK && !ok) st = plan_pick_default(p, s);  // reuses built partitions
    }
    if (st != MERBIT_OK) {
        merbit_plan_destroy(p);
        return st;
    }
    *plan = p;
    return MERBIT_OK;
}

int merbit_plan_destroy(merbit_plan plan) {
    if (!plan) return MERBIT_OK;
    // the plan's launches may still run on any stream: wait for the device,
    // as cudaFree does, then hand the blocks back to the pool
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != plan->device) cudaSetDevice(plan->device);
    cudaDeviceSynchronize();
    for (auto& q : plan->parts) dev_free(q.coords, nullptr);
    for (auto& kv : plan->spmm_slots) {
        dev_free(kv.second.words, nullptr);
        dev_free(kv.second.state, nullptr);
    }
    dev_free(plan->carry.words, nullptr);
    for (auto& c : plan->old_carries) dev_free(c.words, nullptr);
    dev_free(plan->state, nullptr);
    dev_free(plan->row_of, nullptr);
    dev_free(plan->partials, nullptr);
    for (void* q : plan->owned) dev_free(q, nullptr);
    if (cur != plan->device) cudaSetDevice(cur);
    delete plan;
    return MERBIT_OK;
}

int merbit_plan_get_info(merbit_plan plan, merbit_plan_info* info) {
    if (!plan || !info) return fail(MERBIT_ERR_INVALID, "plan_get_info: null pointer");
    const SpmvConfig c = spmv_config(plan->dtype, plan->cfg);
    info->nrow = plan->nrow;
    info->ncol = plan->ncol;
    info->nnz = plan->nnz;
    info->dtype = plan->dtype;
    info->block = c.block;
    info->items_per_thread = c.ipt;
    info->tile_items = spmv_tile_items(c);
    info->num_tiles = 0;
    int64_t slots = plan->carry.slots;
    for (auto& c : plan->old_carries) slots += c.slots;
    int64_t meta = sizeof(LaunchState) + slots * 4 * (int64_t)sizeof(unsigned long long);
    for (auto& q : plan->parts) {
        if (q.tile_items == info->tile_items) info->num_tiles = q.num_tiles;
        meta += (int64_t)(q.num_tiles + 1) * (int64_t)sizeof(int2);
    }
    info->vectorized = plan->vec ? 1 : 0;
    info->kind = c.kind;
    info->l1_carveout = c.carveout;
    info->gather_l2_only = c.cg;
    info->metadata_bytes = meta;
    info->max_row_len = plan->max_row_len;
    info->algorithmic_bytes = 4.0 * (plan->nrow + 1.0) +
                              (double)plan->nnz * (4.0 + (double)dtype_size(plan->dtype)) +
                              (double)xy_size(plan->dtype) * ((double)plan->ncol + plan->nrow);
    return MERBIT_OK;
}

int merbit_plan_set_values(merbit_plan plan, const void* d_vals) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "plan_set_values: plan is null");
    if (plan->nnz > 0 && !d_vals) return fail(MERBIT_ERR_INVALID, "plan_set_values: vals is null");
    plan->vals = d_vals;
    plan->vec = aligned16(plan->col) && aligned16(d_vals) && aligned16(plan->row_ptr);
    bool ok = false;
    int st = plan_config_ok(plan, plan->cfg, &ok, nullptr);
    if (st == MERBIT_OK && !ok) st = plan_pick_default(plan, nullptr);
    return st;
}

int merbit_spmv(merbit_plan plan, double alpha, const void* d_x, double beta, void* d_y,
                void* stream) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "spmv: plan is null");
    if (plan->nrow == 0) return MERBIT_OK;
    if (!d_y || (plan->ncol > 0 && !d_x)) return fail(MERBIT_ERR_INVALID, "spmv: x/y is null");
    return run_spmv(plan, plan->cfg, alpha, d_x, beta, d_y, (cudaStream_t)stream);
}

int merbit_pagerank_step(merbit_plan plan, double damp, const void* d_x, const void* d_teleport,
                         void* d_y, double* d_residual, void* stream) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "pagerank_step: plan is null");
    if (plan->nrow != plan->ncol) return fail(MERBIT_ERR_INVALID, "pagerank_step: plan is not square");
    if (plan->nrow == 0) {
        if (d_residual) MERBIT_CUDA(cudaMemsetAsync(d_residual, 0, sizeof(double), (cudaStream_t)stream));
        return MERBIT_OK;
    }
    if (!d_x || !d_y || !d_teleport) return fail(MERBIT_ERR_INVALID, "pagerank_step: null vector");
    if (d_x == d_y) return fail(MERBIT_ERR_INVALID, "pagerank_step: x and y must differ");
    if (!(damp >= 0.0 && damp <= 1.0)) return fail(MERBIT_ERR_INVALID, "pagerank_step: damp outside [0, 1]");
    // on the plan's device for this call; the caller's current device is restored
    int cur = 0;
    MERBIT_CUDA(cudaGetDevice(&cur));
    if (cur != plan->device) MERBIT_CUDA(cudaSetDevice(plan->device));
    const int st = run_spmv(plan, plan->cfg, damp, d_x, 1.0 - damp, d_y, (cudaStream_t)stream,
                            d_teleport, d_residual);
    if (cur != plan->device) cudaSetDevice(cur);
    return st;
}

int merbit_plan_tune(merbit_plan plan, const void* d_x, void* d_y, void* stream) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "plan_tune: plan is null");
    if (plan->nrow == 0) return MERBIT_OK;
    if (!d_y || (plan->ncol > 0 && !d_x)) return fail(MERBIT_ERR_INVALID, "plan_tune: x/y is null");
    cudaStream_t s = (cudaStream_t)stream;
    cudaEvent_t e0, e1;
    MERBIT_CUDA(cudaEventCreate(&e0));
    MERBIT_CUDA(cudaEventCreate(&e1));
    const int n = spmv_num_configs(plan->dtype);
    int best = plan->cfg;
    int st = MERBIT_OK;
    // ms of `reps` back-to-back launches of configuration c
    auto time_cfg = [&](int c, int reps, float* ms) -> int {
        int rc = MERBIT_OK;
        cudaEventRecord(e0, s);
        for (int r = 0; r < reps && rc == MERBIT_OK; ++r) rc = run_spmv(plan, c, 1.0, d_x, 0.0, d_y, s);
        cudaEventRecord(e1, s);
        cudaError_t ce = cudaEventSynchronize(e1);
        if (ce != cudaSuccess) return cuda_fail(ce, "plan_tune");
        if (rc != MERBIT_OK) return rc;
        cudaEventElapsedTime(ms, e0, e1);
        *ms /= (float)reps;
        return MERBIT_OK;
    };
    // 1. every usable configuration, 5 launches after 2 warm-up launches
    std::vector<std::pair<float, int>> timed;
    for (int c = 0; c < n && st == MERBIT_OK; ++c) {
        bool ok = false;
        st = plan_config_ok(plan, c, &ok, s);
        if (st != MERBIT_OK) break;
        if (!ok) continue;
        for (int w = 0; w < 2 && st == MERBIT_OK; ++w) st = run_spmv(plan, c, 1.0, d_x, 0.0, d_y, s);
        float ms = 0.f;
        if (st == MERBIT_OK) st = time_cfg(c, 5, &ms);
        if (st == MERBIT_OK) timed.push_back({ms, c});
    }
    // 2. the three fastest again, best of three rounds of 10 launches each
    //    (a single short round cannot separate entries within a few percent)
    if (st == MERBIT_OK && !timed.empty()) {
        std::stable_sort(timed.begin(), timed.end());
        const size_t top = std::min<size_t>(3, timed.size());
        float best_ms = 1e30f;
        best = timed[0].second;
        for (int round = 0; round < 3 && st == MERBIT_OK; ++round)
            for (size_t i = 0; i < top && st == MERBIT_OK; ++i) {
                float ms = 0.f;
                st = time_cfg(timed[i].second, 10, &ms);
                if (st == MERBIT_OK && ms < best_ms) {
                    best_ms = ms;
                    best = timed[i].second;
                }
            }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != MERBIT_OK) return st;
    plan->cfg = best;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[signature(plan, plan->max_row_len)] = Tuned{best, plan->max_row_len};
    return MERBIT_OK;
}

int merbit_num_configs(merbit_dtype dtype) {
    if (dtype != MERBIT_F64 && dtype != MERBIT_F32 && dtype != MERBIT_BF16) return 0;
    return spmv_num_configs(dtype);
}

int merbit_config_desc(merbit_dtype dtype, int32_t idx, int32_t* kind, int32_t* block,
                       int32_t* items_per_thread) {
    if (idx < 0 || idx >= merbit_num_configs(dtype) || !kind || !block || !items_per_thread)
        return fail(MERBIT_ERR_INVALID, "config_desc: bad index");
    const SpmvConfig c = spmv_config(dtype, idx);
    *kind = c.kind;
    *block = c.block;
    *items_per_thread = c.ipt;
    return MERBIT_OK;
}

int merbit_plan_set_config(merbit_plan plan, int32_t idx, void* stream) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "plan_set_config: plan is null");
    if (idx < 0 || idx >= spmv_num_configs(plan->dtype))
        return fail(MERBIT_ERR_INVALID, "plan_set_config: bad index");
    bool ok = false;
    int st = plan_config_ok(plan, idx, &ok, (cudaStream_t)stream);
    if (st != MERBIT_OK) return st;
    if (!ok)
        return fail(MERBIT_ERR_INVALID,
                    "plan_set_config: configuration cannot run this plan (needs 16-byte aligned "
                    "arrays, or the matrix ends too many rows in one tile)");
    plan->cfg = idx;
    return MERBIT_OK;
}

int merbit_plan_config_usable(merbit_plan plan, int32_t idx, int32_t* usable, void* stream) {
    if (!plan || !usable) return fail(MERBIT_ERR_INVALID, "plan_config_usable: null pointer");
    if (idx < 0 || idx >= spmv_num_configs(plan->dtype))
        return fail(MERBIT_ERR_INVALID, "plan_config_usable: bad index");
    bool ok = false;
    int st = plan_config_ok(plan, idx, &ok, (cudaStream_t)stream);
    *usable = ok ? 1 : 0;
    return st;
}

int merbit_plan_check(merbit_plan plan, void* stream) {
    if (!plan) return fail(MERBIT_ERR_INVALID, "plan_check: plan is null");
    cudaStream_t s = (cudaStream_t)stream;
    auto take = [&](LaunchState* ls) -> int {  // reads and clears one state's error
        int err = 0;
        MERBIT_CUDA(cudaMemcpyAsync(&err, &ls->error, sizeof(int), cudaMemcpyDeviceToHost, s));
        MERBIT_CUDA(cudaStreamSynchronize(s));
        if (err == 0) return MERBIT_OK;
        const int zero = 0;
        MERBIT_CUDA(cudaMemcpyAsync(&ls->error, &zero, sizeof(int), cudaMemcpyHostToDevice, s));
        MERBIT_CUDA(cudaStreamSynchronize(s));
        return fail(err, "a device-side carry wait ran out");
    };
    // the plan's launch state (also the first carry block's) and those of the
    // blocks that followed
    int st = take(plan->state);
    if (plan->carry.state && plan->carry.state != plan->state) {
        const int r = take(plan->carry.state);
        if (st == MERBIT_OK) st = r;
    }
    for (auto& c : plan->old_carries) {
        if (c.state == plan->state) continue;
        const int r = take(c.state);
        if (st == MERBIT_OK) st = r;
    }
    return st;
}

}  // extern "C"
