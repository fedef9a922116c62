// dataset.cu -- device-resident column store (the engine's view of the
// reference's ModelData / CompressedDataMatrix).
//
// HBM layout (one dataset, shared read-only by every engine and fit):
//   d_fmt[J]          int32 column formats
//   d_col_ptr[J+1]    int64 offsets into d_idx
//   d_idx[nnz]        int32 row ids, ascending within a column; one flat
//                     array so a column is one contiguous, coalesced range
//   d_val_ptr[J+1]    int64 offsets into d_val
//   d_val[...]        float64 SPARSE values (parallel to d_idx) and DENSE
//                     columns (K values each)
//   d_y, d_time[K]    float64
//   d_strat[K]        int32 stratum of each row, renumbered by runs
//   d_strat_ptr[S+1]  int32 first row of each stratum
// plus, on first computeXBeta with a nonzero coefficient, a row-major copy
// (d_row_ptr / d_row_col / d_row_val) whose per-row column order equals the
// reference's column-by-column axpy order.
#include "row_terms.cuh"

#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <atomic>

namespace cyc {

static thread_local std::string g_last_error;
void set_error(const std::string& msg) { g_last_error = msg; }

static std::atomic<long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

namespace {
std::mutex g_pinned_mutex;
std::vector<void*>& pinned_free() {
    static std::vector<void*>* v = new std::vector<void*>();   // lives to process exit
    return *v;
}
}  // namespace

void* pinned_block() {
    std::lock_guard<std::mutex> lk(g_pinned_mutex);
    auto& fl = pinned_free();
    if (fl.empty()) {
        char* chunk = nullptr;
        CYC_CHECK_CUDA(cudaMallocHost(reinterpret_cast<void**>(&chunk), 64 * 512));
        for (int i = 511; i >= 0; --i) fl.push_back(chunk + 64 * i);
    }
    void* p = fl.back();
    fl.pop_back();
    return p;
}

void release_pinned_block(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_pinned_mutex);
    pinned_free().push_back(p);
}

cudaStream_t& alloc_stream() {
    static thread_local cudaStream_t s = nullptr;
    return s;
}

// Every kernel of the library, by one of each source file.  CUDA loads a kernel at
// its first launch, and loading waits for the kernels that run: with persistent
// kernels of seconds, calls that meet an instance for the first time stood still
// behind other callers' fits (120 served requests, 32 hardware queues: 53 done in
// 60 s; 120 in 35 with all loaded before).  Loading takes 0.55 s a device, so only
// callers that share it pay.
static std::vector<const void*>& kernel_files() {
    static auto* v = new std::vector<const void*>();
    return *v;
}
KernelFile::KernelFile(const void* kernel) { kernel_files().push_back(kernel); }

static void load_kernels(int device) {
    static std::mutex m;
    static std::vector<int> done;
    std::lock_guard<std::mutex> lk(m);
    if (std::find(done.begin(), done.end(), device) != done.end()) return;
    done.push_back(device);
    CYC_CHECK_CUDA(cudaSetDevice(device));
    auto entry = [](const char* name) -> void* {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPointByVersion(name, &p, 12040, cudaEnableDefault, &found);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? p : nullptr;
    };
    const auto module_of = reinterpret_cast<decltype(&cuFuncGetModule)>(entry("cuFuncGetModule"));
    const auto count = reinterpret_cast<decltype(&cuModuleGetFunctionCount)>(entry("cuModuleGetFunctionCount"));
    const auto list = reinterpret_cast<decltype(&cuModuleEnumerateFunctions)>(entry("cuModuleEnumerateFunctions"));
    const auto load = reinterpret_cast<decltype(&cuFuncLoad)>(entry("cuFuncLoad"));
    if (!module_of || !count || !list || !load) return;      // an older driver: at their first launch
    for (const void* kernel : kernel_files()) {
        cudaFunction_t f;
        CUmodule module;
        unsigned n = 0;
        CYC_CHECK_CUDA(cudaGetFuncBySymbol(&f, kernel));
        if (module_of(&module, (CUfunction)f) != CUDA_SUCCESS || count(&n, module) != CUDA_SUCCESS) continue;
        std::vector<CUfunction> all(n);
        if (n == 0 || list(all.data(), n, module) != CUDA_SUCCESS) continue;
        for (CUfunction g : all) load(g);
    }
}

// freed memory stays in the device's default pool for the next allocation
// instead of going back to the driver at every synchronisation (a setting of
// this process's pool, not of the GPU)
void prepare_pool(int device) {
    static std::mutex m;
    static std::vector<int> done;
    std::lock_guard<std::mutex> lk(m);
    for (int d : done)
        if (d == device) return;
    cudaMemPool_t pool;
    CYC_CHECK_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
    unsigned long long keep = ~0ull;
    CYC_CHECK_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    done.push_back(device);
}

size_t Dataset::device_bytes() const {
    return d_fmt.bytes() + d_col_ptr.bytes() + d_val_ptr.bytes() + d_idx.bytes() + d_val.bytes() +
           d_y.bytes() + d_time.bytes() + d_strat.bytes() + d_strat_ptr.bytes() + d_row_ptr.bytes() +
           d_row_col.bytes() + d_row_val.bytes() + d_entry_strat.bytes();
}

// on the calling thread's allocation stream (the dataset's, during uploads)
template <class T>
static void upload(DevBuf<T>& buf, const T* src, size_t n) {
    buf.alloc(n);
    if (n) CYC_CHECK_CUDA(cudaMemcpyAsync(buf.get(), src, n * sizeof(T), cudaMemcpyHostToDevice, alloc_stream()));
}

// ---- the row-major copy ----------------------------------------------------------
//
// Each row lists its columns ascending (the order of zeroXBeta + axpyXBeta per
// j, CyclicCoordinateDescent.cpp:1452-1470).  The rows are counted with
// atomics and scanned; then a warp takes a range of rows and walks the columns
// in order, 32 at a time: the columns' entries in its rows (k_splits), laid end
// to end, are placed 32 a step, entries of one row in the order of their
// lanes.  Bound by a load latency a step: 1.3M entries (100k rows, 600 Zipf
// columns and 5 dense ones) 21 ms as a counting sort on the host, 0.2 here.  The
// splits of all columns over all warps may be large, so columns go in parts, and
// the rows' cursors wait in memory between them (fewer warps instead: 1M columns
// of 10 entries over 100k rows 321 ms; 170 on the host, 37 in parts).

namespace {

constexpr int kCsrRows = 512;          // rows of a warp: its cursors, in shared memory
constexpr int kCsrWarps = 8;

__global__ void k_csr_count(long long n, const int* __restrict__ idx, int* __restrict__ cnt) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        atomicAdd(cnt + idx[e], 1);
}

const KernelFile g_kernels((const void*)(&k_csr_count));

// row offsets: exclusive sums of cnt + `every` (the dense columns), by one block
__global__ void k_csr_scan(int K, int every, const int* __restrict__ cnt, long long* __restrict__ rp) {
    constexpr int kItems = 8;
    __shared__ long long s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long carry = 0;
    for (long long base = 0; base < K; base += (long long)blockDim.x * kItems) {
        const long long k0 = base + (long long)threadIdx.x * kItems;
        int c[kItems];
        long long sum = 0;
        #pragma unroll
        for (int q = 0; q < kItems; ++q) {
            c[q] = k0 + q < K ? cnt[k0 + q] + every : 0;
            sum += c[q];
        }
        long long in = sum;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, in, o);
            if (lane >= o) in += u;
        }
        if (lane == 31) s_w[warp] = in;
        __syncthreads();
        long long at = carry + in - sum;
        for (int q = 0; q < warp; ++q) at += s_w[q];
        #pragma unroll
        for (int q = 0; q < kItems; ++q) {
            if (k0 + q < K) rp[k0 + q] = at;
            at += c[q];
        }
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) carry += s_w[q];
        __syncthreads();
    }
    if (threadIdx.x == 0) rp[K] = carry;
}

// rows [part[w], part[w + 1]) by warp w; `split` as k_splits leaves it; the J
// columns are `col0` and the ones after it, `placed` the entries of each row so far
__global__ void __launch_bounds__(32 * kCsrWarps)
k_csr_fill(int J, int col0, int W, int* __restrict__ placed, const int* __restrict__ part, const int* __restrict__ split, const int* __restrict__ fmt,
           const long long* __restrict__ col_ptr, const long long* __restrict__ val_ptr, const int* __restrict__ idx,
           const double* __restrict__ val, const long long* __restrict__ rp, int* __restrict__ rc,
           double* __restrict__ rv) {
    __shared__ int s_cur[kCsrWarps][kCsrRows];
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = blockIdx.x * kCsrWarps + (threadIdx.x >> 5);
    if (w >= W) return;
    int* cur = s_cur[threadIdx.x >> 5];
    const int r0 = part[w], r1 = part[w + 1];
    for (int q = lane; q < r1 - r0; q += 32) cur[q] = placed[r0 + q];
    __syncwarp();
    for (int j0 = 0; j0 < J; j0 += 32) {
        const int j = j0 + lane;
        int f = CYC_INDICATOR, first = 0, n = 0;
        long long cp = 0, vp = 0;
        if (j < J) {
            f = fmt[j];
            first = split[(size_t)j * (W + 1) + w];
            n = split[(size_t)j * (W + 1) + w + 1] - first;
            cp = col_ptr[j];
            vp = val_ptr[j];
        }
        const bool dense = f == CYC_DENSE || f == CYC_INTERCEPT;
        // the entry's place in the column's ids and values; no values: 1
        const long long ci = dense ? -1 : cp + first;
        const long long vi = f == CYC_SPARSE || f == CYC_DENSE ? vp + first : -1;
        int in = n;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(full, in, o);
            if (lane >= o) in += u;
        }
        const int total = __shfl_sync(full, in, 31), before = in - n;
        for (int t0 = 0; t0 < total; t0 += 32) {
            const int t = t0 + lane;
            int src = 0;                       // the column of entry t: columns whose entries end at or before t
            #pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int end = __shfl_sync(full, in, src + o - 1);
                if (end <= t) src += o;
            }
            const int e = t - __shfl_sync(full, before, src);
            const int fs = __shfl_sync(full, first, src);
            const long long c = __shfl_sync(full, ci, src), v = __shfl_sync(full, vi, src);
            const bool on = t < total;
            const int k = !on ? -1 - lane : (c < 0 ? fs + e : __ldg(idx + c + e));
            const unsigned same = __match_any_sync(full, k);
            if (on) {
                const int rank = __popc(same & ((1u << lane) - 1u));
                const long long p = rp[k] + cur[k - r0] + rank;
                rc[p] = col0 + j0 + src;
                rv[p] = v < 0 ? 1.0 : __ldg(val + v + e);
            }
            __syncwarp();
            if (on && lane == __ffs(same) - 1) cur[k - r0] += __popc(same);
            __syncwarp();
        }
    }
    for (int q = lane; q < r1 - r0; q += 32) placed[r0 + q] = cur[q];
}

}  // namespace

void Dataset::ensure_csr() {
    std::lock_guard<std::mutex> lock(csr_mutex);
    if (have_csr) return;
    StreamScope scope(stream);
    int every = 0;
    for (int j = 0; j < J; ++j) every += fmt[j] == CYC_DENSE || fmt[j] == CYC_INTERCEPT;
    const size_t total = (size_t)nnz_idx + (size_t)every * K;
    DevBuf<int> cnt, d_part, d_split;
    cnt.alloc(std::max(1, K));
    CYC_CHECK_CUDA(cudaMemsetAsync(cnt.get(), 0, std::max(1, K) * sizeof(int), stream));
    d_row_ptr.alloc((size_t)K + 1);
    d_row_col.alloc(total);
    d_row_val.alloc(total);
    if (nnz_idx)
        launch(k_csr_count, grid_for(nnz_idx, 4), kThreads, 0, stream, nnz_idx, (const int*)d_idx.get(), cnt.get());
    launch(k_csr_scan, 1, 1024, 0, stream, K, every, (const int*)cnt.get(), d_row_ptr.get());
    CYC_CHECK_CUDA(cudaMemsetAsync(cnt.get(), 0, std::max(1, K) * sizeof(int), stream));
    // as many warps as fill the device, kCsrRows rows a warp (more rows than they
    // hold take turns), and 64 MB of splits (more columns go in parts)
    const int W = 148 * 16;
    const int cols = std::min(J, (1 << 24) / (W + 1));
    std::vector<int> part(W + 1);
    d_split.alloc((size_t)cols * (W + 1));
    for (long long k0 = 0; k0 < K && total > 0; k0 += (long long)W * kCsrRows) {
        const long long rows = std::min<long long>((long long)W * kCsrRows, K - k0);
        for (int w = 0; w <= W; ++w) part[w] = (int)(k0 + rows * w / W);
        upload(d_part, part.data(), part.size());
        for (int j = 0; j < J; j += cols) {
            const int n = std::min(cols, J - j);
            const int* fm = d_fmt.get() + j;
            const long long *cp = d_col_ptr.get() + j, *vp = d_val_ptr.get() + j;
            launch(k_splits, grid_for((long long)n * (W + 1), 1, 1 << 30), kThreads, 0, stream, n, W, fm, cp,
                   (const int*)d_idx.get(), (const int*)d_part.get(), d_split.get());
            launch(k_csr_fill, (W + kCsrWarps - 1) / kCsrWarps, 32 * kCsrWarps, 0, stream, n, j, W, cnt.get(),
                   (const int*)d_part.get(), (const int*)d_split.get(), fm, cp, vp, (const int*)d_idx.get(),
                   (const double*)d_val.get(), (const long long*)d_row_ptr.get(), d_row_col.get(), d_row_val.get());
        }
    }
    CYC_CHECK_CUDA(cudaStreamSynchronize(stream));   // usable from every stream
    have_csr = true;
}

__global__ void k_entry_strata(long long n, const int* __restrict__ idx, const int* __restrict__ strat,
                               int* __restrict__ out) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        out[e] = strat[idx[e]];
}

int Dataset::event_rows() {
    std::lock_guard<std::mutex> lock(csr_mutex);
    if (n_event_rows < 0) n_event_rows = (int)(K - std::count(y.begin(), y.end(), 0.0));
    return n_event_rows;
}

void Dataset::ensure_entry_strata() {
    std::lock_guard<std::mutex> lock(csr_mutex);
    if (have_entry_strata) return;
    StreamScope scope(stream);
    d_entry_strat.alloc(std::max<long long>(1, nnz_idx));
    if (nnz_idx)
        launch(k_entry_strata, grid_for(nnz_idx, 4), kThreads, 0, stream, nnz_idx, (const int*)d_idx.get(),
               (const int*)d_strat.get(), d_entry_strat.get());
    CYC_CHECK_CUDA(cudaStreamSynchronize(stream));   // usable from every stream
    have_entry_strata = true;
}

}  // namespace cyc

using namespace cyc;

extern "C" const char* cyc_last_error(void) { return g_last_error.c_str(); }
extern "C" int cyc_version(void) { return CYC_ABI_VERSION; }
extern "C" long long cyc_launch_count(void) { return g_launches.load(); }

extern "C" int cyc_dataset_create(const cyc_data_desc* d, int device, cyc_dataset** out) {
    return guarded([&] {
        NvtxRange range("cyc_dataset_create");
        CYC_REQUIRE(d && out, CYC_ERR_ARGUMENT, "null argument");
        *out = nullptr;
        CYC_REQUIRE(d->K > 0 && d->J > 0, CYC_ERR_ARGUMENT, "K and J must be positive");
        CYC_REQUIRE(d->model >= CYC_LR && d->model <= CYC_COX, CYC_ERR_ARGUMENT, "Invalid model type.");
        CYC_REQUIRE(d->y && d->col_format && d->col_ptr && d->val_ptr, CYC_ERR_ARGUMENT, "missing arrays");
        CYC_REQUIRE(d->model != CYC_COX || d->time, CYC_ERR_ARGUMENT, "cox needs survival times");
        // a NaN or an infinity among the outcomes, times or covariate values
        // leaves every fit undefined (the reference's fit on such data comes
        // back ILLCONDITIONED with NaN coefficients), so such data is refused
        // before any device work
        auto finite = [](const double* a, long long n) {
            for (long long i = 0; i < n; ++i)
                if (!std::isfinite(a[i])) return false;
            return true;
        };
        CYC_REQUIRE(finite(d->y, d->K), CYC_ERR_ARGUMENT, "non-finite outcome (y)");
        CYC_REQUIRE(!d->time || finite(d->time, d->K), CYC_ERR_ARGUMENT, "non-finite time");
        CYC_REQUIRE(d->val_ptr[d->J] >= 0, CYC_ERR_ARGUMENT, "offsets must not decrease");
        CYC_REQUIRE(!d->col_val || finite(d->col_val, d->val_ptr[d->J]), CYC_ERR_ARGUMENT,
                    "non-finite covariate value");
        int ndev = 0;
        CYC_CHECK_CUDA(cudaGetDeviceCount(&ndev));
        CYC_REQUIRE(device >= 0 && device < ndev, CYC_ERR_ARGUMENT, "no such CUDA device");
        CYC_CHECK_CUDA(cudaSetDevice(device));

        auto* h = new cyc_dataset();
        std::unique_ptr<cyc_dataset> guard(h);
        Dataset& s = h->ds;
        s.device = device;
        prepare_pool(device);
        CYC_CHECK_CUDA(cudaStreamCreateWithFlags(&s.own.s, cudaStreamNonBlocking));
        s.stream = s.own.s;
        StreamScope scope(s.stream);
        s.model = d->model;
        s.K = d->K;
        s.J = d->J;
        s.has_offset = d->has_offset != 0;
        s.has_intercept = d->has_intercept != 0;
        s.fmt.assign(d->col_format, d->col_format + d->J);
        s.col_ptr.assign(d->col_ptr, d->col_ptr + d->J + 1);
        s.val_ptr.assign(d->val_ptr, d->val_ptr + d->J + 1);
        s.nnz_idx = s.col_ptr[d->J];
        s.nnz_val = s.val_ptr[d->J];
        CYC_REQUIRE(s.col_ptr[0] == 0 && s.val_ptr[0] == 0, CYC_ERR_ARGUMENT, "offsets must start at 0");
        CYC_REQUIRE(s.nnz_idx == 0 || d->col_idx, CYC_ERR_ARGUMENT, "missing col_idx");
        CYC_REQUIRE(s.nnz_val == 0 || d->col_val, CYC_ERR_ARGUMENT, "missing col_val");
        for (int j = 0; j < d->J; ++j) {
            const int f = s.fmt[j];
            CYC_REQUIRE(f >= CYC_DENSE && f <= CYC_INTERCEPT, CYC_ERR_ARGUMENT, "bad column format");
            const long long ni = s.col_ptr[j + 1] - s.col_ptr[j];
            const long long nv = s.val_ptr[j + 1] - s.val_ptr[j];
            CYC_REQUIRE(ni >= 0 && nv >= 0, CYC_ERR_ARGUMENT, "offsets must not decrease");
            if (f == CYC_DENSE) CYC_REQUIRE(nv == d->K && ni == 0, CYC_ERR_ARGUMENT, "dense column needs K values");
            if (f == CYC_SPARSE) CYC_REQUIRE(nv == ni, CYC_ERR_ARGUMENT, "sparse column values/indices mismatch");
            if (f == CYC_INDICATOR) CYC_REQUIRE(nv == 0, CYC_ERR_ARGUMENT, "indicator column holds no values");
            if (f == CYC_INTERCEPT) CYC_REQUIRE(nv == 0 && ni == 0, CYC_ERR_ARGUMENT, "intercept column holds nothing");
            if (f == CYC_SPARSE || f == CYC_INDICATOR) {
                const int* r = d->col_idx + s.col_ptr[j];
                for (long long e = 0; e < ni; ++e) {
                    CYC_REQUIRE(r[e] >= 0 && r[e] < d->K, CYC_ERR_ARGUMENT, "row index out of range");
                    CYC_REQUIRE(e == 0 || r[e] > r[e - 1], CYC_ERR_ARGUMENT, "row ids must ascend within a column");
                }
            }
        }
        if (d->has_offset) CYC_REQUIRE(s.fmt[0] == CYC_DENSE, CYC_ERR_ARGUMENT, "offset column must be dense");
        s.y.assign(d->y, d->y + d->K);
        if (d->time) s.time.assign(d->time, d->time + d->K);
        s.h_idx.assign(d->col_idx ? d->col_idx : (const int*)nullptr,
                       d->col_idx ? d->col_idx + s.nnz_idx : (const int*)nullptr);

        // strata renumbered by runs (src/RcppModelData.cpp:878-900)
        s.strat.resize(d->K);
        if (d->pid) {
            int cur = 0, last = d->pid[0];
            for (int k = 0; k < d->K; ++k) {
                if (d->pid[k] != last) { ++cur; last = d->pid[k]; }
                s.strat[k] = cur;
            }
            s.S = cur + 1;
        } else {
            for (int k = 0; k < d->K; ++k) s.strat[k] = k;
            s.S = d->K;
        }
        s.strat_ptr.assign(s.S + 1, 0);
        for (int k = 0; k < d->K; ++k) s.strat_ptr[s.strat[k] + 1]++;
        for (int i = 0; i < s.S; ++i) s.strat_ptr[i + 1] += s.strat_ptr[i];

        upload(s.d_fmt, s.fmt.data(), s.fmt.size());
        upload(s.d_col_ptr, s.col_ptr.data(), s.col_ptr.size());
        upload(s.d_val_ptr, s.val_ptr.data(), s.val_ptr.size());
        upload(s.d_idx, d->col_idx, (size_t)s.nnz_idx);
        upload(s.d_val, d->col_val, (size_t)s.nnz_val);
        upload(s.d_y, d->y, (size_t)d->K);
        if (d->time) upload(s.d_time, d->time, (size_t)d->K);
        upload(s.d_strat, s.strat.data(), s.strat.size());
        upload(s.d_strat_ptr, s.strat_ptr.data(), s.strat_ptr.size());
        CYC_CHECK_CUDA(cudaStreamSynchronize(s.stream));   // usable from every stream
        *out = guard.release();
    });
}

extern "C" int cyc_dataset_destroy(cyc_dataset* ds) {
    return guarded([&] {
        if (!ds) return;
        cudaSetDevice(ds->ds.device);
        delete ds;
    });
}

extern "C" int cyc_dataset_info(const cyc_dataset* ds, int* K, int* J, long long* nnz, size_t* bytes) {
    return guarded([&] {
        CYC_REQUIRE(ds, CYC_ERR_ARGUMENT, "null dataset");
        if (K) *K = ds->ds.K;
        if (J) *J = ds->ds.J;
        if (nnz) *nnz = ds->ds.nnz_idx;
        if (bytes) *bytes = ds->ds.device_bytes();
    });
}

extern "C" int cyc_dataset_set_sharing(cyc_dataset* ds, int calls) {
    return guarded([&] {
        CYC_REQUIRE(ds, CYC_ERR_ARGUMENT, "null dataset");
        CYC_REQUIRE(calls >= 1, CYC_ERR_ARGUMENT, "at least one call uses the device");
        if (calls > 1) load_kernels(ds->ds.device);
        ds->ds.share = calls;
    });
}
