// gt_table.cu — result tables of the C ABI: row counts, single columns and
// gt_table_export, which widens several columns at once to the dtypes of the
// reference's DataFrame (gpu_tracking_macros/src/lib.rs:138-147): on the device
// into pinned destinations, else on host threads through per-device pools of
// pinned staging lanes.
#include <memory>
#include <thread>

#include "gt_runtime.cuh"

using namespace gt;
using namespace gt::rt;

extern "C" {

int64_t gt_table_nrows(const gt_table* t) { return t ? t->n : 0; }

int32_t gt_table_has_column(const gt_table* t, int32_t column) {
    if (!t || column < 0 || column >= GT_NUM_COLUMNS) return 0;
    return t->has[column] ? 1 : 0;
}

gt_status gt_table_column_f32(const gt_table* t, int32_t column, float* dst) {
    if (!t || !dst || column < 0 || column >= GT_NUM_COLUMNS) return GT_ERR_INVALID_ARGUMENT;
    if (!t->has[column]) return GT_ERR_INVALID_ARGUMENT;
    if (t->n == 0) return GT_OK;
    cudaSetDevice(t->device);
    if (column == GT_COL_FRAME || column == GT_COL_PARTICLE || column == GT_COL_DURATION) {
        std::vector<int64_t> v(t->n);
        const TBuf& b = column == GT_COL_FRAME ? t->frame : (column == GT_COL_PARTICLE ? t->particle : t->duration);
        if (cudaMemcpy(v.data(), b.p, t->n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return cuda_failed();
        for (int64_t i = 0; i < t->n; i++) dst[i] = (float)v[i];
        return GT_OK;
    }
    if (cudaMemcpy(dst, t->col[column].p, t->n * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return cuda_failed();
    return GT_OK;
}

gt_status gt_table_column_i64(const gt_table* t, int32_t column, int64_t* dst) {
    if (!t || !dst) return GT_ERR_INVALID_ARGUMENT;
    if (column != GT_COL_FRAME && column != GT_COL_PARTICLE && column != GT_COL_DURATION)
        return GT_ERR_INVALID_ARGUMENT;
    if (!t->has[column]) return GT_ERR_INVALID_ARGUMENT;
    if (t->n == 0) return GT_OK;
    cudaSetDevice(t->device);
    const TBuf& b = column == GT_COL_FRAME ? t->frame : (column == GT_COL_PARTICLE ? t->particle : t->duration);
    if (cudaMemcpy(dst, b.p, t->n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return cuda_failed();
    return GT_OK;
}

namespace {

// Table export: each lane (one host thread) owns two pinned slots and a
// stream; it copies its share of the rows chunk by chunk into one slot while
// it widens the previous chunk from the other into the destination.
constexpr int kExportLanes = 8;
constexpr size_t kExportSlot = (size_t)1 << 20;
constexpr int kExportMaxDevices = 64;

struct ExportLane {
    char* slot[2] = {nullptr, nullptr};
    cudaStream_t st = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
};

struct ExportPool {
    std::mutex mu;
    bool ready = false;
    ExportLane lane[kExportLanes];
};

// One pool per device for the life of the process (never destroyed: no CUDA
// call runs from a static destructor after the runtime has shut down).
ExportPool* export_pool(int device) {
    static ExportPool* pools = new ExportPool[kExportMaxDevices];
    return device >= 0 && device < kExportMaxDevices ? &pools[device] : nullptr;
}

// All or nothing: on a failure everything created so far is released and the
// next call tries again.
cudaError_t export_pool_init(ExportPool& p) {
    if (p.ready) return cudaSuccess;
    char* block = nullptr;
    cudaError_t e = cudaHostAlloc((void**)&block, 2 * kExportLanes * kExportSlot, cudaHostAllocDefault);
    if (e != cudaSuccess) return e;
    for (int l = 0; l < kExportLanes && e == cudaSuccess; l++) {
        ExportLane& L = p.lane[l];
        L.slot[0] = block + (2 * l) * kExportSlot;
        L.slot[1] = block + (2 * l + 1) * kExportSlot;
        e = cudaStreamCreateWithFlags(&L.st, cudaStreamNonBlocking);
        for (int s = 0; s < 2 && e == cudaSuccess; s++) e = cudaEventCreateWithFlags(&L.ev[s], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
        for (ExportLane& L : p.lane) {
            for (cudaEvent_t& ev : L.ev)
                if (ev) cudaEventDestroy(ev), ev = nullptr;
            if (L.st) cudaStreamDestroy(L.st), L.st = nullptr;
            L.slot[0] = L.slot[1] = nullptr;
        }
        cudaFreeHost(block);
        return e;
    }
    p.ready = true;
    return cudaSuccess;
}

struct ExportItem {
    const char* src;   // device rows
    char* dst;         // host rows
    int64_t rows;
    bool widen;        // float32 -> double; otherwise int64 copied as is
};

cudaError_t export_lane(int device, ExportLane& L, const std::vector<ExportItem>& items) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    auto issue = [&](size_t i) {
        const ExportItem& it = items[i];
        const size_t bytes = (size_t)it.rows * (it.widen ? 4 : 8);
        cudaError_t r = cudaMemcpyAsync(L.slot[i & 1], it.src, bytes, cudaMemcpyDeviceToHost, L.st);
        return r != cudaSuccess ? r : cudaEventRecord(L.ev[i & 1], L.st);
    };
    if (items.empty()) return cudaSuccess;
    if ((e = issue(0)) != cudaSuccess) return e;
    for (size_t i = 0; i < items.size(); i++) {
        // slot (i + 1) & 1 held item i - 1, already widened by this thread
        if (i + 1 < items.size() && (e = issue(i + 1)) != cudaSuccess) break;
        if ((e = cudaEventSynchronize(L.ev[i & 1])) != cudaSuccess) break;
        const ExportItem& it = items[i];
        if (it.widen) {
            const float* s = (const float*)L.slot[i & 1];
            double* d = (double*)it.dst;
            for (int64_t j = 0; j < it.rows; j++) d[j] = (double)s[j];
        } else {
            memcpy(it.dst, L.slot[i & 1], (size_t)it.rows * 8);
        }
    }
    // nothing may still land in the slots once the pool is handed on
    cudaError_t e2 = cudaStreamSynchronize(L.st);
    return e != cudaSuccess ? e : e2;
}

}  // namespace

namespace {

// Columns widened on the device into pinned host columns of 8-byte values: a
// float column as doubles, an integer column as it is.  Blocks of threads
// stride over the rows of column blockIdx.y and store across PCIe: no staging
// on the device or the host.
struct PinnedColumns {
    const void* src[GT_NUM_COLUMNS];
    unsigned long long* dst[GT_NUM_COLUMNS];
    uint8_t widen[GT_NUM_COLUMNS];
};
__global__ void widen_columns_kernel(const PinnedColumns c, int64_t n) {
    const int k = blockIdx.y;
    unsigned long long* const o = c.dst[k];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (!c.widen[k]) {
            o[i] = ((const unsigned long long*)c.src[k])[i];
            continue;
        }
        const unsigned u = ((const unsigned*)c.src[k])[i];
        // a NaN keeps its sign and payload, as the host's conversion does
        o[i] = (u & 0x7FFFFFFFu) > 0x7F800000u
                   ? ((unsigned long long)(u >> 31) << 63) | 0x7FF8000000000000ull |
                         ((unsigned long long)(u & 0x7FFFFFu) << 29)
                   : (unsigned long long)__double_as_longlong((double)__uint_as_float(u));
    }
}

// Where the device stores to host memory `p` of `bytes` bytes, 8-byte aligned
// and inside one pinned allocation; nullptr for other memory.
unsigned long long* pinned_address(void* p, size_t bytes) {
    cudaPointerAttributes at, end;
    if ((uintptr_t)p % 8 != 0 || cudaPointerGetAttributes(&at, p) != cudaSuccess ||
        cudaPointerGetAttributes(&end, (char*)p + bytes - 1) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    const bool one = at.type == cudaMemoryTypeHost && end.type == cudaMemoryTypeHost && at.devicePointer &&
                     (char*)end.devicePointer == (char*)at.devicePointer + bytes - 1;
    return one ? (unsigned long long*)at.devicePointer : nullptr;
}

const TBuf& table_column(const gt_table* t, int32_t c) {
    return c == GT_COL_FRAME ? t->frame
                             : (c == GT_COL_PARTICLE ? t->particle : (c == GT_COL_DURATION ? t->duration : t->col[c]));
}

bool integer_column(int32_t c) { return c == GT_COL_FRAME || c == GT_COL_PARTICLE || c == GT_COL_DURATION; }

// Columns of the table widened into the pinned columns c.dst (on a stream of
// the caller's: the call that made the table has finished its work on it).
gt_status widen_columns(const gt_table* t, const int32_t* columns, int32_t ncolumns, PinnedColumns& c,
                        cudaStream_t st) {
    for (int32_t k = 0; k < ncolumns; k++) {
        c.src[k] = table_column(t, columns[k]).p;
        c.widen[k] = integer_column(columns[k]) ? 0 : 1;
    }
    const dim3 grid((unsigned)std::min<int64_t>((t->n + 255) / 256, 1024), ncolumns);
    widen_columns_kernel<<<grid, 256, 0, st>>>(c, t->n);
    const cudaError_t e = cudaGetLastError(), e2 = cudaStreamSynchronize(st);
    return e == cudaSuccess && e2 == cudaSuccess ? GT_OK : cuda_failed();
}

// The export into pinned columns; false where one of them is not.
bool export_to_pinned(const gt_table* t, const int32_t* columns, int32_t ncolumns, void* const* dst, gt_status* st) {
    PinnedColumns c;
    for (int32_t k = 0; k < ncolumns; k++) {
        c.dst[k] = pinned_address(dst[k], (size_t)t->n * 8);
        if (!c.dst[k]) return false;
    }
    *st = widen_columns(t, columns, ncolumns, c, cudaStreamPerThread);
    return true;
}

gt_status table_export_impl(const gt_table* t, const int32_t* columns, int32_t ncolumns, void* const* dst) {
    if (!t || ncolumns < 0 || (ncolumns > 0 && (!columns || !dst))) return GT_ERR_INVALID_ARGUMENT;
    for (int32_t k = 0; k < ncolumns; k++) {
        const int32_t c = columns[k];
        if (c < 0 || c >= GT_NUM_COLUMNS || !t->has[c] || !dst[k]) return GT_ERR_INVALID_ARGUMENT;
    }
    const int64_t N = t->n;
    if (N == 0 || ncolumns == 0) return GT_OK;
    if (cudaSetDevice(t->device) != cudaSuccess) return cuda_failed();
    gt_status st = GT_OK;
    if (ncolumns <= GT_NUM_COLUMNS && export_to_pinned(t, columns, ncolumns, dst, &st)) return st;
    ExportPool* pool = export_pool(t->device);
    if (!pool) return GT_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lock(pool->mu);
    if (export_pool_init(*pool) != cudaSuccess) return cuda_failed();
    const size_t bytes = (size_t)N * 8;
    if (ncolumns <= GT_NUM_COLUMNS && bytes * ncolumns <= kExportSlot) {
        // a result of one slot: widened on the device into the slot, one copy a
        // column from there (2000 rows of 11 columns: 31 us; a copy and an
        // event a column: 74)
        ExportLane& L = pool->lane[0];
        PinnedColumns c;
        for (int32_t k = 0; k < ncolumns; k++) c.dst[k] = (unsigned long long*)(L.slot[0] + bytes * k);
        if ((st = widen_columns(t, columns, ncolumns, c, L.st)) != GT_OK) return st;
        for (int32_t k = 0; k < ncolumns; k++) memcpy(dst[k], L.slot[0] + bytes * k, bytes);
        return GT_OK;
    }
    // lanes: one per 256k rows, at most kExportLanes and half the host threads
    const int hw = std::max(1, (int)std::thread::hardware_concurrency() / 2);
    const int lanes = (int)std::max<int64_t>(1, std::min<int64_t>({kExportLanes, hw, (N + (1 << 18) - 1) >> 18}));
    std::vector<std::vector<ExportItem>> work(lanes);
    for (int l = 0; l < lanes; l++) {
        const int64_t r0 = N * l / lanes, r1 = N * (l + 1) / lanes;
        for (int32_t k = 0; k < ncolumns; k++) {
            const int32_t c = columns[k];
            const bool integer = integer_column(c);
            const TBuf& b = table_column(t, c);
            const int64_t chunk = (int64_t)(kExportSlot / (integer ? 8 : 4));
            for (int64_t r = r0; r < r1; r += chunk) {
                ExportItem it;
                it.rows = std::min(chunk, r1 - r);
                it.src = (const char*)b.p + (size_t)r * (integer ? 8 : 4);
                it.dst = (char*)dst[k] + (size_t)r * 8;
                it.widen = !integer;
                work[l].push_back(it);
            }
        }
    }
    std::vector<cudaError_t> err(lanes, cudaSuccess);
    std::vector<std::thread> th;
    // lanes whose thread cannot be started run on the calling thread
    for (int l = 1; l < lanes; l++) {
        try {
            th.emplace_back([&, l] { err[l] = export_lane(t->device, pool->lane[l], work[l]); });
        } catch (...) {
            err[l] = export_lane(t->device, pool->lane[l], work[l]);
        }
    }
    err[0] = export_lane(t->device, pool->lane[0], work[0]);
    for (auto& x : th) x.join();
    for (cudaError_t e : err)
        if (e != cudaSuccess) return cuda_failed();
    return GT_OK;
}

}  // namespace

gt_status gt_table_export_pinned(const gt_table* t, const int32_t* columns, int32_t ncolumns, void* block) {
    if (!t || ncolumns < 0 || ncolumns > GT_NUM_COLUMNS || (ncolumns > 0 && (!columns || !block)))
        return GT_ERR_INVALID_ARGUMENT;
    void* dst[GT_NUM_COLUMNS];
    for (int32_t k = 0; k < ncolumns; k++) dst[k] = (char*)block + (size_t)k * (size_t)t->n * 8;
    return gt_table_export(t, columns, ncolumns, dst);
}

void* gt_host_alloc(size_t bytes) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes ? bytes : 1, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void gt_host_free(void* p) {
    if (p && cudaFreeHost(p) != cudaSuccess) cudaGetLastError();
}

gt_status gt_table_export(const gt_table* t, const int32_t* columns, int32_t ncolumns, void* const* dst) {
    try {
        return table_export_impl(t, columns, ncolumns, dst);
    } catch (...) {
        return GT_ERR_INTERNAL;   // no C++ exception crosses the C ABI
    }
}

void gt_table_free(gt_table* t) {
    if (!t) return;
    cudaSetDevice(t->device);
    delete t;
}

}  // extern "C"

namespace gt {
namespace rt {

// Uploads of at least this size from pageable memory use the lanes.  The
// driver's own staging moves 116 MB in 10-13 ms; eight threads that fill 1 MB
// pinned slots move it in 3-4 ms (a pinned source: 2.1 ms).  Below a few MB
// the threads cost what they save.
constexpr size_t kUploadLanesMin = (size_t)4 << 20;

bool upload_blocks(const void* src, size_t bytes) {
    if (bytes < kUploadLanesMin) return false;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, src) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

static cudaError_t upload_lane(int device, ExportLane& L, char* dst, const char* src, size_t bytes, int lane, int lanes) {
    cudaError_t e = cudaSetDevice(device);
    int k = 0;
    for (size_t o = (size_t)lane * kExportSlot; e == cudaSuccess && o < bytes; o += (size_t)lanes * kExportSlot, k++) {
        const size_t n = std::min(kExportSlot, bytes - o);
        if (k >= 2 && (e = cudaEventSynchronize(L.ev[k & 1])) != cudaSuccess) break;   // the slot's last copy
        memcpy(L.slot[k & 1], src + o, n);
        e = cudaMemcpyAsync(dst + o, L.slot[k & 1], n, cudaMemcpyHostToDevice, L.st);
        if (e == cudaSuccess) e = cudaEventRecord(L.ev[k & 1], L.st);
    }
    // nothing may still leave the slots once the pool is handed on
    const cudaError_t e2 = cudaStreamSynchronize(L.st);
    return e != cudaSuccess ? e : e2;
}

cudaError_t upload_host(int device, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    ExportPool* const pool = upload_blocks(src, bytes) ? export_pool(device) : nullptr;
    if (!pool) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    // what `st` still has to do before dst may be written
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(pool->mu);
    if ((e = export_pool_init(*pool)) != cudaSuccess) return e;
    const int hw = std::max(1, (int)std::thread::hardware_concurrency() / 2);
    const int lanes = (int)std::max<int64_t>(1, std::min<int64_t>({kExportLanes, hw, (int64_t)(bytes / (2 * kExportSlot))}));
    cudaError_t err[kExportLanes];
    std::thread th[kExportLanes];
    for (int l = 1; l < lanes; l++) {
        err[l] = cudaSuccess;
        // lanes whose thread cannot be started run on the calling thread
        try {
            th[l] = std::thread([=, &err] { err[l] = upload_lane(device, pool->lane[l], (char*)dst, (const char*)src, bytes, l, lanes); });
        } catch (...) {
            err[l] = upload_lane(device, pool->lane[l], (char*)dst, (const char*)src, bytes, l, lanes);
        }
    }
    err[0] = upload_lane(device, pool->lane[0], (char*)dst, (const char*)src, bytes, 0, lanes);
    for (int l = 1; l < lanes; l++)
        if (th[l].joinable()) th[l].join();
    for (int l = 0; l < lanes; l++)
        if (err[l] != cudaSuccess) return err[l];
    return cudaSuccess;
}

}  // namespace rt
}  // namespace gt
