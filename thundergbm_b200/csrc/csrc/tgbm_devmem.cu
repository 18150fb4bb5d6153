// Device memory of the library's buffers.
//
// A training call allocates and frees a few dozen buffers of up to several GB.  With cudaMalloc / cudaFree that costs
// 10-30 ms per call on one GPU and several times that when the host threads of an n_device = N call contend for the
// driver (cudaFree also unmaps the memory from every peer NCCL opened).  Released blocks are therefore kept, per
// device, and handed out again to the next request of (nearly) the same size: a call that follows another of the same
// shape allocates nothing.  The blocks are plain cudaMalloc memory, so whatever holds for cudaMalloc'ed buffers (peer
// access between the GPUs of one process, which NCCL relies on) holds for them.  A stream-ordered memory pool
// (cudaMallocFromPoolAsync) opened to the peer GPUs was measured too: with it the set-up of a call on 4 GPUs took
// 400 ms instead of 150 ms, every growth of such a pool being mapped on every peer.
//
// The interface keeps the meaning of cudaMalloc / cudaFree: dev_free waits for the device before the block goes back
// to the cache, so a block is never handed out again while work that was queued before its release still runs.
//
// What the cache holds between calls is bounded: at the end of every entry point of the C ABI (dev_trim) it is cut
// back to TGBM_POOL_KEEP_MB megabytes per device (default 16384; 0 = keep nothing), largest blocks first.
// TGBM_NO_POOL=1 selects plain cudaMalloc / cudaFree.
#include <cuda_runtime.h>
#include <pthread.h>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstdint>
#include <cstring>
#include <functional>
#include <iterator>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "tgbm_common.h"
#include "tgbm_device.cuh"
#include "tgbm_workers.h"

namespace tgbm {
namespace {

constexpr int MAX_DEVICES = 64;
constexpr size_t GRANULE = 512;   // request sizes are rounded up to this

struct DeviceCache {
    std::mutex mutex;
    std::multimap<size_t, void *> free_blocks;       // size -> block
    std::unordered_map<void *, size_t> live;         // blocks handed out -> size
    size_t cached_bytes = 0;
    bool dirty = false;                               // something was released since the last trim
};

// never destroyed: a buffer may be released while the process exits (a binding's finaliser, a static object of the
// host program), after the static destructors of this file would have run
DeviceCache *const g_cache = new DeviceCache[MAX_DEVICES];

bool cache_enabled() {
    static const bool on = getenv("TGBM_NO_POOL") == nullptr;
    return on;
}

size_t keep_bytes() {
    static const size_t keep = [] {
        const char *e = getenv("TGBM_POOL_KEEP_MB");
        const double mb = e ? atof(e) : 16384.0;
        return mb > 0 ? (size_t)(mb * 1048576.0) : (size_t)0;
    }();
    return keep;
}

// a cached block may serve a request when it wastes at most an eighth of it (or 64 KB)
bool fits(size_t block, size_t want) { return block >= want && block - want <= std::max<size_t>(want / 8, 65536); }

// gives cached blocks of device `dev` (the current device) back to the driver until at most `keep` bytes remain
void release_down_to(DeviceCache &c, size_t keep) {
    std::vector<void *> victims;
    {
        std::lock_guard<std::mutex> lock(c.mutex);
        while (c.cached_bytes > keep && !c.free_blocks.empty()) {
            auto it = std::prev(c.free_blocks.end());
            c.cached_bytes -= it->first;
            victims.push_back(it->second);
            c.free_blocks.erase(it);
        }
    }
    for (void *p : victims) cudaFree(p);
}

[[noreturn]] void fail(cudaError_t e, size_t bytes) {
    cudaGetLastError();
    throw Error(std::string("CUDA error: ") + cudaGetErrorString(e) + " allocating " + std::to_string(bytes) + " bytes of device memory");
}

}  // namespace

void *dev_alloc(size_t bytes) {
    if (bytes == 0) return nullptr;
    void *p = nullptr;
    int dev = 0;
    if (!cache_enabled() || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) {
        const cudaError_t e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) fail(e, bytes);
        return p;
    }
    DeviceCache &c = g_cache[dev];
    const size_t want = (bytes + GRANULE - 1) / GRANULE * GRANULE;
    {
        std::lock_guard<std::mutex> lock(c.mutex);
        auto it = c.free_blocks.lower_bound(want);
        if (it != c.free_blocks.end() && fits(it->first, want)) {
            p = it->second;
            c.live[p] = it->first;
            c.cached_bytes -= it->first;
            c.free_blocks.erase(it);
            return p;
        }
    }
    cudaError_t e = cudaMalloc(&p, want);
    if (e == cudaErrorMemoryAllocation) {   // the cache may hold what is missing
        cudaGetLastError();
        release_down_to(c, 0);
        e = cudaMalloc(&p, want);
    }
    if (e != cudaSuccess) fail(e, bytes);
    std::lock_guard<std::mutex> lock(c.mutex);
    c.live[p] = want;
    return p;
}

void dev_free(void *p) noexcept {
    if (!p) return;
    int owner = -1, cur = 0;
    cudaPointerAttributes attr = {};
    if (cudaPointerGetAttributes(&attr, p) == cudaSuccess) owner = attr.device;
    else cudaGetLastError();
    cudaGetDevice(&cur);
    if (!cache_enabled() || owner < 0 || owner >= MAX_DEVICES) { cudaFree(p); return; }
    DeviceCache &c = g_cache[owner];
    size_t size = 0;
    {
        std::lock_guard<std::mutex> lock(c.mutex);
        auto it = c.live.find(p);
        if (it != c.live.end()) { size = it->second; c.live.erase(it); }
    }
    if (size == 0) { cudaFree(p); return; }              // not one of ours
    if (owner != cur) cudaSetDevice(owner);               // a buffer may be released by another thread than the one that made it
    cudaDeviceSynchronize();                              // cudaFree's promise: nothing queued before the release still uses the block
    if (owner != cur) cudaSetDevice(cur);
    std::lock_guard<std::mutex> lock(c.mutex);
    c.free_blocks.emplace(size, p);
    c.cached_bytes += size;
    c.dirty = true;
}

static void trim_all(size_t keep, bool only_dirty) noexcept {
    if (!cache_enabled()) return;
    int cur = -1;
    for (int dev = 0; dev < MAX_DEVICES; ++dev) {
        DeviceCache &c = g_cache[dev];
        {
            std::lock_guard<std::mutex> lock(c.mutex);
            if ((only_dirty && !c.dirty) || c.cached_bytes <= keep) { c.dirty = false; continue; }
            c.dirty = false;
        }
        if (cur < 0 && cudaGetDevice(&cur) != cudaSuccess) { cudaGetLastError(); return; }
        cudaSetDevice(dev);
        release_down_to(c, keep);
    }
    if (cur >= 0) cudaSetDevice(cur);
}

// ---- copies between the device and pageable host memory ------------------------------------------------------------
// cudaMemcpyAsync from pageable memory (what a NumPy caller hands over) is staged by the driver through one small
// pinned buffer: 10.8 GB/s measured for the 2.4 GB of a Higgs-sized CSR, a fifth of what the link carries from pinned
// memory (page-locking the caller's arrays in place with cudaHostRegister runs at 11 GB/s too).  A few worker threads do
// the staging instead: they copy pieces into page-locked slots (two per thread, kept for the next call) and send each
// slot on with cudaMemcpyAsync on a stream of their own.  Page-locked or registered host memory, and copies of less than
// STAGE_MIN bytes (which the driver finishes before the workers have woken up), go to cudaMemcpyAsync directly.
//
// The slots are written with stores that go round the cache: nothing on the host reads them again, and an ordinary store
// first fetches the line that it overwrites (15 threads, 1.2 GB: 51 ms instead of 52.5; 8 threads 58 instead of 60).
//
// The workers outlive a call: starting eight threads with a stream and two events each cost 0.6-1 ms per upload.  At
// most WORKERS of them exist; several calling threads share them, a call that finds all of them busy waits.
namespace {

constexpr size_t STAGE_BYTES = 8u << 20;       // size of a slot and largest piece
constexpr size_t STAGE_PIECE_MIN = 256u << 10; // smallest piece
constexpr size_t STAGE_MIN = 1u << 20;
constexpr int WORKERS = 15;
constexpr int STAGE_KEEP = 2 * WORKERS;        // slots that stay allocated between calls (240 MB)

std::mutex &g_stage_mutex = *new std::mutex;
std::vector<void *> &g_stage_free = *new std::vector<void *>;

void *stage_acquire() {
    {
        std::lock_guard<std::mutex> lock(g_stage_mutex);
        if (!g_stage_free.empty()) { void *p = g_stage_free.back(); g_stage_free.pop_back(); return p; }
    }
    void *p = nullptr;
    if (cudaHostAlloc(&p, STAGE_BYTES, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return p;
}

void stage_release(void *p) {
    if (!p) return;
    {
        std::lock_guard<std::mutex> lock(g_stage_mutex);
        if ((int)g_stage_free.size() < STAGE_KEEP) { g_stage_free.push_back(p); return; }
    }
    cudaFreeHost(p);
}

bool host_is_pageable(const void *p) {
    cudaPointerAttributes attr = {};
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) { cudaGetLastError(); return true; }
    return attr.type == cudaMemoryTypeUnregistered;
}

void check_cuda(cudaError_t e, const char *what) {
    if (e != cudaSuccess) { cudaGetLastError(); throw Error(std::string("CUDA error: ") + cudaGetErrorString(e) + " in " + what); }
}

// stream and events of one worker on one device
struct Lane {
    cudaStream_t st = nullptr;
    cudaEvent_t done[2] = {nullptr, nullptr};
};

#if defined(__x86_64__)
__attribute__((target("avx2"))) void copy_past_cache_avx2(char *dst, const char *src, size_t n) {   // dst on a 32-byte boundary
    size_t i = 0;
    for (; i + 128 <= n; i += 128) {
        const __m256i a = _mm256_loadu_si256((const __m256i *)(src + i)), b = _mm256_loadu_si256((const __m256i *)(src + i + 32));
        const __m256i c = _mm256_loadu_si256((const __m256i *)(src + i + 64)), d = _mm256_loadu_si256((const __m256i *)(src + i + 96));
        _mm256_stream_si256((__m256i *)(dst + i), a); _mm256_stream_si256((__m256i *)(dst + i + 32), b);
        _mm256_stream_si256((__m256i *)(dst + i + 64), c); _mm256_stream_si256((__m256i *)(dst + i + 96), d);
    }
    _mm_sfence();
    if (i < n) memcpy(dst + i, src + i, n - i);
}
#endif

// into a slot (page-locked, so on a page boundary)
void copy_past_cache(void *dst, const void *src, size_t n) {
#if defined(__x86_64__)
    static const bool avx2 = __builtin_cpu_supports("avx2");
    if (avx2) { copy_past_cache_avx2(static_cast<char *>(dst), static_cast<const char *>(src), n); return; }
#endif
    memcpy(dst, src, n);
}

// the low halves of n ints; false if one of them does not fit 16 bits
#if defined(__x86_64__)
__attribute__((target("avx2"))) bool copy_low16_avx2(uint16_t *dst, const int *src, size_t n) {   // dst on a 32-byte boundary
    __m256i high = _mm256_setzero_si256();
    const __m256i mask = _mm256_set1_epi32((int)0xffff0000u);
    size_t i = 0;
    for (; i + 32 <= n; i += 32) {
        const __m256i a = _mm256_loadu_si256((const __m256i *)(src + i)), b = _mm256_loadu_si256((const __m256i *)(src + i + 8));
        const __m256i c = _mm256_loadu_si256((const __m256i *)(src + i + 16)), d = _mm256_loadu_si256((const __m256i *)(src + i + 24));
        high = _mm256_or_si256(high, _mm256_and_si256(mask, _mm256_or_si256(_mm256_or_si256(a, b), _mm256_or_si256(c, d))));
        _mm256_stream_si256((__m256i *)(dst + i), _mm256_permute4x64_epi64(_mm256_packus_epi32(a, b), 0xd8));
        _mm256_stream_si256((__m256i *)(dst + i + 16), _mm256_permute4x64_epi64(_mm256_packus_epi32(c, d), 0xd8));
    }
    _mm_sfence();
    int rest = 0;
    for (; i < n; ++i) { dst[i] = (uint16_t)src[i]; rest |= src[i]; }
    return _mm256_testz_si256(high, high) && !((unsigned)rest >> 16);
}
#endif
bool copy_low16(uint16_t *dst, const int *src, size_t n) {
#if defined(__x86_64__)
    static const bool avx2 = __builtin_cpu_supports("avx2");
    if (avx2) return copy_low16_avx2(dst, src, n);
#endif
    int all = 0;
    for (size_t i = 0; i < n; ++i) { dst[i] = (uint16_t)src[i]; all |= src[i]; }
    return !((unsigned)all >> 16);
}

struct Worker {
    Lane lanes[MAX_DEVICES];
    Worker() = default;
    Worker(const Worker &) = delete;
    Worker &operator=(const Worker &) = delete;
    ~Worker() {   // (of a caller that works itself; the threads keep theirs)
        for (Lane &l : lanes) {
            for (cudaEvent_t e : l.done)
                if (e) cudaEventDestroy(e);
            if (l.st) cudaStreamDestroy(l.st);
        }
    }
    Lane &lane(int dev) {
        Lane &l = lanes[dev];
        if (!l.st) {
            check_cuda(cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking), "cudaStreamCreate");
            for (int k = 0; k < 2; ++k) check_cuda(cudaEventCreateWithFlags(&l.done[k], cudaEventDisableTiming), "cudaEventCreate");
        }
        return l;
    }
};

using Pool = WorkerPool<Worker>;

// Never destroyed: the workers wait on it until the process ends.  A process that fork() made has no workers, so it gets a
// pool of its own.
Pool &pool() {
    static std::atomic<Pool *> current{nullptr};
    static const int registered = pthread_atfork(nullptr, nullptr, [] { current = nullptr; });
    (void)registered;
    Pool *p = current;
    if (!p) {
        Pool *made = new Pool(WORKERS);
        if (current.compare_exchange_strong(p, made)) p = made;
        else delete made;
    }
    return *p;
}

// One copy cut into pieces that the workers take in turn.  A worker fills one of its slots while the other is on its way.
struct Transfer {
    char *dev;                 // device side
    char *host;                // host side (read when up, written when down)
    size_t bytes, piece;
    bool up;
    bool narrow = false;       // up: the host side is ints, the device side their low halves
    std::atomic<bool> fits{true};
    std::atomic<size_t> next{0};
    Transfer(void *d, const void *h, size_t n, bool up_, int workers)
        : dev(static_cast<char *>(d)), host(static_cast<char *>(const_cast<void *>(h))), bytes(n), up(up_) {
        piece = std::min(STAGE_BYTES, std::max(STAGE_PIECE_MIN, (n / ((size_t)workers * 4) + 65535) / 65536 * 65536));
    }
    void work(Lane &l, void *const slot[2]) {
        struct Pending { size_t off, len; } pending[2] = {{0, 0}, {0, 0}};
        auto finish = [&](int k) {
            if (!pending[k].len) return;
            check_cuda(cudaEventSynchronize(l.done[k]), "cudaEventSynchronize");
            if (!up) memcpy(host + pending[k].off, slot[k], pending[k].len);
            pending[k].len = 0;
        };
        for (int k = 0;; k ^= 1) {
            const size_t off = next.fetch_add(piece);
            if (off >= bytes) break;
            const size_t len = std::min(piece, bytes - off);
            finish(k);
            if (up) {
                if (!narrow) copy_past_cache(slot[k], host + off, len);
                else if (!fits || !copy_low16(static_cast<uint16_t *>(slot[k]), reinterpret_cast<const int *>(host + 2 * off), len / 2)) { fits = false; break; }
                check_cuda(cudaMemcpyAsync(dev + off, slot[k], len, cudaMemcpyHostToDevice, l.st), "cudaMemcpyAsync");
            } else {
                check_cuda(cudaMemcpyAsync(slot[k], dev + off, len, cudaMemcpyDeviceToHost, l.st), "cudaMemcpyAsync");
            }
            check_cuda(cudaEventRecord(l.done[k], l.st), "cudaEventRecord");
            pending[k] = {off, len};
        }
        for (int k = 0; k < 2; ++k) finish(k);
    }
};

// runs the transfer on the workers; `side` (may be empty) is called by every worker first
void run_staged(Transfer *tr, int n_threads, const std::function<void(int)> &side) {
    int dev = 0;
    TGBM_CUDA(cudaGetDevice(&dev));
    TGBM_CHECK(dev >= 0 && dev < MAX_DEVICES, "device index out of range");
    const int T = std::max(1, std::min(n_threads, WORKERS));
    std::vector<std::string> errors(T);
    pool().run(T, [&](Worker &w, int t) {
        void *slot[2] = {nullptr, nullptr};
        Lane *l = nullptr;
        try {
            if (tr) {
                check_cuda(cudaSetDevice(dev), "cudaSetDevice");
                l = &w.lane(dev);
                for (auto &p : slot)
                    if (!(p = stage_acquire())) throw Error("no page-locked memory for a copy");
                tr->work(*l, slot);
            }
            if (side) side(t);
        } catch (const std::exception &e) {
            errors[t] = e.what();
            if (l) cudaStreamSynchronize(l->st);   // nothing may still use the slots when they go back
        }
        for (void *p : slot) stage_release(p);
    });
    for (const auto &e : errors)
        if (!e.empty()) throw Error(e);
}

bool staging_on() {
    static const bool on = getenv("TGBM_NO_STAGED_UPLOAD") == nullptr;
    return on;
}

}  // namespace

void host_parallel(int n, const std::function<void(int)> &f) {
    if (n <= 1) { if (n == 1) f(0); return; }
    std::vector<std::string> errors(n);
    pool().run(n, [&](Worker &, int t) {
        try { f(t); } catch (const std::exception &e) { errors[t] = e.what(); }
    });
    for (const auto &e : errors)
        if (!e.empty()) throw Error(e);
}

int upload_threads() {
    static const int n = [] {
        if (const char *e = getenv("TGBM_UPLOAD_THREADS")) return std::max(1, std::min(WORKERS, atoi(e)));
        const int hw = (int)std::thread::hardware_concurrency();
        // one core is left to the caller.  16 cores, 1.2 GB of values with 1.2 GB of column ids to look through: 8 / 10 / 12 / 15
        // threads take 58 / 57 / 54 / 51 ms
        return std::max(1, std::min(WORKERS, hw - 1));
    }();
    return n;
}

void upload_h2d(void *dst, const void *src, size_t bytes, cudaStream_t stream, int n_threads) {
    if (bytes == 0) return;
    if (!staging_on() || bytes < STAGE_MIN || n_threads < 1 || !host_is_pageable(src)) {
        TGBM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream));
        return;
    }
    Transfer tr(dst, src, bytes, true, n_threads);
    run_staged(&tr, n_threads, {});   // the pieces are on the device when the workers return: whatever is queued next sees them
}

bool upload_ids16(uint16_t *dst, const int *src, size_t n, int n_threads) {
    if (!staging_on() || sizeof(uint16_t) * n < STAGE_MIN || n_threads < 1 || !host_is_pageable(src)) return false;
    for (size_t i = 0; i < n; i += n / 64 + 1)
        if ((unsigned)src[i] > 0xffffu) return false;   // a glance first
    Transfer tr(dst, src, sizeof(uint16_t) * n, true, n_threads);
    tr.narrow = true;
    run_staged(&tr, n_threads, {});
    return tr.fits;
}

bool upload_csr_values(float *dst, const float *val, const int *row_ptr, const int *col, int n_rows, int n_cols, cudaStream_t stream, int n_threads) {
    const size_t nnz = (size_t)row_ptr[n_rows], bytes = sizeof(float) * nnz;
    // candidates: every row of equal length, first and last row complete
    bool dense = n_rows > 0 && n_cols > 0 && nnz == (size_t)n_rows * (size_t)n_cols && row_ptr[0] == 0 && row_ptr[1] == n_cols;
    auto row_ok = [&](int r) {
        int bad = row_ptr[r] ^ (r * n_cols);
        const int *c = col + (size_t)r * n_cols;
        for (int j = 0; j < n_cols; ++j) bad |= c[j] ^ j;
        return bad == 0;
    };
    dense = dense && row_ok(0) && row_ok(n_rows - 1);
    const bool threads = staging_on() && n_threads >= 1 && bytes >= STAGE_MIN;
    const bool staged = threads && host_is_pageable(val);
    if (!staged && bytes) TGBM_CUDA(cudaMemcpyAsync(dst, val, bytes, cudaMemcpyHostToDevice, stream));
    if (!dense && !staged) return false;
    std::atomic<bool> ok{dense};
    if (!threads) {
        for (int r = 0; r < n_rows && ok; ++r) ok = row_ok(r);
        return ok;
    }
    // The column ids are read while the values are on their way: blocks of rows against one block of 0 .. n_cols - 1 over
    // and over, which stays in the cache.
    std::atomic<int> next{0};
    const int rows = std::max(1, (16 << 10) / std::max(1, n_cols));
    std::vector<int> pattern;
    if (dense) {
        pattern.resize((size_t)rows * n_cols);
        for (size_t i = 0; i < pattern.size(); ++i) pattern[i] = (int)(i % (size_t)n_cols);
    }
    auto check_rows = [&](int) {
        for (;;) {
            const long long r0 = (long long)next.fetch_add(1) * rows;
            if (r0 >= n_rows || !ok) return;
            const int r1 = (int)std::min<long long>(n_rows, r0 + rows);
            int bad = 0;
            for (int r = (int)r0; r < r1; ++r) bad |= row_ptr[r] ^ (r * n_cols);
            if (bad || memcmp(col + (size_t)r0 * n_cols, pattern.data(), sizeof(int) * (size_t)(r1 - r0) * n_cols)) { ok = false; return; }
        }
    };
    std::function<void(int)> side;
    if (dense) side = check_rows;
    if (staged) {
        Transfer tr(dst, val, bytes, true, n_threads);
        run_staged(&tr, n_threads, side);
    } else {
        run_staged(nullptr, n_threads, side);
    }
    return ok;
}

void download_d2h(void *dst, const void *src, size_t bytes, cudaStream_t stream, int n_threads) {
    if (bytes == 0) return;
    if (!staging_on() || bytes < STAGE_MIN || n_threads < 1 || !host_is_pageable(dst)) {
        TGBM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream));
        TGBM_CUDA(cudaStreamSynchronize(stream));
        return;
    }
    TGBM_CUDA(cudaStreamSynchronize(stream));   // what the workers read has been written
    Transfer tr(const_cast<void *>(src), dst, bytes, false, n_threads);
    run_staged(&tr, n_threads, {});
}

void dev_trim() noexcept { trim_all(keep_bytes(), true); }
void dev_release_all() noexcept {
    trim_all(0, false);
    std::vector<void *> slots;
    {
        std::lock_guard<std::mutex> lock(g_stage_mutex);
        slots.swap(g_stage_free);
    }
    for (void *p : slots) cudaFreeHost(p);
}

}  // namespace tgbm
