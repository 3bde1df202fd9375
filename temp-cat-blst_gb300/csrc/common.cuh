// Shared host/device plumbing for the sm_103a BLS12-381 G1 library:
// per-thread CUDA context (stream, grow-only device and pinned buffers) and
// error helpers.  All public entry points are synchronous and fail closed.
#pragma once
#include <cuda_runtime.h>
#include <array>
#include <atomic>
#include <cstring>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

namespace catmsm {

// SMs of a GB300 (two dies of 76): used only by host-side plan models that
// run without a device; launches size their grids from device_sms().
constexpr int kGB300SMs = 152;

// SM count of the current device, queried once per device (devices past the
// cache are queried on every call); grids are sized in multiples of it.  The
// cache is shared by every calling thread: atomic entries, each written with
// the same value by whichever thread gets there first.
inline int device_sms()
{
    static std::atomic<int> cache[64];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    if (dev >= 0 && dev < 64) {
        const int v = cache[dev].load(std::memory_order_relaxed);
        if (v > 0) return v;
    }
    int sms = 0;
    if (dev < 0 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return kGB300SMs;   // only reached with a broken context; the next launch reports the error
    if (dev < 64) cache[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
    uint32_t moves = 0;      // times the address changed: what holds it (a captured graph) is stale after that
    void* get(size_t bytes)
    {
        if (bytes == 0) bytes = 256;
        if (bytes > cap) {
            release();
            moves++;
            if (cudaMalloc(&p, bytes) != cudaSuccess) {
                cudaGetLastError();      // the null pointer reports it; the next call's launches must not
                p = nullptr;
                return nullptr;
            }
            cap = bytes;
        }
        return p;
    }
    void release()
    {
        if (!p) return;
        cudaFree(p);
        p = nullptr;
        cap = 0;
        moves++;
    }
};

struct PinnedBuf {
    void* p = nullptr;
    size_t cap = 0;
    void* get(size_t bytes)
    {
        if (bytes == 0) bytes = 256;
        if (bytes > cap) {
            if (p) cudaFreeHost(p);
            p = nullptr;
            cap = 0;
            if (cudaHostAlloc(&p, bytes, cudaHostAllocDefault) != cudaSuccess) {
                cudaGetLastError();
                p = nullptr;
                return nullptr;
            }
            cap = bytes;
        }
        return p;
    }
    void release()
    {
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
    }
};

// A second stream of a pipeline, forked from and joined to its own.
struct AuxStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    // created on first use, at the pipeline stream's priority
    cudaError_t ensure(cudaStream_t st)
    {
        cudaError_t e = cudaSuccess;
        if (!stream) {
            int prio = 0;
            e = cudaStreamGetPriority(st, &prio);
            if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&stream, cudaStreamNonBlocking, prio);
        }
        if (e == cudaSuccess && !fork) e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
        if (e == cudaSuccess && !join) e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
        return e;
    }
    cudaError_t begin(cudaStream_t st) const
    {
        const cudaError_t e = cudaEventRecord(fork, st);
        return e == cudaSuccess ? cudaStreamWaitEvent(stream, fork, 0) : e;
    }
    // Failing, it waits: the pipeline's next work must not meet what is queued here.
    cudaError_t end(cudaStream_t st) const
    {
        cudaError_t e = cudaEventRecord(join, stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(st, join, 0);
        if (e != cudaSuccess) cudaStreamSynchronize(stream);
        return e;
    }
    void release()
    {
        for (cudaEvent_t* e : {&fork, &join}) {
            if (*e) cudaEventDestroy(*e);
            *e = nullptr;
        }
        if (stream) cudaStreamDestroy(stream);
        stream = nullptr;
    }
};

// Workspaces of the batch-affine accumulation (bucket_affine.cu): one set per
// stream of the two its slices alternate between, and the second stream (which
// runs the second half of a large decode too).
struct AffWork {
    struct Set {
        DevBuf pts0, pts1, key0, key1, meta, pairpos, prefix, rest, gtot;
        std::array<DevBuf*, 9> bufs()
        {
            return {&pts0, &pts1, &key0, &key1, &meta, &pairpos, &prefix, &rest, &gtot};
        }
    } set[2];
    AuxStream aux;
    uint32_t moves()
    {
        uint32_t m = 0;
        for (Set& w : set)
            for (const DevBuf* b : w.bufs()) m += b->moves;
        return m;
    }
    void release_lists()
    {
        for (Set& w : set)
            for (DevBuf* b : w.bufs()) b->release();
    }
    void release()
    {
        release_lists();
        aux.release();
    }
};

// Device workspaces of one MSM pipeline instance.
struct MsmWork {
    DevBuf points, scalars, digits, ranks, counts, offsets, block_sums, sorted_pt, sorted_key,
        buckets, head, tail, seg, total, status, misc, glv_pts, glv_sc, glv_sign;
    AffWork aff;
    void release()
    {
        for (DevBuf* b : {&points, &scalars, &digits, &ranks, &counts, &offsets, &block_sums, &sorted_pt,
                          &sorted_key, &buckets, &head, &tail, &seg, &total, &status, &misc, &glv_pts,
                          &glv_sc, &glv_sign})
            b->release();
        aff.release();
    }
};

struct FftWork {
    DevBuf values, roots, glv, scratch, prod, meta;
    AuxStream aux;
    void release()
    {
        aux.release();
        for (DevBuf* b : {&values, &roots, &glv, &scratch, &prod, &meta}) b->release();
    }
};

// Per-stage CUDA-event timing of the MSM pipeline (off by default).
constexpr int kMsmStages = 8;   // prep (memsets, GLV scalar split), digits, scan, scatter (+ GLV points), accumulate, fixup, reduce, host fold
struct StageProfile {
    bool enabled = false;
    cudaEvent_t ev[kMsmStages + 1] = {};
    double ms[kMsmStages] = {};
    long calls = 0;
    double entries = 0;   // bucket entries (nonzero digits) accumulated
};

struct Ctx {
    int device = -1;
    cudaStream_t stream = nullptr;
    MsmWork msm;
    FftWork fft;
    PinnedBuf h_points, h_scalars, h_out, h_values, h_meta;
    StageProfile prof;
    bool glv = true;   // GLV split of scalars wider than 128 bits (catmsm_msm_glv)
    int affine_rounds = -1;   // batch-affine accumulation rounds (-1: by size; catmsm_msm_affine_rounds)
    cudaStream_t copy_stream = nullptr;    // host->device point copies that overlap the scalar stages
    cudaEvent_t points_ready = nullptr;
};

// Per-thread context bound to the thread's current device.  A thread's
// contexts (their streams, events and grow-only workspaces: ~15 GB after a
// 2^22-point MSM) are released when the thread exits; the main thread's are
// left to process teardown.
Ctx* get_ctx();

// Launch-time stats, readable through catmsm_last_launches() for the bench.
struct LaunchStats {
    int launches = 0;
};
extern thread_local LaunchStats g_stats;

#define CATMSM_CHECK(x)                    \
    do {                                   \
        cudaError_t e__ = (x);             \
        if (e__ != cudaSuccess) return e__; \
    } while (0)

// Waits for the stream, also after a failure: nothing that is queued uses the
// caller's memory after the return.
inline cudaError_t wait_stream(cudaStream_t st, cudaError_t err)
{
    const cudaError_t e = cudaStreamSynchronize(st);
    return err == cudaSuccess ? e : err;
}

inline unsigned div_up(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

// Host copy between caller memory and pinned staging.  Large copies are
// split over up to 8 host threads: one core moves ~10-20 GB/s, and a batch's
// scalars or an FFT batch's values (tens of MB) would otherwise cost
// milliseconds next to a device pass of similar length.
inline void host_copy(void* dst, const void* src, size_t bytes)
{
    constexpr size_t kSplit = size_t(8) << 20;
    if (bytes < kSplit) {
        std::memcpy(dst, src, bytes);
        return;
    }
    unsigned nt = std::thread::hardware_concurrency();
    nt = nt < 2 ? 1 : (nt > 8 ? 8 : nt);
    if (nt == 1) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const size_t part = ((bytes + nt - 1) / nt + 63) & ~size_t(63);
    std::vector<std::thread> th;
    th.reserve(nt);
    for (unsigned k = 0; k < nt; k++) {
        const size_t off = (size_t)k * part;
        if (off >= bytes) break;
        const size_t len = bytes - off < part ? bytes - off : part;
        try {
            th.emplace_back([=] { std::memcpy((char*)dst + off, (const char*)src + off, len); });
        } catch (...) {
            std::memcpy((char*)dst + off, (const char*)src + off, len);
        }
    }
    for (auto& t : th) t.join();
}

// Gather the descriptor walk of multi_scalar.cpp:830-841 into contiguous
// host staging; returns the contiguous base directly when possible.
// Rank of this lane's entry within bucket `key` (kNoBucket: no entry), with
// one atomic per distinct key of the warp: lanes that share a bucket take
// consecutive ranks.  Uniform scalars rarely share one (no measurable cost at
// 2^20); all-equal scalars or 0/1 coefficients put whole warps on one counter,
// which serialised the digit kernels (2^20 equal scalars: 1.93 -> 0.07 ms).
// All 32 lanes of the warp must call it together.
constexpr uint32_t kNoBucket = 0xffffffffu;

__device__ __forceinline__ uint32_t warp_bucket_rank(uint32_t key, uint32_t* counts)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t peers = __match_any_sync(0xffffffffu, key);
    const uint32_t leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (key != kNoBucket && lane == leader) base = atomicAdd(&counts[key], (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(peers & ((1u << lane) - 1));
}

template <typename T>
inline const uint8_t* gather(const T* const arr[], size_t n, size_t elem, PinnedBuf& stage, bool& err)
{
    err = false;
    if (n == 1 || arr[1] == nullptr) return reinterpret_cast<const uint8_t*>(arr[0]);
    uint8_t* dst = (uint8_t*)stage.get(n * elem);
    if (!dst) { err = true; return nullptr; }
    const uint8_t* cur = reinterpret_cast<const uint8_t*>(arr[0]);
    const T* const* next = arr + 1;
    std::memcpy(dst, cur, elem);
    for (size_t i = 1; i < n; i++) {
        if (*next) cur = reinterpret_cast<const uint8_t*>(*next++);
        else cur += elem;
        std::memcpy(dst + i * elem, cur, elem);
    }
    return dst;
}

}  // namespace catmsm
