// Batched commitments over a resident basis (no reference counterpart; the
// reference's closest API is the fixed-base wbits MSM, c_api.cpp:1310-1369).
//
// A basis of n affine points is uploaded once and expanded into fixed-base
// tables T[w][i] = 2^(c w) P_i (affine, w < D = 256/c + 1).  A batch of MSMs,
// MSM j over the first k_j basis points with 255/256-bit scalars, then needs
// no window fold: sum_i k_ji P_i = sum_i sum_w d_jiw T[w][i], so every
// (point, window) digit of MSM j drops into ONE set of 2^(c-1) buckets owned
// by that MSM.  The kernels of the plain pipeline (counting sort, chunked
// accumulation, fixup, running-sum reduction) run unchanged over the key
// space (msm, bucket); the reduction's root is each MSM's result.
//
// The device sequence of a batch (one launch per stage, sizes read from
// device memory) is captured once per (batch size, window, chunk) into a CUDA
// graph and replayed: one graph launch per batch.  A small autotuner times
// candidate (window, chunk) pairs on a caller batch and remembers the winner
// per (device, basis size, batch size, points-per-MSM class) in a text cache.
#include "common.cuh"
#include "curve.cuh"
#include "host_curve.hpp"
#include "catmsm_internal.h"
#include "catmsm_gpu.h"

#include <sys/stat.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

namespace catmsm {

// plain-pipeline kernels (msm.cu)
__global__ void k_scan_local(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                             uint32_t* __restrict__ block_sums, uint32_t M);
__global__ void k_scan_top(uint32_t* __restrict__ block_sums, uint32_t nb, uint32_t* __restrict__ total_out);
__global__ void k_scan_add(uint32_t* __restrict__ out, const uint32_t* __restrict__ block_sums, uint32_t M);
__global__ void k_accumulate(const affine* __restrict__ pts, const uint32_t* __restrict__ sorted_pt,
                             const uint32_t* __restrict__ sorted_key, const uint32_t* __restrict__ total_ptr, uint32_t below,
                             uint32_t L, xyzz* __restrict__ buckets, xyzz* __restrict__ head,
                             xyzz* __restrict__ tail);
__global__ void k_fixup(const uint32_t* __restrict__ sorted_key, const uint32_t* __restrict__ offsets,
                        const uint32_t* __restrict__ total_ptr, uint32_t L, xyzz* __restrict__ buckets,
                        const xyzz* __restrict__ head, const xyzz* __restrict__ tail,
                        uint2* __restrict__ hot_list, uint32_t* __restrict__ hot_count);
__global__ void k_fixup_hot(uint2* __restrict__ hot_list, uint32_t* __restrict__ hot_count,
                            const uint32_t* __restrict__ offsets, uint32_t L, xyzz* __restrict__ buckets,
                            const xyzz* __restrict__ head, const xyzz* __restrict__ tail);
__global__ void k_fixup_seg(const uint32_t* __restrict__ sorted_key, const uint32_t* __restrict__ total_ptr,
                            uint32_t L, xyzz* __restrict__ head);
__global__ void k_fixup_join(const uint32_t* __restrict__ sorted_key, const uint32_t* __restrict__ offsets,
                             const uint32_t* __restrict__ total_ptr, uint32_t L, xyzz* __restrict__ buckets,
                             const xyzz* __restrict__ head, const xyzz* __restrict__ tail,
                             uint2* __restrict__ hot_list, uint32_t* __restrict__ hot_count);
__global__ void k_fixup_hot_seg(uint2* __restrict__ hot_list, uint32_t* __restrict__ hot_count,
                                const uint32_t* __restrict__ offsets, uint32_t L, xyzz* __restrict__ buckets,
                                const xyzz* __restrict__ head, const xyzz* __restrict__ tail);

constexpr int kScanTileB = 1024 * 4;

// ---------------------------------------------------------------- tables
// T[w][i] = 2^(c w) P_i, one point per thread: D-1 runs of c doublings, then
// Montgomery's simultaneous inversion over the D multiples (one field
// inversion per point).  q: D xyzz scratch per point, pre: D prefix products.
__global__ void __launch_bounds__(64) k_build_tables(const affine* __restrict__ pts, uint32_t n, uint32_t c,
                                                     uint32_t D, affine* __restrict__ table, xyzz* __restrict__ tmp,
                                                     fp* __restrict__ pre_buf)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const affine p = pts[i];
    xyzz* q = tmp + (size_t)i * D;
    fp* pre = pre_buf + (size_t)i * D;
    xyzz acc;
    if (aff_is_inf(p)) {
        xyzz_set_inf(acc);
    } else {
        acc.x = p.x; acc.y = p.y;
        fp_set_one(acc.zz); fp_set_one(acc.zzz);
    }
    fp prod;
    fp_set_one(prod);
    for (uint32_t w = 0; w < D; w++) {
        if (w)
            for (uint32_t k = 0; k < c; k++) xyzz_dbl(acc);
        q[w] = acc;
        pre[w] = prod;
        if (!xyzz_is_inf(acc)) {
            fp t;
            fp_mul(t, acc.zz, acc.zzz);
            fp_mul(prod, prod, t);
        }
    }
    fp inv;
    fp_inv(inv, prod);                           // 1 / prod of all (zz zzz)
    for (int w = (int)D - 1; w >= 0; w--) {
        const xyzz e = q[w];
        affine o;
        if (xyzz_is_inf(e)) {
            fp_zero(o.x); fp_zero(o.y);
        } else {
            fp zz_zzz, ie, t;
            fp_mul(zz_zzz, e.zz, e.zzz);
            fp_mul(ie, inv, pre[w]);             // 1 / (zz zzz) of entry w
            fp_mul(inv, inv, zz_zzz);            // drop entry w from the running inverse
            fp_mul(t, ie, e.zzz);                // 1 / zz
            fp_mul(o.x, e.x, t);
            fp_mul(t, ie, e.zz);                 // 1 / zzz
            fp_mul(o.y, e.y, t);
            fp_canon(o.x, o.x);
            fp_canon(o.y, o.y);
        }
        table[(size_t)w * n + i] = o;
    }
}

// ---------------------------------------------------------------- bucket sort
// Signed c-bit window digit w of the scalar k (9 words, k[8] = 0), the same
// recoding as the plain pipeline; carry is the running carry.
__device__ __forceinline__ int32_t batch_digit(const uint32_t* k, uint32_t w, uint32_t c, uint32_t& carry)
{
    const uint32_t bit = w * c, word = bit >> 5, sh = bit & 31;
    uint32_t raw = k[word] >> sh;
    if (sh && word + 1 < 9) raw |= k[word + 1] << (32 - sh);
    raw &= (1u << c) - 1;
    int32_t d = (int32_t)(raw + carry);
    carry = d > (int32_t)(1u << (c - 1)) ? 1u : 0u;
    return d - (int32_t)(carry << c);
}

__device__ __forceinline__ void load_scalar32(uint32_t* k, const uint8_t* s)
{
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(s)), b = __ldg(reinterpret_cast<const uint4*>(s) + 1);
    k[0] = a.x; k[1] = a.y; k[2] = a.z; k[3] = a.w;
    k[4] = b.x; k[5] = b.y; k[6] = b.z; k[7] = b.w;
    k[8] = 0;
}

// Part sort: a block takes one part, up to kPartPairs consecutive pairs of ONE
// MSM (part p: MSM part[2 p], first pair part[2 p + 1], until the part's size or
// the MSM's end).  k_part_count counts its digits per bucket in shared memory,
// then one global atomic per (part, bucket) reserves the part's ranks.
// k_part_scatter sorts the part in shared memory and copies each bucket's run
// to its place, a warp per bucket, so the writes are runs and not single words.
// No digit, rank or index arrays (400 MB written and read again for 33 M entries) and
// ~24 times fewer global atomics, which bounded the per-pair form below: 1.11 ->
// 0.28 ms for 1024 MSMs of 33 M entries in all (single-word scattered writes: 0.81).
// For MSMs of at most kPartMaxB buckets whose part fits shared memory: up to
// kPartAnyB buckets always, above in batches of at least kPartMinFill entries per
// bucket of an MSM.  With fewer the launches last as long as one block, whose copies
// go over all buckets; the form per pair lasts as long as a thread's D digits.  Per pair
// against by parts, us: 12 bits, 8 x 4096 pairs (352 a bucket) 44 / 62, 16 x 4096 (704)
// 75 / 62; 13 bits, 24 x 4096 (480) 85 / 91, 32 x 4096 (640) 113 / 92; 11 bits, 8 x 4096
// (768) 49 / 50, 256 x 100 (600) 45 / 45; 9 bits, 64 x 100 (725) 41 / 30; 8 bits, one MSM of
// 500 (129) 40 / 30, of 2000 (516) 39 / 45.
constexpr uint32_t kPartPairs = 1024;
constexpr uint32_t kPartThreads = 512;
constexpr uint32_t kPartMaxB = 4096;
constexpr size_t kPartMinFill = 600, kPartAnyB = 512;
constexpr size_t kPartMaxSmem = 220 * 1024;

static size_t part_smem(uint32_t c, uint32_t D) { return ((size_t)2 << (c - 1)) * 4 + 128 + (size_t)kPartPairs * D * 4; }

__global__ void __launch_bounds__(kPartThreads) k_part_count(const uint8_t* __restrict__ scalars,
                                                             const uint32_t* __restrict__ off,
                                                             const uint32_t* __restrict__ part,
                                                             const uint32_t* __restrict__ nparts, uint32_t c,
                                                             uint32_t D, uint32_t* __restrict__ counts,
                                                             uint2* __restrict__ base)
{
    extern __shared__ uint32_t cnt[];
    if (blockIdx.x >= *nparts) return;
    const uint32_t B = 1u << (c - 1);
    const uint32_t j = part[2 * blockIdx.x], f0 = part[2 * blockIdx.x + 1];
    const uint32_t f1 = min(f0 + kPartPairs, off[j + 1]);
    for (uint32_t i = threadIdx.x; i < B; i += kPartThreads) cnt[i] = 0;
    __syncthreads();
    for (uint32_t f = f0 + threadIdx.x; f < f1; f += kPartThreads) {
        uint32_t k[9], carry = 0;
        load_scalar32(k, scalars + (size_t)f * 32);
        for (uint32_t w = 0; w < D; w++) {
            const int32_t d = batch_digit(k, w, c, carry);
            if (d != 0) atomicAdd(&cnt[(d < 0 ? -d : d) - 1], 1u);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < B; i += kPartThreads)       // (rank of the part's first entry, entries)
        base[(size_t)blockIdx.x * B + i] = make_uint2(cnt[i] ? atomicAdd(&counts[j * B + i], cnt[i]) : 0, cnt[i]);
}

__global__ void __launch_bounds__(kPartThreads) k_part_scatter(const uint8_t* __restrict__ scalars,
                                                               const uint32_t* __restrict__ off,
                                                               const uint32_t* __restrict__ part,
                                                               const uint32_t* __restrict__ nparts, uint32_t n,
                                                               uint32_t c, uint32_t D, const uint2* __restrict__ base,
                                                               const uint32_t* __restrict__ offsets,
                                                               uint32_t* __restrict__ sorted_pt,
                                                               uint32_t* __restrict__ sorted_key)
{
    extern __shared__ uint32_t sh[];
    if (blockIdx.x >= *nparts) return;
    const uint32_t B = 1u << (c - 1);
    uint32_t* end = sh;                   // cursor of each bucket's run, finally its end
    uint32_t* dst = sh + B;               // global position of the run
    uint32_t* sums = dst + B;             // 32 words: warp sums of the scan
    uint32_t* val = sums + 32;            // the sorted part
    const uint32_t j = part[2 * blockIdx.x], f0 = part[2 * blockIdx.x + 1];
    const uint32_t f1 = min(f0 + kPartPairs, off[j + 1]);
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    // exclusive scan of the part's counts, B / kPartThreads (or 1) buckets a thread
    const uint32_t per = (B + kPartThreads - 1) / kPartThreads, b0 = tid * per;
    uint32_t sum = 0;
    for (uint32_t i = b0; i < min(b0 + per, B); i++) {
        const uint2 e = base[(size_t)blockIdx.x * B + i];
        dst[i] = offsets[j * B + i] + e.x;
        end[i] = sum;
        sum += e.y;
    }
    uint32_t x = sum;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) sums[wid] = x;
    __syncthreads();
    uint32_t pre = x - sum;
    for (uint32_t w = 0; w < wid; w++) pre += sums[w];
    for (uint32_t i = b0; i < min(b0 + per, B); i++) end[i] += pre;
    __syncthreads();
    for (uint32_t f = f0 + tid; f < f1; f += kPartThreads) {
        uint32_t k[9], carry = 0;
        load_scalar32(k, scalars + (size_t)f * 32);
        for (uint32_t w = 0; w < D; w++) {
            const int32_t d = batch_digit(k, w, c, carry);
            if (d == 0) continue;
            const uint32_t pos = atomicAdd(&end[(d < 0 ? -d : d) - 1], 1u);
            val[pos] = (w * n + (f - off[j])) | (d < 0 ? 0x80000000u : 0u);
        }
    }
    __syncthreads();
    for (uint32_t i = wid; i < B; i += kPartThreads / 32) {
        const uint32_t s = i ? end[i - 1] : 0, m = end[i] - s, o = dst[i];
        for (uint32_t e = lane; e < m; e += 32) {
            sorted_pt[o + e] = val[s + e];
            sorted_key[o + e] = j * B + i;
        }
    }
}

// Per-pair sort (wider windows): one thread per (MSM, point) pair in flat order;
// off[j] = first pair of MSM j (off[nmsm] = total pairs).  The key is j * B +
// (|d| - 1) and the point index the table slot w * n + i.
__global__ void k_digits_batch(const uint8_t* __restrict__ scalars, const uint32_t* __restrict__ off,
                               uint32_t nmsm, uint32_t n, uint32_t c, uint32_t D, uint32_t cap,
                               uint32_t* __restrict__ digits, uint32_t* __restrict__ ranks,
                               uint32_t* __restrict__ pidx, uint32_t* __restrict__ counts)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t P = off[nmsm];
    if (f >= P || f >= cap) return;
    uint32_t lo = 0, hi = nmsm;                   // find j with off[j] <= f < off[j+1]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (off[mid] <= f) lo = mid;
        else hi = mid;
    }
    const uint32_t j = lo, i = f - off[j];
    uint32_t k[9], carry = 0;
    load_scalar32(k, scalars + (size_t)f * 32);
    const uint32_t B = 1u << (c - 1);
    for (uint32_t w = 0; w < D; w++) {
        const int32_t d = batch_digit(k, w, c, carry);
        const size_t o = (size_t)f * D + w;
        if (d == 0) {
            digits[o] = 0xffffffffu;
        } else {
            // plain atomics: an MSM of the batch has at most n points per
            // bucket, and warp aggregation cost more than it saved here
            const uint32_t key = j * B + (uint32_t)(d < 0 ? -d : d) - 1;
            ranks[o] = atomicAdd(&counts[key], 1u);
            digits[o] = key | (d < 0 ? 0x80000000u : 0u);
            pidx[o] = w * n + i;
        }
    }
}

__global__ void k_scatter_batch(const uint32_t* __restrict__ digits, const uint32_t* __restrict__ ranks,
                                const uint32_t* __restrict__ pidx, const uint32_t* __restrict__ offsets,
                                const uint32_t* __restrict__ off, uint32_t nmsm, uint32_t D, uint32_t cap,
                                uint32_t* __restrict__ sorted_pt, uint32_t* __restrict__ sorted_key)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nD = off[nmsm] * D;
    if (t >= nD || t >= cap) return;
    const uint32_t dg = digits[t];
    if (dg == 0xffffffffu) return;
    const uint32_t key = dg & 0x7fffffffu;
    const uint32_t pos = offsets[key] + ranks[t];
    sorted_pt[pos] = pidx[t] | (dg & 0x80000000u);
    sorted_key[pos] = key;
}

// results: root Q (xyzz) of each MSM -> Jacobian with canonical coordinates
__global__ void k_batch_out(const xyzz* __restrict__ roots, uint32_t nmsm, jac* __restrict__ out)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nmsm) return;
    xyzz p = roots[j];
    jac o;
    xyzz_to_jac(o, p);
    if (!fp_is_zero(o.z)) {
        fp_canon(o.x, o.x);
        fp_canon(o.y, o.y);
        fp_canon(o.z, o.z);
    } else {
        jac_set_inf(o);
    }
    out[j] = o;
}

// ---------------------------------------------------------------- basis object
// How a batch of one size runs, by its entries: the affine rounds of its accumulation,
// the form of its sort, and whether its buckets hold two entries or more (with rounds
// they do, and the window alone gives the sort).
struct BatchRoute {
    uint32_t rounds = 0;
    bool parts = false, dense = false;
    uint32_t kind() const { return rounds ? 3 + rounds : (parts ? 1 : 0) + (dense ? 2 : 0); }
};

// The captured graphs of a workspace, one per route: batches of one size whose
// entries lie on both sides of a threshold alternate between them.
struct BatchGraph {
    static constexpr uint32_t kMaxRounds = 3, kKinds = 4 + kMaxRounds;
    cudaGraphExec_t exec[kKinds] = {};
    uint32_t nmsm = 0, c = 0, L = 0;
    uint32_t moves = 0;      // BatchWork::moves() at the capture: the graphs hold the buffers' addresses
    size_t cap = 0;
};

struct Basis;

// Device/pinned workspace of one batch pipeline instance (a basis has one;
// a server worker has its own, sharing the basis tables).
struct BatchWork {
    DevBuf scal, off, digits, ranks, pidx, base, counts, offsets, bsums, sorted_pt, sorted_key, buckets, head, tail,
        hot, seg, out;
    PinnedBuf h_scal, h_off, h_out;
    AffWork aff;
    BatchGraph graph;
    std::array<DevBuf*, 17> bufs()
    {
        return {&scal, &off, &digits, &ranks, &pidx, &base, &counts, &offsets, &bsums, &sorted_pt,
                &sorted_key, &buckets, &head, &tail, &hot, &seg, &out};
    }
    uint32_t moves()
    {
        uint32_t m = aff.moves();
        for (const DevBuf* d : bufs()) m += d->moves;
        return m;
    }
    // Whether the graphs are of nmsm MSMs over b's tables and address the buffers as they are.
    bool graph_fits(const Basis* b, uint32_t nmsm);
    void drop_graph()
    {
        for (cudaGraphExec_t e : graph.exec)
            if (e) cudaGraphExecDestroy(e);
        graph = BatchGraph();
    }
    void release()
    {
        drop_graph();
        aff.release();
        for (DevBuf* d : bufs()) d->release();
        PinnedBuf* hb[] = {&h_scal, &h_off, &h_out};
        for (PinnedBuf* h : hb) {
            if (h->p) cudaFreeHost(h->p);
            h->p = nullptr;
            h->cap = 0;
        }
    }
};

struct Basis {
    int device = -1;
    size_t n = 0;
    uint32_t c = 0, D = 0, L = 16;
    bool tables = false;   // the tables of window c are built (not after a failed rebuild: batches fail)
    cudaStream_t stream = nullptr;
    DevBuf points, table, tmp;
    BatchWork work;
    std::mutex mu;     // serialises the direct calls (batches, reconfiguration, autotuning): they share the
                       // basis's workspace and stream, and a rebuild replaces the tables a batch reads
};

// A buffer that moved since the capture (a larger batch, another chunk length, an
// allocation that failed half-way) leaves the graphs with freed addresses.
bool BatchWork::graph_fits(const Basis* b, uint32_t nmsm)
{
    return graph.moves == moves() && graph.nmsm == nmsm && graph.c == b->c && graph.L == b->L;
}

static cudaError_t build_tables(Basis* b, uint32_t c)
{
    const uint32_t D = 256 / c + 1;
    b->tables = false;
    affine* table = (affine*)b->table.get((size_t)D * b->n * sizeof(affine));
    xyzz* tmp = (xyzz*)b->tmp.get((size_t)D * b->n * (sizeof(xyzz) + sizeof(fp)));
    if (!table || !tmp) return cudaErrorMemoryAllocation;
    k_build_tables<<<div_up(b->n, 64), 64, 0, b->stream>>>((const affine*)b->points.p, (uint32_t)b->n, c, D,
                                                          table, tmp, (fp*)(tmp + (size_t)D * b->n));
    CATMSM_CHECK(cudaGetLastError());
    CATMSM_CHECK(cudaStreamSynchronize(b->stream));
    b->tmp.release();
    b->c = c;
    b->D = D;
    b->tables = true;
    b->work.drop_graph();
    return cudaSuccess;
}

// Whether a batch of that many entries takes the part sort, and the most parts it can have.
static bool part_sort(const Basis* b, size_t entries)
{
    const size_t B = (size_t)1 << (b->c - 1);
    return B <= kPartMaxB && part_smem(b->c, b->D) <= kPartMaxSmem &&
           (B <= kPartAnyB || entries >= kPartMinFill * B);
}

static size_t max_parts(uint32_t nmsm, size_t cap) { return cap / kPartPairs + nmsm; }

// Workspace for batches of up to nmsm MSMs and cap pairs.
static cudaError_t ensure_work(const Basis* b, BatchWork* w, uint32_t nmsm, size_t cap, bool parts)
{
    const uint32_t B = 1u << (b->c - 1);
    const size_t M = (size_t)nmsm * B;
    const size_t nD = cap * b->D;
    const size_t chunks = (nD + b->L - 1) / b->L + 1;
    const size_t lvl1 = (size_t)nmsm * ((B + 7) / 8);
    const size_t lvl2 = (size_t)nmsm * ((B + 15) / 16) + nmsm;
    const size_t meta = (nmsm + 2 + 2 * max_parts(nmsm, cap)) * 4;      // off, number of parts, parts
    const bool sorts = parts ? w->base.get(max_parts(nmsm, cap) * B * sizeof(uint2)) != nullptr
                                    : w->digits.get(nD * 4) && w->ranks.get(nD * 4) && w->pidx.get(nD * 4);
    bool ok = sorts && w->scal.get(cap * 32) && w->off.get(meta) && w->counts.get(M * 4) &&
              w->offsets.get((M + 1) * 4) &&
              w->bsums.get(((M + kScanTileB - 1) / kScanTileB) * 4 + 4) && w->sorted_pt.get(nD * 4) &&
              w->sorted_key.get(nD * 4) && w->buckets.get(M * sizeof(xyzz)) &&
              w->head.get(chunks * sizeof(xyzz)) && w->tail.get(chunks * sizeof(xyzz)) &&
              w->hot.get(256 + chunks * sizeof(uint2)) && w->seg.get(2 * (lvl1 + lvl2) * sizeof(xyzz)) &&
              w->out.get((size_t)nmsm * sizeof(jac)) && w->h_off.get(meta) &&
              w->h_out.get((size_t)nmsm * sizeof(jac));
    return ok ? cudaSuccess : cudaErrorMemoryAllocation;
}

// The device sequence of one batch (everything after the input copies).  *kernels:
// the number of kernels it launched.
static cudaError_t enqueue_batch(const Basis* b, BatchWork* w, cudaStream_t st, uint32_t nmsm, size_t cap,
                                 BatchRoute route, uint32_t* kernels)
{
    const uint32_t rounds = route.rounds;
    const bool parts = route.parts;
    const uint32_t c = b->c, D = b->D, L = b->L, B = 1u << (c - 1);
    const size_t M = (size_t)nmsm * B;
    const size_t nD = cap * D;
    const size_t chunks = (nD + L - 1) / L + 1;
    const uint32_t nblocks = (uint32_t)((M + kScanTileB - 1) / kScanTileB);
    const size_t lvl1 = (size_t)nmsm * ((B + 7) / 8);
    const size_t lvl2 = (size_t)nmsm * ((B + 15) / 16) + nmsm;
    uint32_t* off = (uint32_t*)w->off.p;
    uint32_t* counts = (uint32_t*)w->counts.p;
    uint32_t* offsets = (uint32_t*)w->offsets.p;
    uint32_t* total = offsets + M;
    uint32_t* hot_count = (uint32_t*)w->hot.p;
    uint2* hot_list = reinterpret_cast<uint2*>(hot_count + 64);
    xyzz* buckets = (xyzz*)w->buckets.p;
    xyzz* head = (xyzz*)w->head.p;
    xyzz* tail = (xyzz*)w->tail.p;
    xyzz* seg = (xyzz*)w->seg.p;
    cudaMemsetAsync(counts, 0, M * 4, st);
    cudaMemsetAsync(buckets, 0, M * sizeof(xyzz), st);
    cudaMemsetAsync(hot_count, 0, 12, st);
    const uint32_t* nparts = off + nmsm + 1;
    const unsigned pgrid = (unsigned)max_parts(nmsm, cap);
    uint32_t* sorted_pt = (uint32_t*)w->sorted_pt.p;
    uint32_t* sorted_key = (uint32_t*)w->sorted_key.p;
    if (parts)
        k_part_count<<<pgrid, kPartThreads, B * 4, st>>>((const uint8_t*)w->scal.p, off, nparts + 1, nparts, c, D,
                                                         counts, (uint2*)w->base.p);
    else
        k_digits_batch<<<div_up(cap, 256), 256, 0, st>>>((const uint8_t*)w->scal.p, off, nmsm, (uint32_t)b->n, c, D,
                                                        (uint32_t)cap, (uint32_t*)w->digits.p,
                                                        (uint32_t*)w->ranks.p, (uint32_t*)w->pidx.p, counts);
    k_scan_local<<<nblocks, 1024, 0, st>>>(counts, offsets, (uint32_t*)w->bsums.p, (uint32_t)M);
    k_scan_top<<<1, 1024, 0, st>>>((uint32_t*)w->bsums.p, nblocks, total);
    k_scan_add<<<div_up(M, 256), 256, 0, st>>>(offsets, (uint32_t*)w->bsums.p, (uint32_t)M);
    if (parts)
        k_part_scatter<<<pgrid, kPartThreads, part_smem(c, D), st>>>((const uint8_t*)w->scal.p, off, nparts + 1,
                                                                     nparts, (uint32_t)b->n, c, D,
                                                                     (const uint2*)w->base.p, offsets, sorted_pt,
                                                                     sorted_key);
    else
        k_scatter_batch<<<div_up(nD, 256), 256, 0, st>>>((const uint32_t*)w->digits.p, (const uint32_t*)w->ranks.p,
                                                        (const uint32_t*)w->pidx.p, offsets, off, nmsm, D,
                                                        (uint32_t)nD, sorted_pt, sorted_key);
    int aff_launches = 0;
    if (rounds)
        CATMSM_CHECK(aff_accumulate(w->aff, b->table.p, sorted_pt, sorted_key, total, msm_affine_min_entries(rounds), L,
                                    chunks, rounds, buckets, head, tail, st, &aff_launches));
    else
        k_accumulate<<<div_up(chunks, 128), 128, 0, st>>>((const affine*)b->table.p, sorted_pt, sorted_key, total,
                                                          0xffffffffu, L, buckets, head, tail);
    k_fixup_seg<<<div_up(chunks, 128), 128, 0, st>>>(sorted_key, total, L, head);
    k_fixup_join<<<div_up(chunks, 128), 128, 0, st>>>(sorted_key, offsets, total, L, buckets,
                                                      head, tail, hot_list, hot_count);
    k_fixup_hot_seg<<<2 * device_sms(), 128, 0, st>>>(hot_list, hot_count, offsets, L, buckets, head, tail);
    fixup_giants(hot_list, hot_count, offsets, L, buckets, head, tail, true, st);
    xyzz* bufA[2] = {seg, seg + 2 * lvl1};
    xyzz* bufQ[2] = {seg + lvl1, seg + 2 * lvl1 + lvl2};
    const xyzz* inA = buckets;
    const xyzz* inQ = nullptr;
    // digits .. fixup giants (11) and batch_out
    uint32_t m = B, pp = 0, launches = rounds ? 11 + (uint32_t)aff_launches : 12;
    bool first = true;
    while (m > 1) {
        launches++;
        if (!first && m <= msm_reduce_tail_max(nmsm)) {
            msm_reduce_tail(inA, inQ, m, nmsm, bufQ[pp], st);
            inQ = bufQ[pp];
            break;
        }
        const uint32_t F = first ? 8 : 2;
        const uint32_t m_out = (m + F - 1) / F;
        if (first)
            msm_reduce_level(inA, m, F, nmsm, route.dense, bufA[pp], bufQ[pp], st);
        else
            msm_reduce_pair(inA, inQ, m, nmsm, bufA[pp], bufQ[pp], st);
        inA = bufA[pp];
        inQ = bufQ[pp];
        pp ^= 1;
        m = m_out;
        first = false;
    }
    k_batch_out<<<div_up(nmsm, 128), 128, 0, st>>>(inQ ? inQ : inA, nmsm, (jac*)w->out.p);
    *kernels = launches;
    return cudaGetLastError();
}

// Captures enqueue_batch as one of w->graph's.  The capture is ended whatever fails.
static cudaError_t capture_batch(const Basis* b, BatchWork* w, cudaStream_t st, uint32_t nmsm, size_t cap,
                                 BatchRoute route)
{
    BatchGraph& g = w->graph;
    if (!w->graph_fits(b, nmsm) || g.cap != cap) {
        w->drop_graph();
        g.nmsm = nmsm;
        g.c = b->c;
        g.L = b->L;
        g.moves = w->moves();
        g.cap = cap;
    }
    CATMSM_CHECK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    uint32_t kernels = 0;
    const cudaError_t queued = enqueue_batch(b, w, st, nmsm, cap, route, &kernels);
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaError_t e = cudaStreamEndCapture(st, &graph);
    if (queued != cudaSuccess) e = queued;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    CATMSM_CHECK(e);
    g.exec[route.kind()] = exec;
    return cudaSuccess;
}

// H2D of the batch's scalars.  Page-locked caller memory is read in place (run_batch
// waits for the stream, also after a failure); anything else goes through pinned staging, by
// several host threads (a copy of 44 MB: ~1 ms of a 14 ms batch).
static cudaError_t copy_scalars(BatchWork* w, const uint8_t* scalars, size_t bytes, cudaStream_t st)
{
    if (bytes == 0) return cudaSuccess;
    bool pinned = true;
    for (const uint8_t* p : {scalars, scalars + bytes - 1}) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess || at.type != cudaMemoryTypeHost) pinned = false;
    }
    cudaGetLastError();
    if (pinned) {
        if (cudaMemcpyAsync(w->scal.p, scalars, bytes, cudaMemcpyHostToDevice, st) == cudaSuccess) return cudaSuccess;
        cudaGetLastError();              // not one page-locked range after all
    }
    if (!w->h_scal.get(bytes)) return cudaErrorMemoryAllocation;
    host_copy(w->h_scal.p, scalars, bytes);
    return cudaMemcpyAsync(w->scal.p, w->h_scal.p, bytes, cudaMemcpyHostToDevice, st);
}

// Queues the copies of a batch (`bytes` of scalars, np parts) and its device sequence.
static cudaError_t queue_batch(const Basis* b, BatchWork* w, cudaStream_t st, uint32_t nmsm, size_t cap,
                               BatchRoute route, const uint8_t* scalars, size_t bytes, uint32_t np, bool use_graph)
{
    CATMSM_CHECK(copy_scalars(w, scalars, bytes, st));
    CATMSM_CHECK(cudaMemcpyAsync(w->off.p, w->h_off.p, (nmsm + 2 + 2 * (size_t)np) * 4, cudaMemcpyHostToDevice, st));
    if (use_graph) {
        const BatchGraph& g = w->graph;
        if (!w->graph_fits(b, nmsm) || g.cap != cap || !g.exec[route.kind()])
            CATMSM_CHECK(capture_batch(b, w, st, nmsm, cap, route));
        CATMSM_CHECK(cudaGraphLaunch(g.exec[route.kind()], st));
        g_stats.launches += 1;
    } else {
        uint32_t kernels = 0;
        CATMSM_CHECK(enqueue_batch(b, w, st, nmsm, cap, route, &kernels));
        g_stats.launches += kernels;
    }
    CATMSM_CHECK(cudaGetLastError());
    return cudaMemcpyAsync(w->h_out.p, w->out.p, (size_t)nmsm * sizeof(jac), cudaMemcpyDeviceToHost, st);
}

// rounds false: no affine rounds, whatever the entries (their memory is not to be had).
// exact_cap: size the work for exactly the pairs of this batch (serving);
// otherwise for its pairs rounded up to a sixteenth of full-basis MSMs, or for
// the captured graph's if they fit it, so one graph serves batches of one size.
static cudaError_t run_batch(Basis* b, BatchWork* w, cudaStream_t st, blst_p1* out, uint32_t nmsm,
                             const size_t* counts, const uint8_t* scalars, bool use_graph, bool exact_cap,
                             bool rounds = true)
{
    if (!b->tables) return cudaErrorMemoryAllocation;
    size_t P = 0;
    for (uint32_t j = 0; j < nmsm; j++) {
        if (counts[j] > b->n) return cudaErrorInvalidValue;
        P += counts[j];
    }
    const size_t full = (size_t)nmsm * b->n;
    if ((exact_cap ? P : full) * b->D >= 0x7fffffffu) return cudaErrorInvalidValue;
    size_t cap = P ? P : 1;
    if (!exact_cap) {
        const size_t step = (full + 15) / 16;
        cap = std::min(full, (P / step + 1) * step);
        if (use_graph && w->graph_fits(b, nmsm) && w->graph.cap >= P) cap = w->graph.cap;
    }
    BatchRoute route;
    route.parts = part_sort(b, P * b->D);
    route.dense = P * b->D >= 2 * ((size_t)nmsm << (b->c - 1));
    CATMSM_CHECK(ensure_work(b, w, nmsm, cap, route.parts));
    uint32_t* off = (uint32_t*)w->h_off.p;
    uint32_t* parts = off + nmsm + 2;
    uint32_t np = 0, f = 0;
    for (uint32_t j = 0; j < nmsm; j++) {
        off[j] = f;
        for (uint32_t i = 0; i < counts[j]; i += kPartPairs) {
            parts[2 * np] = j;
            parts[2 * np + 1] = f + i;
            np++;
        }
        f += (uint32_t)counts[j];
    }
    off[nmsm] = f;
    off[nmsm + 1] = np;
    // Batch-affine rounds by the entries this batch holds (the plain MSM's rule;
    // 1024 MSMs, 33 M entries, 32 a bucket: 15.4 ms without, 14.1 with).  Without
    // the memory for their lists the batch keeps the mixed additions.
    if (rounds)
        route.rounds = std::min(msm_affine_rounds(P * b->D, (size_t)nmsm << (b->c - 1)), BatchGraph::kMaxRounds);
    if (route.rounds && aff_prepare(w->aff, b->L, (cap * b->D + b->L - 1) / b->L + 1, st) != cudaSuccess) {
        cudaGetLastError();
        route.rounds = 0;
    }
    cudaError_t err = queue_batch(b, w, st, nmsm, cap, route, scalars, P * 32, np, use_graph);
    if (err != cudaSuccess && w->aff.aux.stream) cudaStreamSynchronize(w->aff.aux.stream);
    const cudaError_t done = cudaStreamSynchronize(st);      // the caller's scalars are not read after return
    if (err == cudaSuccess) err = done;
    if (err == cudaSuccess) std::memcpy(out, w->h_out.p, (size_t)nmsm * sizeof(jac));
    else cudaGetLastError();                                 // err reports it
    return err;
}

BatchWork* batch_work_new() { return new (std::nothrow) BatchWork(); }

void batch_work_free(BatchWork* w)
{
    if (!w) return;
    w->release();
    delete w;
}

cudaError_t batch_run(Basis* b, BatchWork* w, cudaStream_t st, blst_p1* out, uint32_t nmsm, const size_t* counts,
                      const uint8_t* scalars, bool rounds)
{
    return run_batch(b, w, st, out, nmsm, counts, scalars, false, true, rounds);
}

size_t basis_points(const Basis* b) { return b->n; }
uint32_t basis_window(const Basis* b) { return b->c; }
int basis_device(const Basis* b) { return b->device; }
const void* basis_points_device(const Basis* b) { return b->points.p; }

// ---------------------------------------------------------------- autotune cache
static std::mutex g_tune_mu;

static std::string tune_path()
{
    const char* p = std::getenv("CATMSM_TUNE_CACHE");
    if (p && *p) return p;
    const char* home = std::getenv("HOME");
    return std::string(home && *home ? home : "/tmp") + "/.cache/catmsm_tune.txt";
}

static std::string tune_key(size_t n, uint32_t nmsm, size_t pairs)
{
    char name[256] = "gpu";
    cudaDeviceProp prop;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaGetDeviceProperties(&prop, dev) == cudaSuccess)
        std::snprintf(name, sizeof(name), "%s", prop.name);
    for (char* q = name; *q; q++)
        if (*q == ' ') *q = '_';
    // points-per-MSM class: log2 of the mean, rounded
    const double mean = nmsm ? (double)pairs / nmsm : 0;
    int cls = 0;
    while ((double)(1u << (cls + 1)) <= mean) cls++;
    char key[384];
    std::snprintf(key, sizeof(key), "%s n=%zu nmsm=%u mean2^%d", name, n, nmsm, cls);
    return key;
}

static bool tune_lookup(const std::string& key, uint32_t* c, uint32_t* L)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    FILE* f = std::fopen(tune_path().c_str(), "r");
    if (!f) return false;
    char line[512];
    bool found = false;
    while (std::fgets(line, sizeof(line), f)) {
        char* bar = std::strchr(line, '|');
        if (!bar) continue;
        *bar = 0;
        unsigned cc = 0, ll = 0;
        if (key == line && std::sscanf(bar + 1, "%u %u", &cc, &ll) == 2) {
            *c = cc;
            *L = ll;
            found = true;
        }
    }
    std::fclose(f);
    return found;
}

static void tune_store(const std::string& key, uint32_t c, uint32_t L)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    const std::string path = tune_path();
    for (size_t pos = path.find('/', 1); pos != std::string::npos; pos = path.find('/', pos + 1))
        mkdir(path.substr(0, pos).c_str(), 0755);    // existing directories are fine
    FILE* f = std::fopen(path.c_str(), "a");
    if (!f) return;
    std::fprintf(f, "%s|%u %u\n", key.c_str(), c, L);
    std::fclose(f);
}

}  // namespace catmsm

using namespace catmsm;

extern "C" {

void* catmsm_basis_create(const blst_p1_affine* points, size_t n, size_t window)
{
    if (!points || n == 0 || n > (1u << 24) || window > 20 || (window != 0 && window < 2)) return nullptr;
    Basis* b = new (std::nothrow) Basis();
    if (!b) return nullptr;
    if (cudaGetDevice(&b->device) != cudaSuccess || msm_setup_device() != cudaSuccess ||
        cudaFuncSetAttribute(k_part_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPartMaxSmem) !=
            cudaSuccess ||
        cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete b;
        return nullptr;
    }
    b->n = n;
    void* dp = b->points.get(n * sizeof(affine));
    if (!dp || cudaMemcpy(dp, points, n * sizeof(affine), cudaMemcpyHostToDevice) != cudaSuccess ||
        build_tables(b, window ? (uint32_t)window : 11) != cudaSuccess) {
        catmsm_basis_destroy(b);
        return nullptr;
    }
    return b;
}

void catmsm_basis_destroy(void* handle)
{
    Basis* b = (Basis*)handle;
    if (!b) return;
    b->work.release();
    b->points.release();
    b->table.release();
    b->tmp.release();
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

int catmsm_basis_config(void* handle, size_t* window, size_t* chunk)
{
    Basis* b = (Basis*)handle;
    if (!b) return (int)cudaErrorInvalidValue;
    std::lock_guard<std::mutex> lk(b->mu);
    if (window) *window = b->c;
    if (chunk) *chunk = b->L;
    return 0;
}

// catmsm_basis_set_config with b->mu held by the caller.
static int set_config_locked(Basis* b, size_t window, size_t chunk)
{
    if (window < 2 || window > 20 || chunk < 2 || chunk > 256) return (int)cudaErrorInvalidValue;
    b->L = (uint32_t)chunk;
    if (window != b->c || !b->tables) return (int)build_tables(b, (uint32_t)window);
    return 0;
}

int catmsm_basis_set_config(void* handle, size_t window, size_t chunk)
{
    Basis* b = (Basis*)handle;
    if (!b) return (int)cudaErrorInvalidValue;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return (int)cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(b->mu);
    return set_config_locked(b, window, chunk);
}

int catmsm_basis_msm_batch(void* handle, blst_p1* out, size_t nmsm, const size_t* counts, const blst_byte* scalars,
                           int use_graph)
{
    Basis* b = (Basis*)handle;
    if (!b || !out || !counts || (!scalars && nmsm) || nmsm == 0 || nmsm > (1u << 20)) return (int)cudaErrorInvalidValue;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return (int)cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(b->mu);
    return (int)run_batch(b, &b->work, b->stream, out, (uint32_t)nmsm, counts, scalars, use_graph != 0, false);
}

int catmsm_basis_autotune(void* handle, size_t nmsm, const size_t* counts, const blst_byte* scalars, int force)
{
    Basis* b = (Basis*)handle;
    if (!b || !counts || !scalars || nmsm == 0) return (int)cudaErrorInvalidValue;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return (int)cudaErrorInvalidDevice;
    size_t pairs = 0;
    for (size_t j = 0; j < nmsm; j++) pairs += counts[j];
    const std::string key = tune_key(b->n, (uint32_t)nmsm, pairs);
    uint32_t c = 0, L = 0;
    std::lock_guard<std::mutex> lk(b->mu);       // the whole sweep: it reconfigures and runs the basis
    if (!force && tune_lookup(key, &c, &L)) return set_config_locked(b, c, L);
    std::vector<blst_p1> out(nmsm);
    cudaEvent_t e0, e1;
    CATMSM_CHECK(cudaEventCreate(&e0));
    CATMSM_CHECK(cudaEventCreate(&e1));
    float best = 1e30f;
    uint32_t bc = b->c, bl = b->L;
    const uint32_t cs[] = {9, 10, 11, 12, 13};
    const uint32_t ls[] = {8, 16, 32, 48, 64, 96, 128, 192, 256};   // chunk lengths (96 measured best at 1024 x ~1.4k)
    for (uint32_t cc : cs) {
        for (uint32_t ll : ls) {
            if (set_config_locked(b, cc, ll) != 0) continue;
            if (run_batch(b, &b->work, b->stream, out.data(), (uint32_t)nmsm, counts, scalars, true, false) !=
                cudaSuccess)
                continue;
            float tot = 0.f;
            for (int r = 0; r < 2; r++) {
                cudaEventRecord(e0, b->stream);
                if (run_batch(b, &b->work, b->stream, out.data(), (uint32_t)nmsm, counts, scalars, true, false) !=
                    cudaSuccess)
                    break;
                cudaEventRecord(e1, b->stream);
                cudaEventSynchronize(e1);
                float ms = 0.f;
                cudaEventElapsedTime(&ms, e0, e1);
                tot += ms;
            }
            if (tot < best) {
                best = tot;
                bc = cc;
                bl = ll;
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    int rc = set_config_locked(b, bc, bl);
    if (rc == 0) tune_store(key, bc, bl);
    return rc;
}

}  // extern "C"
