// The MSM of few points (the plain commitment, small aggregates) as two or three
// launches: signed points and scalar halves, the buckets of every window, and
// the last reduction levels.
//
// What bounds a small MSM is latency: the general pipeline's sort, accumulate,
// fixup and reduce are 12 launches whose chains of dependent point additions
// (5 us each) follow one another.  Here a block owns a range of one window's
// buckets and keeps everything in shared memory:
//   digits   k + sum_w 2^(c w + c - 1) has the signed window digits as plain bit
//            fields (each minus 2^(c - 1)), so a block reads its window's digit of
//            every scalar without the windows below;
//   lists    counting sort of the block's entries by bucket (two passes over the
//            scalars, from the L2);
//   sums     about 368 threads, each with up to L entries of ONE bucket (a bucket of
//            m entries gets ceil(m / L) threads, so one hot bucket still uses them all),
//            then a quad tree over each bucket's threads.
//            A block with too many entries (small_limit; equal scalars: all of a
//            window in one block) raises a flag, the others leave before their sums,
//            and the general pipeline, which spreads a bucket over the whole GPU, runs
//            instead, on the split that is there already;
//   reduce   sum_b (b + 1) S_b of the range by binary (A, Q) levels (the rule of
//            the general reduction), the ranges of a window by k_reduce_tail.
#define CATMSM_INLINE_SQR   // see field.cuh
#define CATMSM_INLINE_MUL2  // see field.cuh
#include "common.cuh"
#include "curve.cuh"
#include "fr.cuh"
#include "scalar.cuh"
#include "catmsm_internal.h"

#include <algorithm>

namespace catmsm {

constexpr size_t kSmallMaxPoints = 24576;      // pipeline points (12288 points of 255-bit scalars)
constexpr size_t kSmallMaxPlain = 3072;        // without the GLV split
constexpr uint32_t kSmallNarrow = 512;         // up to this many: 4-bit windows, one block a window
constexpr uint32_t kSmallThreads = 512;
constexpr uint32_t kSmallSums = 368;           // threads with entries, before one more per bucket
constexpr uint32_t kSmallMaxR = 16;            // buckets per block
// Most entries of a block, and of one bucket: see small_limit.
constexpr uint32_t kSmallAny = 2048, kSmallDense = 5400, kSmallHot = 3600, kSmallMaxBucket = 4000;

// Measured against the general pipeline (host call, us): 255 bits 64 points 170 / 308,
// 4096 306 / 405, 12288 497 / 521, 16384 611 / 553; 64 bits 2048 points 237 / 348,
// 4096 291 / 351, 8192 387 / 368; 100 bits (a narrow top window: one hot
// block) 2048 points 302 / 347, 4096 395 / 360.
bool msm_small_applies(size_t pipeline_points, bool glv)
{
    return pipeline_points >= 1 && pipeline_points <= (glv ? kSmallMaxPoints : kSmallMaxPlain);
}

// 4-bit windows: 8 buckets, so the reduction is 3 levels, for 32 window sums to
// fold on the host; 8-bit windows: 128 buckets in 8 ranges of 16, one
// range a block.  512 points of 255 bits: 236 us with 4 bits, 216 with 8; 200 points 199, 206.
uint32_t msm_small_window(size_t pipeline_points) { return pipeline_points <= kSmallNarrow ? 4 : 8; }

// k + bias needs c D bits: the GLV halves stay below 2^126.5, other scalars
// of c D - 1 bits take one window more.
uint32_t msm_small_windows(size_t pipeline_points, uint32_t bits, bool glv)
{
    const uint32_t c = msm_small_window(pipeline_points);
    return bits / c + 1 + (!glv && (bits + 1) % c == 0 ? 1 : 0);
}

// The signed points and magnitudes of the GLV split, as k_glv_scalars and
// k_glv_points; thread i < n writes s1 P_i, thread n + i s2 phi(P_i).
__global__ void __launch_bounds__(128) k_small_glv(const uint8_t* __restrict__ scalars, uint32_t stride, uint32_t n,
                                                   uint32_t nbits, const affine* __restrict__ pts,
                                                   uint4* __restrict__ mag, affine* __restrict__ gpts,
                                                   uint32_t* __restrict__ stop)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * n) return;
    if (t == 0) *stop = 0;
    const uint32_t i = t < n ? t : t - n;
    uint32_t k[8], m1[4], m2[4];
    bool s1, s2;
    load_scalar(k, scalars + (size_t)i * stride, stride, nbits);
    fr_glv_balanced(m1, m2, s1, s2, k);
    affine p;
    load_affine(p.x, p.y, pts + i);
    const bool inf = aff_is_inf(p);
    if (t >= n) {
        fp beta;
#pragma unroll
        for (int w = 0; w < 12; w++) beta.v[w] = FP_BETA[w];
        fp_mul(p.x, p.x, beta);
        fp_canon(p.x, p.x);
    }
    if (!inf && (t < n ? s1 : s2)) fp_neg(p.y, p.y);
    store_affine(gpts + t, p);
    mag[t] = t < n ? make_uint4(m1[0], m1[1], m1[2], m1[3]) : make_uint4(m2[0], m2[1], m2[2], m2[3]);
}

// Scalars of at most 128 bits as 16-byte magnitudes (no split).
__global__ void __launch_bounds__(128) k_small_scalars(const uint8_t* __restrict__ scalars, uint32_t stride, uint32_t n,
                                                       uint32_t nbits, uint4* __restrict__ mag,
                                                       uint32_t* __restrict__ stop)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0) *stop = 0;
    uint32_t k[8];
    load_scalar(k, scalars + (size_t)i * stride, stride, nbits);
    mag[i] = make_uint4(k[0], k[1], k[2], k[3]);
}

struct SmallArgs {
    const affine* pts;
    const uint4* mag;
    uint32_t n, c, nb, R;       // pipeline points, window, ranges per window, buckets per range
    uint32_t bias[5];           // sum over the windows of 2^(c w + c - 1)
    xyzz* outA;                 // per (window, range): 2^log2(R) S, null with one range
    xyzz* outQ;                 // per (window, range): sum (b + 1) S_b
    uint32_t* entries;          // counter of nonzero digits, or null
    uint32_t* stop;             // set when a block has too many entries (zeroed by the kernel before)
    uint32_t* over;             // page-locked: the same for the host
};

// Signed digit of window w (bits [c w, c w + c) of k + bias, minus 2^(c - 1)).
__device__ __forceinline__ int32_t small_digit(const uint4& k, const SmallArgs& A, uint32_t w)
{
    uint32_t v[6];
    uint64_t s = (uint64_t)k.x + A.bias[0];
    v[0] = (uint32_t)s;
    s = (s >> 32) + k.y + A.bias[1];
    v[1] = (uint32_t)s;
    s = (s >> 32) + k.z + A.bias[2];
    v[2] = (uint32_t)s;
    s = (s >> 32) + k.w + A.bias[3];
    v[3] = (uint32_t)s;
    v[4] = (uint32_t)(s >> 32) + A.bias[4];
    v[5] = 0;
    const uint32_t bit = w * A.c, word = bit >> 5;
    uint32_t lo = v[0], hi = v[1];
#pragma unroll
    for (uint32_t j = 1; j < 5; j++)
        if (word == j) {
            lo = v[j];
            hi = v[j + 1];
        }
    const uint32_t raw = __funnelshift_r(lo, hi, bit & 31) & ((1u << A.c) - 1);
    return (int32_t)raw - (int32_t)(1u << (A.c - 1));
}

// The most entries of a block for which the small kernel runs, out of W of its window:
// kSmallAny; twice its even share, up to kSmallDense; or, if it has most of the window (0/1
// vectors, the carries of short scalars: where the general pipeline has little to do
// elsewhere), 9/40 of the points up to kSmallHot.  Above, the general pipeline is faster although the attempt
// comes before it (about 15 us).  The top window of uniform GLV halves, below 2^126.4, has
// 1.49 shares in a block.  Small kernel against general pipeline, us: 6000 points, 43%
// ones (2580 entries) 289 / 322; 8192, 43% (3522) 330 / 362; 12288, 43% (5284) 432 / 350; 6000, a
// quarter ones and the rest random (1.75 shares) 388 / 470; 10000 scalars of 127 bits (1.8) 494 / 554, 12288 (1.8,
// 5542 entries) 556 / 509.
__device__ __forceinline__ uint32_t small_limit(uint32_t s, uint32_t W, const SmallArgs& A)
{
    return max(kSmallAny, 2 * s > W ? min(A.n * 9 / 40, kSmallHot) : min(2 * ((A.n + A.nb - 1) / A.nb), kSmallDense));
}

constexpr uint32_t kSmallAcc = kSmallSums + kSmallMaxR;
constexpr size_t kSmallFixed = (kSmallAcc + 3 * kSmallMaxR) * sizeof(xyzz);

__global__ void __launch_bounds__(kSmallThreads) k_small_buckets(SmallArgs A)
{
    extern __shared__ __align__(16) unsigned char small_smem[];
    xyzz* acc = reinterpret_cast<xyzz*>(small_smem);          // a partial sum per thread
    xyzz* lev = acc + kSmallAcc;                              // bucket sums, then (Q | A) of the levels
    uint32_t* list = reinterpret_cast<uint32_t*>(lev + 3 * kSmallMaxR);
    __shared__ uint32_t cnt[kSmallMaxR], start[kSmallMaxR + 1], ts[kSmallMaxR + 1], shape[4], W;
    const uint32_t tid = threadIdx.x, R = A.R;
    const uint32_t w = blockIdx.x / A.nb, b0 = blockIdx.x % A.nb * R;
    if (tid < kSmallMaxR) cnt[tid] = 0;
    if (tid == 0) W = 0;
    __syncthreads();
    uint32_t nonzero = 0;
    for (uint32_t i = tid; i < A.n; i += blockDim.x) {
        const int32_t d = small_digit(__ldg(A.mag + i), A, w);
        const uint32_t b = (uint32_t)(d < 0 ? -d : d) - 1 - b0;          // d = 0 wraps past R
        nonzero += d != 0;
        if (d != 0 && b < R && atomicAdd(&cnt[b], 1u) == kSmallMaxBucket) {      // one bucket is too many already
            *(volatile uint32_t*)A.stop = 1;
            *A.over = 1;
        }
    }
    nonzero = __reduce_add_sync(0xffffffffu, nonzero);
    if ((tid & 31) == 0) atomicAdd(&W, nonzero);
    __syncthreads();
    if (tid == 0) {
        uint32_t s = 0;
        for (uint32_t b = 0; b < R; b++) {
            start[b] = s;
            s += cnt[b];
            cnt[b] = start[b];
        }
        start[R] = s;
        const uint32_t L = max(1u, (s + kSmallSums - 1) / kSmallSums);
        uint32_t t = 0, most = 0;
        for (uint32_t b = 0; b < R; b++) {
            ts[b] = t;
            const uint32_t m = (start[b + 1] - start[b] + L - 1) / L;
            most = max(most, m);
            t += m;
        }
        ts[R] = t;
        shape[0] = L;
        shape[1] = most;
        shape[2] = s > small_limit(s, W, A);
        if (shape[2]) {
            *(volatile uint32_t*)A.stop = 1;
            *A.over = 1;
        }
        if (*(volatile uint32_t*)A.stop) shape[2] = 1;
        if (A.entries) atomicAdd(A.entries, s);
    }
    __syncthreads();
    if (shape[2]) return;                     // the caller runs the general pipeline

    for (uint32_t i = tid; i < A.n; i += blockDim.x) {
        const int32_t d = small_digit(__ldg(A.mag + i), A, w);
        const uint32_t b = (uint32_t)(d < 0 ? -d : d) - 1 - b0;
        if (d != 0 && b < R) list[atomicAdd(&cnt[b], 1u)] = i | (d < 0 ? 0x80000000u : 0u);
    }
    // Some block has raised the flag: no sums here either.  A block that read it too early
    // computes in vain (its results are not used); nothing waits for it.
    if (tid == 0) shape[3] = *(volatile uint32_t*)A.stop;
    __syncthreads();
    if (shape[3]) return;
    if (tid < ts[R]) {
        uint32_t b = 0;
        while (ts[b + 1] <= tid) b++;
        const uint32_t L = shape[0];
        const uint32_t e0 = start[b] + (tid - ts[b]) * L, e1 = min(e0 + L, start[b + 1]);
        xyzz sum;
        xyzz_set_inf(sum);
#pragma unroll 1
        for (uint32_t e = e0; e < e1; e++) {
            const uint32_t v = list[e];
            fp x, y;
            load_affine(x, y, A.pts + (v & 0x7fffffffu));
            if (fp_is_zero_raw(x) && fp_is_zero_raw(y)) continue;
            if (v >> 31) fp_neg(y, y);
            xyzz_madd(sum, x, y);
        }
        store_xyzz(acc + tid, sum);
    }
    // each bucket's partial sums: partial 2 d s += partial 2 d s + d, quads.  The
    // quads of a warp look for their pairs first and add together: an addition
    // inside the search ran once per distinct bucket (30-80k cycles a level, not 10k).
    const quad_lane ql = quad_of(tid & 31);
    const uint32_t most = shape[1];
    for (uint32_t d = 1; d < most; d <<= 1) {
        __syncthreads();
        for (uint32_t p0 = tid >> 5 << 3;; p0 += blockDim.x >> 2) {
            uint32_t p = p0 + ((tid & 31) >> 2), b = 0;
#pragma unroll 1
            for (; b < R; b++) {
                const uint32_t m = ts[b + 1] - ts[b];
                const uint32_t pairs = m > d ? (m - d + 2 * d - 1) / (2 * d) : 0;
                if (p < pairs) break;
                p -= pairs;
            }
            __syncwarp();
            if (!__any_sync(0xffffffffu, b < R)) break;
            if (b < R) {
                xyzz* at = acc + ts[b] + 2 * d * p;
                fp s = qd_load(at, ql.k);
                qd_add(s, qd_load(at + d, ql.k), ql);
                qd_store(at, s, ql);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    // bucket sums: level 0 of the (A, Q) pairs, Q = A = S
    for (uint32_t i = tid; i < R * 12; i += blockDim.x) {
        const uint32_t b = i / 12;
        const uint4 v = ts[b + 1] > ts[b] ? reinterpret_cast<const uint4*>(acc + ts[b])[i % 12] : make_uint4(0, 0, 0, 0);
        reinterpret_cast<uint4*>(lev)[i] = v;
    }
    __syncthreads();
    // binary levels: node u: Q = A_1 + Q_0 + Q_1 (warp 0's quads), A = 2 (A_0 + A_1) (warp 1's)
    const xyzz* srcA = lev;
    const xyzz* srcQ = lev;
    xyzz* dst = lev + kSmallMaxR;
    for (uint32_t m = R; m > 1; m >>= 1) {
        const uint32_t u = (tid & 31) >> 2;
        const bool q_role = tid < 32;
        if (tid < 64 && u < m / 2 && (q_role || m > 2 || A.outA)) {
            fp s = qd_load((q_role ? srcQ : srcA) + 2 * u, ql.k);
            qd_add(s, qd_load(srcA + 2 * u + 1, ql.k), ql);
            if (q_role) qd_add(s, qd_load(srcQ + 2 * u + 1, ql.k), ql);
            else qd_dbl(s, ql);
            qd_store(dst + (q_role ? 0 : m / 2) + u, s, ql);
        }
        __syncthreads();
        srcQ = dst;
        srcA = dst + m / 2;
        dst = dst == lev + kSmallMaxR ? lev + 2 * kSmallMaxR : lev + kSmallMaxR;
    }
    if (tid < 4) qd_store(A.outQ + blockIdx.x, qd_load(srcQ, ql.k), ql);
    else if (tid < 8 && A.outA) qd_store(A.outA + blockIdx.x, qd_load(srcA, ql.k), ql);
}

cudaError_t msm_small_setup_device()
{
    return cudaFuncSetAttribute(k_small_buckets, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kSmallFixed + kSmallMaxPoints * 4));
}

cudaError_t msm_small(Ctx* ctx, const void* pts, const uint8_t* scalars, uint32_t stride, size_t n, uint32_t nbits,
                      bool glv, uint32_t* entries, SmallMsm& out)
{
    cudaStream_t st = ctx->stream;
    MsmWork& W = ctx->msm;
    const size_t np = glv ? 2 * n : n;
    const uint32_t bits = glv ? 127 : nbits;
    if (!msm_small_applies(np, glv) || bits > 128) return cudaErrorInvalidValue;
    SmallArgs A = {};
    A.n = (uint32_t)np;
    A.c = msm_small_window(np);
    const uint32_t D = msm_small_windows(np, bits, glv);
    A.nb = A.c == 4 ? 1 : D > 9 ? 8 : 16;       // 16 windows x 8 or 9 x 16 blocks: one on each of 152 SMs
    A.R = (1u << (A.c - 1)) / A.nb;
    for (uint32_t w = 0; w < D; w++) {
        const uint32_t bit = w * A.c + A.c - 1;
        A.bias[bit >> 5] |= 1u << (bit & 31);
    }
    uint4* mag = (uint4*)W.glv_sc.get(np * sizeof(uint4));
    affine* gpts = glv ? (affine*)W.glv_pts.get(np * sizeof(affine)) : nullptr;
    xyzz* seg = (xyzz*)W.seg.get((2 * (size_t)D * A.nb + 1) * sizeof(xyzz));
    xyzz* wins = (xyzz*)ctx->h_out.get((size_t)(D + 1) * sizeof(xyzz));
    if (!mag || (glv && !gpts) || !seg || !wins) return cudaErrorMemoryAllocation;
    A.stop = (uint32_t*)(seg + 2 * (size_t)D * A.nb);
    if (glv)
        k_small_glv<<<div_up(np, 64), 64, 0, st>>>(scalars, stride, (uint32_t)n, nbits, (const affine*)pts, mag, gpts,
                                                   A.stop);
    else
        k_small_scalars<<<div_up(np, 128), 128, 0, st>>>(scalars, stride, (uint32_t)n, nbits, mag, A.stop);
    A.pts = glv ? gpts : (const affine*)pts;
    A.mag = mag;
    A.entries = entries;
    A.over = (uint32_t*)(wins + D);
    *A.over = 0;
    A.outA = A.nb > 1 ? seg : nullptr;
    A.outQ = A.nb > 1 ? seg + (size_t)D * A.nb : wins;          // page-locked: written straight to the host
    k_small_buckets<<<D * A.nb, kSmallThreads, kSmallFixed + np * 4, st>>>(A);
    g_stats.launches += 2;
    if (A.nb > 1) {
        msm_reduce_tail(A.outA, A.outQ, A.nb, D, wins, st, A.stop);
        g_stats.launches++;
    }
    out.wins = (const uint64_t*)wins;
    out.over = A.over;
    out.D = D;
    out.c = A.c;
    return cudaGetLastError();
}

}  // namespace catmsm
