// BLS12-381 G1 group-valued FFT on sm_103a.
//
// Drop-in for blst_p1_fft / blst_p1_fft_with_domain /
// blst_p1_ifft_unscaled_with_domain (reference fft_c_api.cpp:51-103,
// fft/ctFft.h:32-124, fft/context.h:182-215).  The transform is the same
// radix-2 decimation-in-time network with the same root indexing
// (root j * n/len, or n - j * n/len when the inverse reads forward roots), so
// outputs equal the reference's for any root table the caller supplies.
//
// Device layout: the points of one or many transforms, concatenated, as XYZZ
// (192 B) between the passes; a job descriptor per transform.
//   k_bitrev_multi     Jacobian input -> XYZZ in bit-reversed order.
//   then passes over the levels, each chosen by fft_plan for the whole batch:
//   k_fft_stage_multi  one level, one lane per butterfly: n/2 scalar multiplications,
//                      one launch.  For sizes whose levels are a whole wave or less
//                      (2^16 points) and for more products than a pass may hold.
//   k_fft_items + k_fft_quarter + k_fft_combine  q levels at once.  Every output of
//                      a 2^q-point block is sum_m +- (root product) x_m; each product
//                      of a point by a root product is an item of its own
//                      ((4^q - 1) / 3 of them per block, all independent), and
//                      the combine adds them up.  A launch that does not fill the GPU
//                      lasts as long as ONE scalar multiplication (0.6 to 1.5
//                      ms), so small transforms take q = 3 and 4.  Products by roots a
//                      quarter of the circle apart are one product and a quarter
//                      turn, which costs a third: for q = 2 three products and a turn
//                      where two levels of butterflies have four, the least work
//                      for launches that fill the GPU (the multiply pipe bounds them).
//                      With turns against without: 2^14 points, inverse, 14.47 -> 11.52 ms,
//                      2^10 2.76 -> 2.66, 2^20 514 -> 414, 64 transforms of 2^10 .. 2^16
//                      581 -> 436 ms.
//   k_fft_finish_multi Jacobian, canonical coordinates.
// The inverse's 1/n scale is multiplied into the roots of a job's last pass.
// Each butterfly is ~1.5k Fp multiplications (~0.9M IMAD) against 768 bytes of
// traffic, so memory never binds.
#define CATMSM_INLINE_SQR   // see field.cuh
#define CATMSM_INLINE_MUL2   // see field.cuh
#include "common.cuh"
#include "curve.cuh"
#include "fr.cuh"
#include "glv_mult.cuh"
#include "catmsm_internal.h"

#include <algorithm>
#include <cstring>
#include <vector>

namespace catmsm {

__device__ __forceinline__ void load_jac(jac& p, const jac* src)
{
    const uint4* q = reinterpret_cast<const uint4*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&p);
#pragma unroll
    for (int k = 0; k < 9; k++) {
        uint4 v = q[k];
        d[4 * k] = v.x; d[4 * k + 1] = v.y; d[4 * k + 2] = v.z; d[4 * k + 3] = v.w;
    }
}

__device__ __forceinline__ void store_jac(jac* dst, const jac& p)
{
    uint4* q = reinterpret_cast<uint4*>(dst);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&p);
#pragma unroll
    for (int k = 0; k < 9; k++) q[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
}

// roots_mont: n Montgomery Fr (caller table); out: n x {k1[4], k2[4]}
__global__ void k_roots_prepare(const uint32_t* __restrict__ roots_mont, uint32_t n, uint32_t* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t m[8], c[8];
    for (int k = 0; k < 8; k++) m[k] = roots_mont[8 * i + k];
    fr_from_mont(c, m);
    fr_glv_split(out + 8 * i, out + 8 * i + 4, c);
}

// The scaled roots of a job's last level: out[j] = root(j) * scale, j < n / 2
// (root(j) = w^j, or entry n - j when the inverse reads forward roots), and
// out[n / 2] = scale, as GLV halves.
__global__ void k_roots_prepare_scaled(const uint32_t* __restrict__ roots_mont, const uint32_t* __restrict__ scale,
                                       uint32_t n, int inv_from_fwd, uint32_t* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n / 2) return;
    uint32_t m[8], c[8];
    for (int k = 0; k < 8; k++) m[k] = scale[k];
    if (i != 0 && i != n / 2) {
        const size_t idx = inv_from_fwd ? n - i : i;
        uint32_t r[8];
        for (int k = 0; k < 8; k++) r[k] = roots_mont[8 * idx + k];
        fr_mul(m, m, r);
    }
    fr_from_mont(c, m);
    fr_glv_split(out + 8 * (size_t)i, out + 8 * (size_t)i + 4, c);
}

// powers of a Montgomery root: out[i] = w^i (Montgomery)
__global__ void k_root_powers(const uint32_t* __restrict__ w, uint32_t n, uint32_t* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t b[8], o[8];
    for (int k = 0; k < 8; k++) b[k] = w[k];
    fr_pow_u32(o, b, i);
    for (int k = 0; k < 8; k++) out[8 * i + k] = o[k];
}

// A batch of transforms shares the launches of every pass.  Job descriptor:
struct FftJob {
    uint32_t val_off;    // first element of this transform in the values buffer
    uint32_t n, logn;
    uint32_t glv_off;    // first prepared root (8 words each); glv_off + n: the scaled roots of the last level
    int32_t inv_from_fwd;
    uint32_t xn;         // inputs [xn, n) are the identity: stage s runs only the
                         // min(xn, n / 2^s) groups holding a non-identity input
    const uint32_t* roots;   // the n Montgomery roots
    const uint32_t* scale;   // Montgomery scale of every output, or null
};

// thread t of a launch over per-job ranges: find the job whose range holds t
// (pre: exclusive prefix of the ranges, `cnt` entries; ids: job per entry)
__device__ __forceinline__ uint32_t find_range(const uint32_t* __restrict__ pre, uint32_t cnt, uint32_t t)
{
    uint32_t lo = 0, hi = cnt;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (pre[mid] <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void k_bitrev_multi(const jac* __restrict__ in, xyzz* __restrict__ out, const FftJob* __restrict__ jobs,
                               const uint32_t* __restrict__ pre, uint32_t njobs, uint32_t total)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const FftJob J = jobs[find_range(pre, njobs, t)];
    const uint32_t i = t - J.val_off;
    const uint32_t r = J.logn ? (__brev(i) >> (32 - J.logn)) : 0;
    jac p;
    load_jac(p, in + t);
    xyzz o;
    jac_to_xyzz(o, p);
    store_xyzz(out + J.val_off + r, o);
}

// Group g of a level with `groups` groups, `active` of them holding a
// non-identity input (bit-reversed positions: the bit reversals of
// 0 .. active - 1).
__device__ __forceinline__ uint32_t active_group(uint32_t g, uint32_t active, uint32_t groups)
{
    return active < groups ? __brev(g) >> (32 - (31 - __clz(groups))) : g;
}

// Stage `len` over every job with n >= len, one lane per butterfly.  lst: for
// this stage, pairs of (job id, exclusive prefix of n/2 butterflies), `cnt`
// entries.  Threads map first onto the non-trivial butterflies (j >= 1), then
// onto the j == 0 ones, so a warp rarely mixes the two.  MinBlocks: resident
// blocks per SM the registers are limited for.  4 (255 registers) is 3% faster
// while one wave holds the launch; above that, 6 (168 registers) shortens the
// last wave: 46080 butterflies 3.5 -> 3.1 ms a level.
template <int MinBlocks>
__global__ void __launch_bounds__(64, MinBlocks) k_fft_stage_multi(xyzz* __restrict__ a, const FftJob* __restrict__ jobs,
                                                        const uint32_t* __restrict__ lst_job,
                                                        const uint32_t* __restrict__ lst_pre, uint32_t cnt,
                                                        uint32_t total, uint32_t len, const uint32_t* __restrict__ glv)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const uint32_t e = find_range(lst_pre, cnt, t);
    const FftJob J = jobs[lst_job[e]];
    const uint32_t b = t - lst_pre[e];
    const uint32_t half = len >> 1;
    const uint32_t groups = J.n / len;
    const uint32_t active = min(groups, J.xn);
    const uint32_t nontriv = active * (half - 1);
    // Non-trivial butterflies: with at least 32 active groups (a multiple of
    // 32), the group index runs fastest, so the lanes of a warp share j and
    // its root and take the width-5 NAF multiplication; otherwise j runs
    // fastest and the lanes, on different roots, keep the fixed windows.
    uint32_t g, j;
    bool shared = false;
    if (b < nontriv) {
        if ((active & 31u) == 0) {
            j = 1 + b / active;
            g = b % active;
            shared = true;
        } else {
            g = b / (half - 1);
            j = 1 + b % (half - 1);
        }
    } else {
        g = b - nontriv;
        j = 0;
    }
    g = active_group(g, active, groups);
    xyzz* base = a + J.val_off;
    const uint32_t i0 = g * len + j, i1 = i0 + half;
    xyzz u, v;
    load_xyzz(v, base + i1);
    const bool scaled = J.scale && len == J.n;       // the job's last level: roots times the scale
    if (j || scaled) {
        uint32_t idx = J.n + j;
        if (!scaled) {
            idx = j * groups;
            if (J.inv_from_fwd) idx = J.n - idx;
        }
        const uint32_t* r = glv + 8 * (size_t)(J.glv_off + idx);
        if (shared) xyzz_mult_glv_shared(v, v, r, r + 4);
        else xyzz_mult_glv(v, v, r, r + 4);
    }
    load_xyzz(u, base + i0);
    if (scaled) {
        const uint32_t* r = glv + 8 * (size_t)(J.glv_off + J.n + half);
        xyzz_mult_glv_shared(u, u, r, r + 4);        // one scale per job, shared by its lanes
    }
    xyzz d;
    xyzz_add_sub(u, d, v);
    store_xyzz(base + i0, u);
    store_xyzz(base + i1, d);
}

// ---------------------------------------------------------------- q levels at once
// Levels s0 + 1 .. s0 + q of a job over its blocks of 2^q h positions (h =
// 2^s0): position j + m h (j < h) of a block holds x_m, and output k of the
// butterfly (block, j) is
//   sum_m (-1)^popc(m & k) C(m, k) x_m,
//   C = product over the set bits i of m of the root of level i at position
//       j + h (k mod 2^i) of its half-block.
// C depends on k only below m's top bit t, so the products of x_m are the 2^t
// items (m, k mod 2^t).  Item 0 is x_0 itself.  Item 1 + (4^t - 1) / 3 +
// (m - 2^t) 2^t + (k mod 2^t) is the product (m, k), so a butterfly has
// 1 + (4^q - 1) / 3 items.
__host__ __device__ __forceinline__ uint32_t pass_items(uint32_t q) { return 1 + ((1u << (2 * q)) - 1) / 3; }

__device__ __forceinline__ uint32_t item_of(uint32_t m, uint32_t k)
{
    if (m == 0) return 0;
    const uint32_t t = 31 - __clz(m), top = 1u << t;
    return 1 + (top * top - 1) / 3 + (m - top) * top + (k & (top - 1));
}

// A pass of one job: its q, blocks and butterflies.
struct PassGeom {
    uint32_t q, groups, active, bf;
};

__device__ __forceinline__ PassGeom pass_geom(const FftJob& J, uint32_t s0, uint32_t q)
{
    PassGeom g;
    g.q = min(q, J.logn - s0);
    g.groups = J.n >> (s0 + g.q);
    g.active = min(g.groups, J.xn);
    g.bf = g.active << s0;
    return g;
}

// Butterfly bf of a job's pass: block g (position-wise) and j < 2^s0.  With a
// multiple of 32 active blocks they run fastest, so the lanes of a warp share
// their roots (true is returned).
__device__ __forceinline__ bool pass_pos(const PassGeom& G, uint32_t s0, uint32_t bf, uint32_t& g, uint32_t& j)
{
    const bool shared = (G.active & 31u) == 0;
    g = active_group(shared ? bf % G.active : bf >> s0, G.active, G.groups);
    j = shared ? bf / G.active : bf & ((1u << s0) - 1);
    return shared;
}

__device__ __constant__ static const uint32_t FR_Z3[8] = {       // z^3 (Montgomery)
    0x55763050u, 0x0c4fa98au, 0x9ff7a200u, 0x4c8ea2c2u,
    0xe43b5ddfu, 0x649fca48u, 0xfc43f9d3u, 0x26c0c34du};

// Quarter turns.  z = -0xd201000000010000 is a 12th root of unity mod r, so the
// roots of order 4 are +-z^3, and z^3 P = |z| phi^2(P) costs 63 doublings and 5
// additions, about a third of a product.  In a table of powers the root of level
// t (from 0, t >= 1) at j + h (k + 2^(t - 1)), k < 2^(t - 1), is +-z^3 times its root at j + h k.
// So of the items with top bit t only those with k < 2^(t - 1) are multiplied, and
//   V = +-z^3 sum over those m of (-1)^popc(m & u) (item (m, k)),  u = k + 2^(t - 1),
// stands for all the items (m, u): 3, 11, 43 products and 1, 3, 7 quarter turns for q
// = 2, 3, 4 instead of 5, 21, 85 products.  The table is the caller's and may hold
// anything: each use compares the two roots, and without the relation the items are
// multiplied.
// Returns 0 (no relation), or +-1: the sign of z^3.
__device__ __forceinline__ int quarter_sign(const FftJob& J, uint32_t s0, uint32_t t, uint32_t pos)
{
    const uint32_t i2 = pos * (J.n >> (s0 + t + 1)), i3 = i2 + (J.n >> 2);   // i3 < n / 2
    uint32_t e[8], r[8];
    for (int w = 0; w < 8; w++) {
        e[w] = FR_Z3[w];
        r[w] = J.roots[8 * (size_t)(J.inv_from_fwd ? J.n - i3 : i3) + w];
    }
    if (pos) {
        uint32_t r2[8];
        for (int w = 0; w < 8; w++) r2[w] = J.roots[8 * (size_t)(J.inv_from_fwd ? J.n - i2 : i2) + w];
        fr_mul(e, e, r2);
    }
    uint32_t d = 0, s[8], z = 0;
    fr_add(s, e, r);
    for (int w = 0; w < 8; w++) {
        d |= e[w] ^ r[w];
        z |= s[w];
    }
    return d == 0 ? 1 : z == 0 ? -1 : 0;
}

// Product `it` of `items` in the order that a pass starts them.  With quarter turns:
// the ones that are multiplied, x_0 (multiplied if the pass scales), the ones a turn
// stands for; so the blocks with work come first and spread evenly over the SMs.
__host__ __device__ __forceinline__ void item_order(uint32_t it, uint32_t items, bool turns, uint32_t& m, uint32_t& k)
{
    const uint32_t x0 = turns ? items / 2 : items - 1;
    m = k = 0;
    if (it == x0) return;
    const bool late = it > x0;
    uint32_t rem = late ? it - x0 : it, top = 1, wide = 1;               // wide: the k of one m
    while (rem >= top * wide) {
        rem -= top * wide;
        top <<= 1;
        wide = turns ? top >> 1 : top;
    }
    m = top + rem / wide;
    k = rem % wide + (late ? wide : 0);
}

// The products of a pass: item-major per job (all items of one kind are
// adjacent, so trivial ones do not share warps with multiplications).  Lanes per
// item: 1, 2 (the pair form) or 4 (the quad form).  Split: the halves k1 x and
// k2 phi(x) of a product are two items (item 2 i + half), with half the additions
// each; the combine adds twice as many.
constexpr uint32_t kItemThreads = 64;

template <int Lanes, bool Split>
__global__ void __launch_bounds__(kItemThreads, Lanes == 2 ? 6 : 4)
k_fft_items(const xyzz* __restrict__ a, xyzz* __restrict__ prod, const FftJob* __restrict__ jobs,
            const uint32_t* __restrict__ lst_job, const uint32_t* __restrict__ lst_pre, uint32_t cnt, uint32_t total,
            uint32_t s0, uint32_t q, uint32_t turns)
{
    __shared__ __align__(16) unsigned char tabs[Lanes == 1   ? 16
                                                : Lanes == 2 ? kItemThreads / 2 * sizeof(pair_table)
                                                             : kItemThreads / 4 * sizeof(quad_table)];
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) / Lanes;
    if (t >= total) return;
    const uint32_t e = find_range(lst_pre, cnt, t);
    const FftJob J = jobs[lst_job[e]];
    const PassGeom G = pass_geom(J, s0, q);
    const uint32_t b = t - lst_pre[e];
    const uint32_t bf = b % G.bf, half = Split ? b / G.bf & 1 : 0;
    const uint32_t it = b / G.bf >> (Split ? 1 : 0);
    const uint32_t h = 1u << s0;
    uint32_t g, j, m, k;
    const bool shared = pass_pos(G, s0, bf, g, j);
    item_order(it, pass_items(G.q), turns != 0, m, k);
    xyzz* dst = prod + lst_pre[e] + (((size_t)item_of(m, k) << (Split ? 1 : 0)) + half) * G.bf + bf;
    if (turns && k) {
        const uint32_t top = 31 - __clz(m), turn = 1u << (top - 1);
        if ((k & turn) && quarter_sign(J, s0, top, j + h * (k - turn))) {    // k_fft_quarter writes V at m = 2^top
            if ((m != 2 * turn || half) && threadIdx.x % Lanes == 0) {
                xyzz o;
                xyzz_set_inf(o);
                store_xyzz(dst, o);
            }
            return;
        }
    }
    xyzz v;
    load_xyzz(v, a + J.val_off + ((size_t)g << (s0 + G.q)) + j + m * h);
    // the coefficient: Montgomery roots multiplied up (root 0 is never read:
    // a j = 0 butterfly has no multiplication)
    uint32_t c[8];
    bool one = true;
    if (J.scale && s0 + G.q == J.logn) {
        for (int w = 0; w < 8; w++) c[w] = J.scale[w];
        one = false;
    }
    for (uint32_t i = 0; i < G.q; i++) {
        if (!((m >> i) & 1u)) continue;
        const uint32_t pos = j + h * (k & ((1u << i) - 1));
        if (pos == 0) continue;
        uint32_t idx = pos * (J.n >> (s0 + i + 1));
        if (J.inv_from_fwd) idx = J.n - idx;
        uint32_t r[8];
        for (int w = 0; w < 8; w++) r[w] = J.roots[8 * (size_t)idx + w];
        if (one) {
            for (int w = 0; w < 8; w++) c[w] = r[w];
            one = false;
        } else {
            fr_mul(c, c, r);
        }
    }
    if (one) {
        if (half) xyzz_set_inf(v);
        if (threadIdx.x % Lanes == 0) store_xyzz(dst, v);
        return;
    }
    uint32_t kc[8], k12[8];
    fr_from_mont(kc, c);
    fr_glv_split(k12, k12 + 4, kc);
    if (Lanes == 1) {
        if (shared) xyzz_mult_glv_shared(v, v, k12, k12 + 4);
        else xyzz_mult_glv(v, v, k12, k12 + 4);
        store_xyzz(dst, v);
    } else if (Lanes == 2) {
        const pair_lane l{(threadIdx.x & 1) != 0, 3u << (threadIdx.x & 30)};
        fp lo, hi;
        pd_mult_glv(lo, hi, v, k12, k12 + 4, reinterpret_cast<pair_table*>(tabs) + threadIdx.x / 2, l);
        const quad_lane w0{l.odd ? 1u : 0u, 0}, w1{l.odd ? 3u : 2u, 0};     // the coordinates this lane holds
        qd_store(dst, lo, w0);
        qd_store(dst, hi, w1);
    } else {
        const quad_lane ql = quad_of(threadIdx.x & 31);
        if (half) {
            fp beta;
#pragma unroll
            for (int w = 0; w < 12; w++) beta.v[w] = FP_BETA[w];
            fp_mul(v.x, v.x, beta);
        }
        qd_store(dst, qd_mult_glv<Split>(v, half ? k12 + 4 : k12, k12 + 4,
                                              reinterpret_cast<quad_table*>(tabs) + threadIdx.x / 4, ql), ql);
    }
}

// The V of a pass: one lane or a quad per (butterfly, u), u < 2^(q - 1), u-major per
// job, which is half a job's outputs; u = 0, the last, has none.  A chain of 63
// doublings: a quad's lasts 0.25 ms up to two blocks per SM and 0.49 at 8192 turns, a lane's
// 0.60 at 16384 (2^16 points, q = 2), so quads take up to a wave of turns and lanes, with
// less work in all, the rest (1.3 waves, q = 3, a batch of 2^15, 2^6 and 2^2: 19.33 ms with
// quads, 19.20 with lanes).
template <bool Quad>
__global__ void __launch_bounds__(64, 4)
k_fft_quarter(xyzz* prod, const FftJob* __restrict__ jobs, const uint32_t* __restrict__ lst_job,
              const uint32_t* __restrict__ lst_pre, const uint32_t* __restrict__ lst_out, uint32_t cnt, uint32_t total,
              uint32_t s0, uint32_t q, uint32_t split)
{
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t t = Quad ? gt >> 2 : gt;
    if (t >= total) return;
    const uint32_t e = find_range(lst_out, cnt, 2 * t);
    const FftJob J = jobs[lst_job[e]];
    const PassGeom G = pass_geom(J, s0, q);
    const uint32_t b = t - lst_out[e] / 2;
    const uint32_t bf = b % G.bf, u = (1u << (G.q - 1)) - 1 - b / G.bf;
    if (u == 0) return;
    const uint32_t turn = 1u << (31 - __clz(u)), k = u - turn, top = 2 * turn;
    uint32_t g, j;
    pass_pos(G, s0, bf, g, j);
    const int sign = quarter_sign(J, s0, 32 - __clz(u), j + (k << s0));
    if (!sign) return;
    xyzz* p = prod + lst_pre[e] + bf;
    xyzz* dst = p + ((size_t)item_of(top, u) << split) * G.bf;
    fp b2;
#pragma unroll
    for (int w = 0; w < 12; w++) b2.v[w] = FP_BETA2[w];
    if (Quad) {
        const quad_lane ql = quad_of(threadIdx.x & 31);
        fp d;
        fp_zero(d);
#pragma unroll 1
        for (uint32_t i = 0; i < top << split; i++) {
            const uint32_t m = top + (i >> split);
            fp v = qd_load(p + (((size_t)item_of(m, k) << split) + (i & split)) * G.bf, ql.k);
            if (((__popc(m & u) & 1) != 0) != (sign < 0) && ql.k == 1) fp_neg(v, v);
            qd_add(d, v, ql);
        }
        const fp x = fp_mul_call(d, b2);
        d = fp_sel(d, x, ql.k == 0);
        const fp base = fp_swap(d, 2, ql);
        fp o;
        qd_times_abs_z(o, fp_sel(base, d, ql.k < 2), ql);
        const fp zz = fp_mul_call(o, d);                 // lanes 2, 3: back from the curve scaled by d's z
        qd_store(dst, fp_sel(o, zz, ql.k >= 2), ql);
    } else {
        xyzz d, v;
        xyzz_set_inf(d);
#pragma unroll 1
        for (uint32_t i = 0; i < top << split; i++) {
            const uint32_t m = top + (i >> split);
            load_xyzz(v, p + (((size_t)item_of(m, k) << split) + (i & split)) * G.bf);
            if (((__popc(m & u) & 1) != 0) != (sign < 0)) fp_neg(v.y, v.y);
            xyzz_add(d, v);
        }
        fp_mul(d.x, d.x, b2);
        jac o;
        times_abs_z(o, d.x, d.y);
        fp zz;
        fp_sqr(zz, o.z);
        fp_mul(d.zz, d.zz, zz);
        fp_mul(zz, zz, o.z);
        fp_mul(d.zzz, d.zzz, zz);
        d.x = o.x;
        d.y = o.y;
        store_xyzz(dst, d);
    }
}

// The sums of a pass: 4 * 2^(q - 1) lanes per output (twice that if split), each
// quad adds two products (the halves of one), then a tree over the output's quads.
__global__ void __launch_bounds__(128) k_fft_combine(const xyzz* __restrict__ prod, xyzz* __restrict__ a,
                                                     const FftJob* __restrict__ jobs,
                                                     const uint32_t* __restrict__ lst_job,
                                                     const uint32_t* __restrict__ lst_pre,
                                                     const uint32_t* __restrict__ lst_out, uint32_t cnt,
                                                     uint32_t total, uint32_t s0, uint32_t q, uint32_t split)
{
    const uint32_t lw = q + 1 + split;               // log2 of the lanes per output
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t o = gt >> lw;
    const bool valid = o < total;
    const quad_lane ql = quad_of(threadIdx.x & 31);
    const uint32_t qi = (gt & ((1u << lw) - 1)) >> 2;
    uint32_t dst = 0;
    fp acc;
    fp_zero(acc);
    if (valid) {
        const uint32_t e = find_range(lst_out, cnt, o);
        const FftJob J = jobs[lst_job[e]];
        const PassGeom G = pass_geom(J, s0, q);
        const uint32_t b = o - lst_out[e];
        const uint32_t k = b / G.bf, bf = b % G.bf;
        uint32_t g, j;
        pass_pos(G, s0, bf, g, j);
        dst = J.val_off + (g << (s0 + G.q)) + j + (k << s0);
        const xyzz* p = prod + lst_pre[e] + bf;
        if (2 * qi < (1u << (G.q + split))) {
            const uint32_t m0 = 2 * qi >> split, m1 = (2 * qi + 1) >> split;
            acc = qd_load(p + ((size_t)item_of(m0, k) << split) * G.bf, ql.k);
            fp v = qd_load(p + (((size_t)item_of(m1, k) << split) + split) * G.bf, ql.k);
            if ((__popc(m0 & k) & 1) && ql.k == 1) fp_neg(acc, acc);
            if ((__popc(m1 & k) & 1) && ql.k == 1) fp_neg(v, v);
            qd_add(acc, v, ql);
        }
    }
    for (uint32_t d = 4; d < (1u << lw); d <<= 1) {
        __syncwarp();
        fp v;
#pragma unroll
        for (int w = 0; w < 12; w++) v.v[w] = __shfl_down_sync(0xffffffffu, acc.v[w], d);
        if (((4 * qi) & (2 * d - 1)) == 0) qd_add(acc, v, ql);
    }
    if (valid && qi == 0) qd_store(a + dst, acc, ql);
}

// Jacobian with canonical coordinates; one-point jobs are scaled here (they
// have no pass).
__global__ void __launch_bounds__(64) k_fft_finish_multi(const xyzz* __restrict__ a, jac* __restrict__ out,
                                                         const FftJob* __restrict__ jobs,
                                                         const uint32_t* __restrict__ pre, uint32_t njobs,
                                                         uint32_t total)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const FftJob J = jobs[find_range(pre, njobs, t)];
    xyzz v;
    load_xyzz(v, a + t);
    if (J.logn == 0 && J.scale) {
        uint32_t c[8], kc[8], k12[8];
        for (int w = 0; w < 8; w++) c[w] = J.scale[w];
        fr_from_mont(kc, c);
        fr_glv_split(k12, k12 + 4, kc);
        xyzz_mult_plain(v, v, k12, k12 + 4);
    }
    jac o;
    xyzz_to_jac(o, v);
    fp_canon(o.x, o.x);
    fp_canon(o.y, o.y);
    fp_canon(o.z, o.z);
    store_jac(out + t, o);
}

// Scalar multiplications that run at once as quads (one wave of k_fft_items).
static size_t fft_quad_wave()
{
    static std::atomic<size_t> by_dev[64];          // shared by every calling thread
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) {
        const size_t v = by_dev[dev].load(std::memory_order_relaxed);
        if (v) return v;
    }
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (k_fft_items<4, false>), kItemThreads, 0);
    size_t v = (sms > 0 && per_sm > 0) ? (size_t)sms * per_sm * 16 : (size_t)device_sms() * 64;
    if (dev >= 0 && dev < 64) by_dev[dev].store(v, std::memory_order_relaxed);
    return v;
}

// One pass: levels s0 + 1 .. s0 + q.
struct FftPass {
    uint32_t s0 = 0, q = 1, group = 0;
    uint32_t split = 0, turns = 0;
    bool quad_turns = false;            // the turns by quads
    enum { kStage, kQuads, kPairs, kLanes } kind = kStage;
    uint32_t off = 0, cnt = 0;          // its entries of the job lists
    uint32_t items = 0, outputs = 0;
};

// Products of a butterfly of a pass that are multiplications: without x_0, items that
// quarter turns stand for and (first pass, j = 0 throughout) those without a root.
static size_t pass_products(uint32_t s0, uint32_t q, bool turns)
{
    size_t c = 0;
    for (uint32_t m = 1; m < (1u << q); m++) {
        const uint32_t top = 1u << (31 - __builtin_clz(m));
        for (uint32_t k = 0; k < (turns && top > 1 ? top / 2 : top); k++) {
            bool root = s0 != 0;
            for (uint32_t i = 1; i < q; i++) root |= ((m >> i) & 1u) && (k & ((1u << i) - 1));
            c += root;
        }
    }
    return c;
}

// Items, multiplications (without and with quarter turns) and outputs of a pass over
// every job that has its first level.
static void pass_counts(const std::vector<const FftJob*>& jobs, uint32_t s0, uint32_t q, size_t& items,
                        size_t products[2], size_t& outputs)
{
    items = products[0] = products[1] = outputs = 0;
    for (const FftJob* job : jobs) {
        const FftJob& J = *job;
        if (J.logn <= s0) continue;
        const uint32_t qe = std::min(q, J.logn - s0);
        const uint32_t groups = J.n >> (s0 + qe);
        const size_t bf = (size_t)std::min(groups, J.xn) << s0;
        items += bf * pass_items(qe);
        outputs += bf << qe;
        const bool scaled = J.scale && s0 + qe == J.logn;          // x_0 as well
        // a block with one non-identity input or none (a truncated prefix): that input is x_0
        const bool only_x0 = J.xn <= groups;
        for (int t = 0; t < 2; t++)
            products[t] += bf * ((only_x0 ? 0 : pass_products(s0, qe, t != 0)) + (scaled ? 1 : 0));
    }
}

// The cheapest sequence of passes by a model of their times (ms), fitted on
// GB300 (wave = 9728 quads, 4 blocks of 16 on each of 152 SMs; three waves' worth of
// pairs and four of lanes are resident at once).  Every form lasts one
// multiplication's latency as long as a warp has its scheduler to itself (quads
// 0.78 ms, the halves of a split product 0.64, pairs 0.99, lanes 1.5; a quarter
// turn by a quad 0.25), more when two share it, and adds up beyond a wave; a sum
// costs kSumMs per product.
static double quads_ms(size_t items, size_t wave, bool split)
{
    if (items <= wave / 2) return items == 0 ? 0.0 : split ? 0.64 : 0.78;
    return (split ? 0.83 : 1.0) * (double)((items + wave - 1) / wave);
}

static double pairs_ms(size_t items, size_t wave)
{
    const size_t rem = items % (3 * wave);
    return 2.03 * (double)(items / (3 * wave)) +
           (rem == 0 ? 0.0 : rem <= wave ? 0.99 : rem <= 3 * wave / 2 ? 1.32 : 2.03);
}

static double lanes_ms(size_t items, size_t wave)
{
    const size_t rem = items % (4 * wave);
    return 2.3 * (double)(items / (4 * wave)) + (rem == 0 ? 0.0 : rem <= 2 * wave ? 1.5 : 2.07);
}

static double quarter_ms(size_t turns, size_t wave)
{
    if (turns <= wave) return turns <= wave / 2 ? 0.26 : turns <= 7 * wave / 10 ? 0.34 : 0.49;
    return 0.62 + 0.8 * (double)(turns / (4 * wave));
}

static double stage_ms(size_t butterflies, size_t wave)
{
    if (butterflies <= 4 * wave) return lanes_ms(butterflies, wave);
    return 0.5 + 2.3 * (double)butterflies / (double)(4 * wave);
}

// Products of a pass of q levels: 50 MB; two levels, the form for large launches (1.5 products
// per output), 805 MB.  64 transforms of 2^10 .. 2^16 (1.4 M points): 110.1 transforms/s at
// one level a pass, 143.9 at two.
static size_t pass_max_items(uint32_t q) { return size_t(1) << (q <= 2 ? 22 : 18); }

// Next to another group of jobs (not solo) the launches share the GPU: there a pass
// costs its part of a full wave, and its forms are a level of butterflies or two levels
// by lanes with quarter turns, the least work.  Without memory for products, a level
// of butterflies a pass.
static std::vector<FftPass> fft_plan(const std::vector<const FftJob*>& jobs, bool solo, bool with_products)
{
    constexpr double kSumMs = 0.5e-6, kSumsMs = 0.03, kFullMs = 0.57;     // kFullMs: wave products of a full launch
    constexpr uint32_t kMaxQ = 4;
    const size_t wave = fft_quad_wave();
    uint32_t maxlog = 0;
    for (const FftJob* J : jobs) maxlog = std::max(maxlog, J->logn);
    std::vector<double> best(maxlog + 1, 1e300);
    std::vector<FftPass> via(maxlog + 1);
    best[0] = 0;
    for (uint32_t s = 0; s < maxlog; s++) {
        for (uint32_t q = 1; q <= (!with_products ? 1 : solo ? kMaxQ : 2) && s + q <= maxlog; q++) {
            size_t items, products[2], outputs;
            pass_counts(jobs, s, q, items, products, outputs);
            FftPass p;
            p.s0 = s;
            p.q = q;
            double ms = 1e300;
            if (q == 1) {
                const double bf = (double)outputs / 2, scaled = std::max(0.0, (double)products[0] - (s ? bf : 0));
                ms = (solo ? stage_ms(outputs / 2, wave) : kFullMs / (double)wave * bf) * (1 + 0.85 * scaled / bf);
            }
            const bool fits = with_products && items <= pass_max_items(q);
            for (uint32_t turns = solo ? 0 : 1; fits && turns < (q > 1 ? 2u : 1u); turns++) {
                // the products of a first pass are not adjacent: its SMs have uneven shares
                const size_t n = s || turns ? products[turns] : products[turns] * 3 / 2;
                const size_t v = outputs / 2 - (outputs >> q);
                const double sums = kSumsMs + kSumMs * (double)outputs * (1u << q);
                const double turn = turns ? quarter_ms(v, wave) : 0.0;
                p.quad_turns = v <= wave;
                if (!solo) {
                    ms = kFullMs / (double)wave * ((double)n + (double)v / 3) + sums;
                    p.kind = FftPass::kLanes;
                    p.turns = 1;
                    continue;
                }
                const struct {
                    decltype(p.kind) kind;
                    uint32_t split;
                    double ms;
                } forms[] = {{FftPass::kLanes, 0, lanes_ms(n, wave) + sums},
                             {FftPass::kPairs, 0, pairs_ms(n, wave) + sums},
                             {FftPass::kQuads, 0, quads_ms(n, wave, false) + sums},
                             {FftPass::kQuads, 1, q <= 3 ? quads_ms(2 * n, wave, true) + 2 * sums : 1e300}};
                for (const auto& f : forms)
                    if (f.ms + turn < ms) {
                        p.kind = f.kind;
                        p.split = f.split;
                        p.turns = turns;
                        ms = f.ms + turn;
                    }
            }
            if (best[s] + ms < best[s + q]) {
                best[s + q] = best[s] + ms;
                via[s + q] = p;
            }
        }
    }
    std::vector<FftPass> plan;
    for (uint32_t s = maxlog; s > 0; s = via[s].s0) plan.push_back(via[s]);
    std::reverse(plan.begin(), plan.end());
    return plan;
}

// Runs every job of `specs` over the concatenated values in d_values
// (job i at element offset sum_{j<i} n_j); results land back in d_values.
cudaError_t fft_run_multi(Ctx* ctx, void* d_values, const FftSpec* specs, size_t count)
{
    cudaStream_t st = ctx->stream;
    FftWork& W = ctx->fft;
    std::vector<FftJob> jobs(count);
    std::vector<uint32_t> vpre(count + 1);
    size_t total = 0, glv_total = 0;
    for (size_t i = 0; i < count; i++) {
        const size_t n = specs[i].n;
        uint32_t lg = 0;
        while (((size_t)1 << lg) < n) lg++;
        jobs[i].val_off = (uint32_t)total;
        jobs[i].n = (uint32_t)n;
        jobs[i].logn = lg;
        jobs[i].inv_from_fwd = specs[i].inv_from_fwd ? 1 : 0;
        jobs[i].glv_off = (uint32_t)glv_total;
        jobs[i].xn = (uint32_t)(specs[i].xn && specs[i].xn < n ? specs[i].xn : n);
        jobs[i].roots = specs[i].roots_mont;
        jobs[i].scale = specs[i].scale_mont;
        vpre[i] = (uint32_t)total;
        total += n;
        glv_total += n + n / 2 + 1;
    }
    vpre[count] = (uint32_t)total;
    if (total >= 0x7fffffffu) return cudaErrorInvalidValue;
    // A batch of more than one wave of lanes runs as two groups of jobs on two
    // streams: a level's last, partly filled wave (46080 butterflies are 1.18
    // waves) overlaps a level of the other group.  Six transforms of 2^10 ..
    // 2^16: 55.5 ms as one group, 46.9 as two.
    const int groups = count > 1 && total / 2 > 4 * fft_quad_wave() ? 2 : 1;
    std::vector<uint32_t> group(count, 0);
    std::vector<const FftJob*> members[2];
    if (groups == 2) {
        std::vector<uint32_t> order(count);
        for (size_t i = 0; i < count; i++) order[i] = (uint32_t)i;
        std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return jobs[a].n > jobs[b].n; });
        size_t load[2] = {0, 0};
        for (uint32_t i : order) {
            group[i] = load[1] < load[0] ? 1 : 0;
            load[group[i]] += (size_t)jobs[i].n * jobs[i].logn;
        }
    }
    for (size_t i = 0; i < count; i++) members[group[i]].push_back(&jobs[i]);
    std::vector<FftPass> plan;
    // per-pass lists of (job, first item, first output)
    std::vector<uint32_t> lst_job, lst_item, lst_out;
    size_t max_items[2];
    bool stages;
    auto make_plan = [&](bool with_products) {
        plan.clear();
        for (std::vector<uint32_t>* l : {&lst_job, &lst_item, &lst_out}) l->clear();
        max_items[0] = max_items[1] = 0;
        stages = false;
        for (int g = 0; g < groups; g++)
            for (FftPass p : fft_plan(members[g], groups == 1, with_products)) {
                p.group = (uint32_t)g;
                plan.push_back(p);
            }
        for (FftPass& p : plan) {
            p.off = (uint32_t)lst_job.size();
            for (size_t i = 0; i < count; i++) {
                const FftJob& J = jobs[i];
                if (group[i] != p.group || J.logn <= p.s0) continue;
                const uint32_t qe = std::min(p.q, J.logn - p.s0);
                const uint32_t bf = std::min(J.n >> (p.s0 + qe), J.xn) << p.s0;
                lst_job.push_back((uint32_t)i);
                lst_item.push_back(p.items);
                lst_out.push_back(p.outputs);
                p.items += p.kind == FftPass::kStage ? bf : bf * pass_items(qe) << p.split;
                p.outputs += bf << qe;
            }
            p.cnt = (uint32_t)lst_job.size() - p.off;
            if (p.kind == FftPass::kStage) stages = true;
            else max_items[p.group] = std::max(max_items[p.group], (size_t)p.items);
        }
    };
    make_plan(true);
    xyzz* prod = (xyzz*)W.prod.get((max_items[0] + max_items[1]) * sizeof(xyzz));
    if (!prod) {                                     // up to 805 MB a group: butterflies need none of it
        make_plan(false);
        prod = (xyzz*)W.prod.get(0);
    }
    const size_t meta_words = count * (sizeof(FftJob) / 4) + (count + 1) + 3 * lst_job.size() + 8;
    xyzz* tmp = (xyzz*)W.scratch.get(total * sizeof(xyzz));
    uint32_t* glv = (uint32_t*)W.glv.get(stages ? glv_total * 32 : 0);
    uint32_t* meta = (uint32_t*)W.meta.get(meta_words * 4);
    uint32_t* hmeta = (uint32_t*)ctx->h_meta.get(meta_words * 4);
    if (!tmp || !prod || !glv || !meta || !hmeta) return cudaErrorMemoryAllocation;
    if (groups == 2) CATMSM_CHECK(W.aux.ensure(st));
    uint32_t* hp = hmeta;
    std::memcpy(hp, jobs.data(), count * sizeof(FftJob));
    hp += count * (sizeof(FftJob) / 4);
    std::memcpy(hp, vpre.data(), (count + 1) * 4);
    hp += count + 1;
    for (const std::vector<uint32_t>* l : {&lst_job, &lst_item, &lst_out}) {
        if (!l->empty()) std::memcpy(hp, l->data(), l->size() * 4);
        hp += l->size();
    }
    CATMSM_CHECK(cudaMemcpyAsync(meta, hmeta, meta_words * 4, cudaMemcpyHostToDevice, st));
    const FftJob* d_jobs = reinterpret_cast<const FftJob*>(meta);
    const uint32_t* d_vpre = meta + count * (sizeof(FftJob) / 4);
    const uint32_t* d_lst_job = d_vpre + count + 1;
    const uint32_t* d_lst_item = d_lst_job + lst_job.size();
    const uint32_t* d_lst_out = d_lst_item + lst_job.size();
    // prepared roots per job (jobs sharing a root table share the work only
    // through the L2; preparation is O(n) next to O(n log n) scalar mults)
    for (size_t i = 0; stages && i < count; i++) {
        k_roots_prepare<<<div_up(jobs[i].n, 256), 256, 0, st>>>(specs[i].roots_mont, jobs[i].n, glv + 8 * (size_t)jobs[i].glv_off);
        if (specs[i].scale_mont)
            k_roots_prepare_scaled<<<div_up(jobs[i].n / 2 + 1, 256), 256, 0, st>>>(
                specs[i].roots_mont, specs[i].scale_mont, jobs[i].n, jobs[i].inv_from_fwd,
                glv + 8 * (size_t)(jobs[i].glv_off + jobs[i].n));
        g_stats.launches += 1 + (specs[i].scale_mont ? 1 : 0);
    }
    k_bitrev_multi<<<div_up(total, 128), 128, 0, st>>>((const jac*)d_values, tmp, d_jobs, d_vpre, (uint32_t)count,
                                                       (uint32_t)total);
    g_stats.launches++;
    if (groups == 2) CATMSM_CHECK(W.aux.begin(st));
    // launches alternate between the groups, so neither stream waits for the host
    std::vector<const FftPass*> seq;
    size_t next[2] = {0, plan.size()};
    while (next[1] > 0 && plan[next[1] - 1].group == 1) next[1]--;
    const size_t first1 = next[1];
    while (next[0] < first1 || next[1] < plan.size()) {
        if (next[0] < first1) seq.push_back(&plan[next[0]++]);
        if (next[1] < plan.size()) seq.push_back(&plan[next[1]++]);
    }
    for (const FftPass* pass : seq) {
        const FftPass& p = *pass;
        cudaStream_t ps = p.group ? W.aux.stream : st;
        xyzz* pp = prod + (p.group ? max_items[0] : 0);
        const uint32_t* lj = d_lst_job + p.off;
        const uint32_t* li = d_lst_item + p.off;
        if (p.kind == FftPass::kStage) {
            if (p.items <= 4 * fft_quad_wave())
                k_fft_stage_multi<4><<<div_up(p.items, 64), 64, 0, ps>>>(tmp, d_jobs, lj, li, p.cnt, p.items,
                                                                         2u << p.s0, glv);
            else
                k_fft_stage_multi<6><<<div_up(p.items, 64), 64, 0, ps>>>(tmp, d_jobs, lj, li, p.cnt, p.items,
                                                                         2u << p.s0, glv);
            g_stats.launches++;
            continue;
        }
        const uint32_t lanes = p.kind == FftPass::kQuads ? 4 : p.kind == FftPass::kPairs ? 2 : 1;
        const unsigned grid = div_up((size_t)lanes * p.items, kItemThreads);
        if (p.split)
            k_fft_items<4, true><<<grid, kItemThreads, 0, ps>>>(tmp, pp, d_jobs, lj, li, p.cnt, p.items, p.s0, p.q, p.turns);
        else if (lanes == 4)
            k_fft_items<4, false><<<grid, kItemThreads, 0, ps>>>(tmp, pp, d_jobs, lj, li, p.cnt, p.items, p.s0, p.q, p.turns);
        else if (lanes == 2)
            k_fft_items<2, false><<<grid, kItemThreads, 0, ps>>>(tmp, pp, d_jobs, lj, li, p.cnt, p.items, p.s0, p.q, p.turns);
        else
            k_fft_items<1, false><<<grid, kItemThreads, 0, ps>>>(tmp, pp, d_jobs, lj, li, p.cnt, p.items, p.s0, p.q, p.turns);
        if (p.turns) {
            const uint32_t turns = p.outputs / 2;
            if (p.quad_turns)
                k_fft_quarter<true><<<div_up(4 * (size_t)turns, 64), 64, 0, ps>>>(
                    pp, d_jobs, lj, li, d_lst_out + p.off, p.cnt, turns, p.s0, p.q, p.split);
            else
                k_fft_quarter<false><<<div_up(turns, 64), 64, 0, ps>>>(pp, d_jobs, lj, li, d_lst_out + p.off, p.cnt,
                                                                       turns, p.s0, p.q, p.split);
            g_stats.launches++;
        }
        k_fft_combine<<<div_up((size_t)p.outputs << (p.q + 1 + p.split), 128), 128, 0, ps>>>(
            pp, tmp, d_jobs, lj, li, d_lst_out + p.off, p.cnt, p.outputs, p.s0, p.q, p.split);
        g_stats.launches += 2;
    }
    if (groups == 2) CATMSM_CHECK(W.aux.end(st));
    k_fft_finish_multi<<<div_up(total, 64), 64, 0, st>>>(tmp, (jac*)d_values, d_jobs, d_vpre, (uint32_t)count,
                                                         (uint32_t)total);
    g_stats.launches++;
    return cudaGetLastError();
}

// single transform: d_values n Jacobian points; d_roots_mont the n
// Montgomery roots the butterflies index; d_scale_mont optional scale
cudaError_t fft_run(Ctx* ctx, void* d_values, size_t n, const uint32_t* d_roots_mont, bool inv_from_fwd,
                    const uint32_t* d_scale_mont, size_t xn)
{
    FftSpec sp{n, d_roots_mont, inv_from_fwd, d_scale_mont, xn};
    return fft_run_multi(ctx, d_values, &sp, 1);
}

cudaError_t fft_root_powers(Ctx* ctx, const uint32_t* d_w_mont, size_t n, uint32_t* d_out)
{
    k_root_powers<<<div_up(n, 256), 256, 0, ctx->stream>>>(d_w_mont, (uint32_t)n, d_out);
    g_stats.launches++;
    return cudaGetLastError();
}

}  // namespace catmsm
