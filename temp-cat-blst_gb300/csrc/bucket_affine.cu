// Batch-affine bucket accumulation: the first rounds of every bucket's sum as
// affine additions behind Montgomery batch inversions, the rest with the XYZZ
// mixed addition.
//
// Reference precedent: the CPU batch-affine Pippenger
// (blst/scalar/curve/multi_scalar_batch_affine.cpp, bulk_addition.h), which
// adds points into affine buckets and shares one inversion among a batch of
// independent additions.  An affine addition P + Q = (l^2 - x1 - x2,
// l (x1 - x3) - y1) with l = (y2 - y1) / (x2 - x1) costs 2M + 1S plus its
// share of the inversion; Montgomery's trick makes that share 3M for a batch,
// so an addition is ~5M + 1S (3336 IMAD) against 8M + 2S for the XYZZ mixed
// addition (5340 IMAD as executed here).
//
// The sorted bucket entries are split into the same chunks of L entries as
// k_accumulate (thread t owns chunk t), so the fixup stage that joins buckets
// across chunks is unchanged.  A round halves each thread's runs: within each
// run of equal bucket keys, items (0,1), (2,3), ... are added and an odd last
// item passes through; the results form the thread's list for the next
// round, still in bucket order.  Round 1 reads the sorted entries (a gather
// of signed points); later rounds read the list the previous round wrote.
// A thread's lists, pair positions and prefix products are slot-major (see
// Slots), so a warp's accesses at one step of the loops are adjacent.
// One round is three launches:
//   forward   each thread walks its pairs from first to last, storing the
//             running product of the denominators before each pair (its
//             prefix) and ending with its total; groups of 16 lanes multiply
//             their totals by shuffles;
//   invert    one thread per group inverts the group's product
//             (fp_inv_vartime: tens of microseconds, not Fermat's ~0.45 ms);
//   backward  a thread's inverse is the group's times the other lanes'
//             product, and each thread walks its pairs from last to first: inv(d_j) = prefix_j * I, I *= d_j,
//             then the affine sum.  The same kernel then runs the next
//             round's forward pass, or, after the last round, folds the
//             remaining list into the chunk's bucket / head / tail exactly as
//             k_accumulate does (XYZZ mixed additions).
// Special cases keep the group law complete: an infinity operand (all-zero
// affine) returns the other operand, x1 = x2 with y1 = y2 doubles
// (l = 3 x1^2 / 2 y1), x1 = x2 with y1 = -y2 gives infinity; their batch
// slots use the denominator 1 (or 2 y1 for the doubling).
#define CATMSM_INLINE_SQR   // see field.cuh
#include "common.cuh"
#include "curve.cuh"
#include "fpinv.cuh"
#include "catmsm_internal.h"

#include <algorithm>

namespace catmsm {

__global__ void k_accumulate(const affine* __restrict__ pts, const uint32_t* __restrict__ sorted_pt,
                             const uint32_t* __restrict__ sorted_key, const uint32_t* __restrict__ total_ptr,
                             uint32_t below, uint32_t L, xyzz* __restrict__ buckets, xyzz* __restrict__ head,
                             xyzz* __restrict__ tail);

constexpr int kAffThreads = 64;         // 128: 2^20 points 5.57 -> 5.53 ms, 300007 2.337 -> 2.325 (shorter last waves)
constexpr uint32_t kAffGroup = 16;      // lanes that share an inversion
// Resident blocks per SM the round kernels are compiled for (register limit
// 65536 / (64 x this)).
#ifndef CATMSM_AFF_MIN_BLOCKS
#define CATMSM_AFF_MIN_BLOCKS 8
#endif

// 48 bytes (one coordinate) from a 16-byte aligned address.  Mutable: data
// this launch may write (a thread's own list slots, prefix products and
// totals, which only that thread writes and reads back), with plain loads --
// coherent with the thread's own earlier stores and cached in L1, so the two
// 16-byte halves of a sector and a thread's consecutive keys hit L1.  The
// others (read-only for the whole launch) take the read-only path.
template <bool Mutable>
__device__ __forceinline__ void load_coord(fp& c, const uint4* q)
{
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint4 v = Mutable ? q[k] : __ldg(q + k);
        c.v[4 * k + 0] = v.x; c.v[4 * k + 1] = v.y; c.v[4 * k + 2] = v.z; c.v[4 * k + 3] = v.w;
    }
}

// 48-byte field elements in global memory as three 16-byte accesses (a
// plain struct copy is twelve 4-byte ones, each a separate sector per lane).
__device__ __forceinline__ void stg_fp(fp* dst, const fp& v)
{
    uint4* q = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int k = 0; k < 3; k++) q[k] = make_uint4(v.v[4 * k], v.v[4 * k + 1], v.v[4 * k + 2], v.v[4 * k + 3]);
}

template <bool Mutable>
__device__ __forceinline__ fp ldg_fp(const fp* src)
{
    fp v;
    load_coord<Mutable>(v, reinterpret_cast<const uint4*>(src));
    return v;
}

// An item's 96-byte row and whether its y is negated.
struct Row {
    const uint4* p;
    bool neg;
};

// Items of round 1: sorted entry base + i, a signed point of the GLV array
// (read-only for the whole accumulation).
struct SrcSorted {
    static constexpr bool kMutable = false;
    const affine* pts;
    const uint32_t* sorted_pt;
    const uint32_t* sorted_key;
    size_t base;
    __device__ __forceinline__ uint32_t key(uint32_t i) const { return sorted_key[base + i]; }
    // the item's token: one load, made a pair or two before the row is needed
    __device__ __forceinline__ uint32_t token(uint32_t i) const { return sorted_pt[base + i]; }
    __device__ __forceinline__ Row row_of(uint32_t v) const
    {
        return Row{reinterpret_cast<const uint4*>(pts + (v & 0x7fffffffu)), (v >> 31) != 0};
    }
    __device__ __forceinline__ Row row(uint32_t i) const { return row_of(token(i)); }
};

// A thread's private arrays (lists, pair positions, prefix products) are
// slot-major: slot i of thread t is element i T + t (T threads in all), so
// the lanes of a warp at the same step of their loops touch adjacent
// elements instead of elements L apart.
struct Slots {
    size_t t, T;
    __device__ __forceinline__ size_t at(uint32_t i) const { return (size_t)i * T + t; }
};

// Items of later rounds: the thread's list.  Its slots may have been written
// earlier in the same launch (by this thread only).
struct SrcList {
    static constexpr bool kMutable = true;
    const affine* pts;
    const uint32_t* keys;
    Slots sl;
    __device__ __forceinline__ uint32_t key(uint32_t i) const { return keys[sl.at(i)]; }
    __device__ __forceinline__ uint32_t token(uint32_t i) const { return i; }
    __device__ __forceinline__ Row row_of(uint32_t i) const
    {
        return Row{reinterpret_cast<const uint4*>(pts + sl.at(i)), false};
    }
    __device__ __forceinline__ Row row(uint32_t i) const { return row_of(i); }
};

template <class Src>
__device__ __forceinline__ void row_x(const Row& r, fp& x)
{
    load_coord<Src::kMutable>(x, r.p);
}

template <class Src>
__device__ __forceinline__ void row_y(const Row& r, fp& y)
{
    load_coord<Src::kMutable>(y, r.p + 3);
    if (r.neg) fp_neg(y, y);
}

enum : uint32_t { kPairAdd = 0, kPairDbl = 1, kPairInf = 2, kPairTakeA = 3, kPairTakeB = 4 };

// Kind of the pair (A, B) and its batch denominator.  Only x is needed for
// the common case; y is loaded when an x is zero or the x coordinates agree.
template <class Src>
__device__ __forceinline__ uint32_t pair_den(const Row& ra, const Row& rb, const fp& x1, const fp& x2, fp& d)
{
    fp_sub(d, x2, x1);
    if (!fp_is_zero_raw(x1) && !fp_is_zero_raw(x2) && !fp_is_zero(d)) return kPairAdd;
    fp y1, y2;
    row_y<Src>(ra, y1);
    row_y<Src>(rb, y2);
    fp_set_one(d);
    if (fp_is_zero_raw(x1) && fp_is_zero_raw(y1)) return kPairTakeB;
    if (fp_is_zero_raw(x2) && fp_is_zero_raw(y2)) return kPairTakeA;
    fp t;
    fp_sub(t, x2, x1);
    if (!fp_is_zero(t)) {
        fp_sub(d, x2, x1);
        return kPairAdd;
    }
    fp_sub(t, y2, y1);
    if (!fp_is_zero(t) || fp_is_zero(y1)) return kPairInf;   // P + (-P), or 2-torsion
    fp_dbl(d, y1);
    return kPairDbl;
}

template <class Src>
__device__ __forceinline__ void copy_item(const Src& src, uint32_t i, affine* dst)
{
    const Row r = src.row(i);
    affine a;
    row_x<Src>(r, a.x);
    row_y<Src>(r, a.y);
    store_affine(dst, a);
}

// Forward pass of one round over the thread's items [0, cnt).
//  Pairing: within each run of equal keys, items (0,1), (2,3), ... pair and an
//  odd last item is a singleton, copied to the output list now; pair slots get
//  their keys.  Keys are read four at a time, so the walk does not wait on one
//  load per item.
//  Prefix products: pair j stores d_0 ... d_{j-1}; the next pair's rows are
//  fetched before this pair's multiplication, so the row lookups (for round 1
//  an index load, then the point) overlap it.
// Returns the product of all denominators; *np_out = pairs, *cnt_out = items
// of the output list.
template <class Src>
__device__ __forceinline__ fp aff_forward(const Src& src, uint32_t cnt, affine* outP, uint32_t* outK, Slots os,
                                          uint32_t* pairpos, fp* prefix, Slots ps, uint32_t* np_out,
                                          uint32_t* cnt_out)
{
    uint32_t o = 0, np = 0, pi = 0, pk = 0;
    bool pend = false;
    for (uint32_t i0 = 0; i0 < cnt; i0 += 4) {
        uint32_t kk[4];
#pragma unroll
        for (int u = 0; u < 4; u++) kk[u] = i0 + u < cnt ? src.key(i0 + u) : 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t i = i0 + u;
            if (i < cnt) {
                if (pend && kk[u] == pk) {
                    pairpos[ps.at(np)] = (pi << 16) | o;
                    outK[os.at(o)] = pk;
                    np++;
                    o++;
                    pend = false;
                } else {
                    if (pend) {
                        copy_item(src, pi, outP + os.at(o));
                        outK[os.at(o)] = pk;
                        o++;
                    }
                    pend = true;
                    pi = i;
                    pk = kk[u];
                }
            }
        }
    }
    if (pend) {
        copy_item(src, pi, outP + os.at(o));
        outK[os.at(o)] = pk;
        o++;
    }
    *np_out = np;
    *cnt_out = o;
    fp q;
    fp_set_one(q);
    if (np == 0) return q;
    // pair j: a, b its tokens; an, bn those of pair j + 1; ip2 the position of pair j + 2
    uint32_t ip = pairpos[ps.at(0)] >> 16;
    uint32_t a = src.token(ip), b = src.token(ip + 1), an = a, bn = b, ip2 = 0;
    if (np > 1) {
        ip = pairpos[ps.at(1)] >> 16;
        an = src.token(ip);
        bn = src.token(ip + 1);
    }
    if (np > 2) ip2 = pairpos[ps.at(2)] >> 16;
    for (uint32_t j = 0; j < np; j++) {
        const Row ra = src.row_of(a), rb = src.row_of(b);
        fp x1, x2, d;
        row_x<Src>(ra, x1);
        row_x<Src>(rb, x2);
        a = an;
        b = bn;
        if (j + 2 < np) {
            an = src.token(ip2);
            bn = src.token(ip2 + 1);
        }
        if (j + 3 < np) ip2 = pairpos[ps.at(j + 3)] >> 16;
        pair_den<Src>(ra, rb, x1, x2, d);
        stg_fp(prefix + ps.at(j), q);
        fp_mul(q, q, d);
    }
    return q;
}

// Backward pass of one round, pairs from last to first: I = inverse of
// d_0 ... d_j, inv(d_j) = prefix_j I, then I = I d_j; pair j's sum goes to
// its output slot.  The previous pair's rows are fetched before this pair's
// arithmetic.
template <class Src>
__device__ __forceinline__ void aff_backward(const Src& src, uint32_t np, affine* outP, Slots os,
                                             const uint32_t* pairpos, const fp* prefix, Slots ps, fp I)
{
    if (np == 0) return;
    // pair j: pp its positions, a, b its tokens; pn, an, bn those of pair j - 1
    uint32_t pp = pairpos[ps.at(np - 1)], pn = 0, an = 0, bn = 0;
    uint32_t a = src.token(pp >> 16), b = src.token((pp >> 16) + 1);
    if (np > 1) pn = pairpos[ps.at(np - 2)];
    for (uint32_t j = np; j-- > 0;) {
        const Row ra = src.row_of(a), rb = src.row_of(b);
        fp x1, y1, x2, y2, d;
        row_x<Src>(ra, x1);
        row_x<Src>(rb, x2);
        row_y<Src>(ra, y1);
        row_y<Src>(rb, y2);
        const uint32_t o = pp & 0xffffu;
        if (j > 0) {
            an = src.token(pn >> 16);
            bn = src.token((pn >> 16) + 1);
        }
        const uint32_t kind = pair_den<Src>(ra, rb, x1, x2, d);
        fp inv;
        fp_mul(inv, ldg_fp<true>(prefix + ps.at(j)), I);   // rewritten by the next forward pass
        pp = pn;
        if (j > 1) pn = pairpos[ps.at(j - 2)];
        a = an;
        b = bn;
        fp_mul(I, I, d);
        affine r;
        if (kind == kPairAdd || kind == kPairDbl) {
            fp num, lam, t;
            if (kind == kPairAdd) {
                fp_sub(num, y2, y1);
            } else {
                fp_sqr(t, x1);
                fp_dbl(num, t);
                fp_add(num, num, t);
            }
            fp_mul(lam, num, inv);
            fp_sqr(t, lam);
            fp_sub(t, t, x1);
            fp_sub(r.x, t, x2);
            fp_sub(t, x1, r.x);
            fp_mul(t, lam, t);
            fp_sub(r.y, t, y1);
        } else if (kind == kPairTakeA) {
            r.x = x1;
            r.y = y1;
        } else if (kind == kPairTakeB) {
            r.x = x2;
            r.y = y2;
        } else {
            fp_zero(r.x);
            fp_zero(r.y);
        }
        store_affine(outP + os.at(o), r);
    }
}

// The lanes of a group share one inversion.  Multiplies their totals by a
// butterfly of shuffles: every lane ends with the group's product (returned) and
// with the product of the other lanes' totals (`rest`), so that the inverse of
// the product times `rest` is the inverse of the lane's own total.  7 dependent
// products for 16 lanes and no barrier; a shared-memory tree over the block's
// 128 threads, formed again by the next launch, was 28 and held 12 KB of the L1.
// Groups of 16: twice the inversions of whole warps (one launch of them lasts
// as long: a warp per scheduler at 2^20 points) and two products fewer.
__device__ __forceinline__ fp group_product(const fp& total, fp& rest)
{
    fp p = total;
#pragma unroll
    for (uint32_t d = 1; d < kAffGroup; d <<= 1) {
        fp o;
#pragma unroll
        for (int k = 0; k < 12; k++) o.v[k] = __shfl_xor_sync(0xffffffffu, p.v[k], d);
        if (d == 1) rest = o;
        else fp_mul(rest, rest, o);
        fp_mul(p, p, o);
    }
    return p;
}

// k_accumulate's fold over the thread's final list: runs of equal keys are
// summed with XYZZ mixed additions; the chunk's first run goes to head[t] if
// the bucket started in an earlier chunk, its last run to tail[t] if the
// bucket continues into the next chunk, every other run to its bucket.
__device__ __forceinline__ void aff_fold(const SrcList& list, uint32_t cnt, const uint32_t* sorted_key,
                                         size_t start, uint32_t E, uint32_t L, uint32_t t, xyzz* buckets,
                                         xyzz* head, xyzz* tail)
{
    if (cnt == 0) return;
    const uint32_t end = (uint32_t)min((size_t)E, start + L);
    uint32_t cur = list.key(0);
    const bool starts_before = start > 0 && sorted_key[start - 1] == cur;
    bool first_run = true;
    xyzz acc;
    xyzz_set_inf(acc);
    for (uint32_t i = 0; i < cnt; i++) {
        const uint32_t key = list.key(i);
        if (key != cur) {
            if (first_run && starts_before) store_xyzz(head + t, acc);
            else store_xyzz(buckets + cur, acc);
            first_run = false;
            xyzz_set_inf(acc);
            cur = key;
        }
        fp x, y;
        const Row r = list.row(i);
        row_x<SrcList>(r, x);
        row_y<SrcList>(r, y);
        if (!(fp_is_zero_raw(x) && fp_is_zero_raw(y))) xyzz_madd(acc, x, y);
    }
    const bool continues_after = end < E && sorted_key[end] == cur;
    if (first_run && starts_before) store_xyzz(head + t, acc);
    else if (continues_after) store_xyzz(tail + t, acc);
    else store_xyzz(buckets + cur, acc);
}

struct AffArgs {
    const affine* pts;            // signed GLV points (round 1 items, through sorted_pt)
    const uint32_t* sorted_pt;
    const uint32_t* sorted_key;
    const uint32_t* total_ptr;    // E, the number of sorted entries
    uint32_t least;               // with fewer entries the launches leave at once
    uint32_t L;                   // chunk length
    size_t T;                     // threads of a slice: the slot-major stride
    affine* list_pts[2];          // per-thread lists: slot i of thread t at i T + t
    uint32_t* list_key[2];
    uint32_t* meta;               // per thread: pairs | output items << 16 of the round in flight
    uint32_t* pairpos;            // pair j of thread t at j T + t: input position << 16 | output slot
    fp* prefix;                   // pair j of thread t at j T + t: its prefix product
    fp* rest;                     // per thread: product of the other lanes' denominators in its group
    fp* gtot;                     // per group: product of its denominators, then its inverse
    xyzz* buckets;
    xyzz* head;
    xyzz* tail;
    uint32_t slice, slices;       // this slice's block b holds the chunks of block b slices + slice
};

// Whether no chunk of the slice's block b holds an entry (a batch's launches
// cover full MSMs, whatever the batch holds), or none is to be done here.
__device__ __forceinline__ bool aff_idle(const AffArgs& A, uint32_t b, uint32_t E)
{
    return ((size_t)b * A.slices + A.slice) * kAffThreads * A.L >= E || E < A.least;
}

// The chunk of this thread.
__device__ __forceinline__ uint32_t aff_chunk(const AffArgs& A)
{
    return (blockIdx.x * A.slices + A.slice) * kAffThreads + threadIdx.x;
}

// Ends a forward pass: the thread's total goes into its group's product.
__device__ __forceinline__ void aff_totals(const AffArgs& A, uint32_t t, const fp& tot)
{
    fp rest;
    const fp g = group_product(tot, rest);
    stg_fp(A.rest + t, rest);
    if (t % kAffGroup == 0) stg_fp(A.gtot + t / kAffGroup, g);
}

// Round 1's forward pass, over the sorted entries.
__global__ void __launch_bounds__(kAffThreads, CATMSM_AFF_MIN_BLOCKS) k_aff_first(AffArgs A)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t E = *A.total_ptr;
    if (aff_idle(A, blockIdx.x, E)) return;
    const size_t start = (size_t)aff_chunk(A) * A.L;
    const uint32_t cnt = start < E ? (uint32_t)min((size_t)A.L, (size_t)E - start) : 0;
    const SrcSorted src{A.pts, A.sorted_pt, A.sorted_key, start};
    uint32_t np = 0, co = 0;
    const Slots sl{t, A.T};
    const fp tot = aff_forward(src, cnt, A.list_pts[0], A.list_key[0], sl, A.pairpos, A.prefix, sl, &np, &co);
    A.meta[t] = np | (co << 16);
    aff_totals(A, t, tot);
}

// One thread per group product: its inverse, in place (about one inversion's
// latency for the whole launch).
__global__ void k_aff_invert(AffArgs A, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || aff_idle(A, i / (kAffThreads / kAffGroup), *A.total_ptr)) return;
    fp r;
    fp_inv_vartime(r, ldg_fp<true>(A.gtot + i));     // overwritten below
    stg_fp(A.gtot + i, r);
}

// Backward pass of round r (inputs: the sorted entries if First, else list
// (r % 2); outputs: list ((r - 1) % 2)), then round r + 1's forward pass into
// list (r % 2), or, if Last, the fold into buckets / head / tail.
template <bool First, bool Last>
__global__ void __launch_bounds__(kAffThreads, CATMSM_AFF_MIN_BLOCKS) k_aff_round(AffArgs A, uint32_t r)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t E = *A.total_ptr;
    if (aff_idle(A, blockIdx.x, E)) return;
    const size_t start = (size_t)aff_chunk(A) * A.L;
    const Slots sl{t, A.T};
    const uint32_t m = A.meta[t];
    const uint32_t np = m & 0xffffu, co = m >> 16;
    fp I;                                                         // both rewritten at the end of this launch
    fp_mul(I, ldg_fp<true>(A.rest + t), ldg_fp<true>(A.gtot + t / kAffGroup));
    __syncwarp();                                                 // the group's inverse is read before lane 0 rewrites it
    const uint32_t out = (r - 1) & 1, in = r & 1;
    if (First) {
        const SrcSorted src{A.pts, A.sorted_pt, A.sorted_key, start};
        aff_backward(src, np, A.list_pts[out], sl, A.pairpos, A.prefix, sl, I);
    } else {
        const SrcList src{A.list_pts[in], A.list_key[in], sl};
        aff_backward(src, np, A.list_pts[out], sl, A.pairpos, A.prefix, sl, I);
    }
    const SrcList list{A.list_pts[out], A.list_key[out], sl};
    if (Last) {
        aff_fold(list, co, A.sorted_key, start, E, A.L, aff_chunk(A), A.buckets, A.head, A.tail);
    } else {
        uint32_t np2 = 0, co2 = 0;
        const fp tot = aff_forward(list, co, A.list_pts[in], A.list_key[in], sl, A.pairpos, A.prefix, sl, &np2,
                                   &co2);
        A.meta[t] = np2 | (co2 << 16);
        aff_totals(A, t, tot);
    }
}

__global__ void k_fp_inv_test(const fp* __restrict__ a, fp* __restrict__ o, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fp r;
    fp_inv_vartime(r, a[i]);
    fp_canon(r, r);
    o[i] = r;
}

cudaError_t fp_inv_test_device(Ctx* ctx, const uint64_t* d_a, uint64_t* d_out, size_t n)
{
    k_fp_inv_test<<<div_up(n, 64), 64, 0, ctx->stream>>>((const fp*)d_a, (fp*)d_out, (uint32_t)n);
    g_stats.launches++;
    return cudaGetLastError();
}

// The chunks run in slices of blocks, alternating between the pipeline's stream
// and the workspace's second one: an inversion launch (one inversion's latency,
// few warps) of one slice overlaps the other stream's round kernel instead of
// idling the GPU.  At most four waves and 2^25 entries a slice (~8 GB of lists
// and prefix products per stream), an even number of slices.  A slice takes every
// count-th block, so all have the same share of the entries however few of
// the chunks a batch fills.  (Two waves a slice: 2^22 points 20.3 -> 20.5 ms.)
struct AffSlices {
    uint32_t count, blocks;     // slices, most blocks of one
};

static AffSlices aff_slices(uint32_t L, uint32_t grid)
{
    if (grid <= 1) return {1, 1};
    const uint32_t waves = 4 * CATMSM_AFF_MIN_BLOCKS * (uint32_t)device_sms();
    const uint32_t most = std::max(1u, std::min(waves, (1u << 25) / (kAffThreads * L)));
    const uint32_t n = 2 * ((grid + 2 * most - 1) / (2 * most));
    return {n, (grid + n - 1) / n};
}

cudaError_t aff_prepare(AffWork& W, uint32_t L, size_t chunks, cudaStream_t st)
{
    if (L == 0 || L > 0xffffu) return cudaErrorInvalidValue;
    const size_t T = (size_t)aff_slices(L, div_up(chunks, kAffThreads)).blocks * kAffThreads;
    const size_t H = (L + 1) / 2;
    for (AffWork::Set& w : W.set) {
        if (!w.pts0.get(T * L * sizeof(affine)) || !w.pts1.get(T * L * sizeof(affine)) || !w.key0.get(T * L * 4) ||
            !w.key1.get(T * L * 4) || !w.meta.get(T * 4) || !w.pairpos.get(T * H * 4) ||
            !w.prefix.get(T * H * sizeof(fp)) || !w.rest.get(T * sizeof(fp)) ||
            !w.gtot.get(T / kAffGroup * sizeof(fp))) {
            W.release_lists();       // the caller goes on without the rounds: the others may need what was got
            return cudaErrorMemoryAllocation;
        }
    }
    return W.aux.ensure(st);
}

cudaError_t aff_accumulate(const AffWork& W, const void* pts, const uint32_t* sorted_pt, const uint32_t* sorted_key,
                           const uint32_t* total, uint32_t least, uint32_t L, size_t chunks, uint32_t rounds,
                           void* buckets, void* head, void* tail, cudaStream_t st, int* launches)
{
    if (rounds == 0 || L == 0 || L > 0xffffu) return cudaErrorInvalidValue;
    const uint32_t grid = div_up(chunks, kAffThreads);
    const AffSlices S = aff_slices(L, grid);
    constexpr uint32_t kGroups = kAffThreads / kAffGroup;      // per block
    AffArgs A[2];
    cudaStream_t sts[2] = {st, W.aux.stream};
    for (int h = 0; h < 2; h++) {
        const AffWork::Set& w = W.set[h];
        A[h].pts = (const affine*)pts;
        A[h].sorted_pt = sorted_pt;
        A[h].sorted_key = sorted_key;
        A[h].total_ptr = total;
        A[h].L = L;
        A[h].least = least;
        A[h].T = (size_t)S.blocks * kAffThreads;
        A[h].list_pts[0] = (affine*)w.pts0.p;
        A[h].list_pts[1] = (affine*)w.pts1.p;
        A[h].list_key[0] = (uint32_t*)w.key0.p;
        A[h].list_key[1] = (uint32_t*)w.key1.p;
        A[h].meta = (uint32_t*)w.meta.p;
        A[h].pairpos = (uint32_t*)w.pairpos.p;
        A[h].prefix = (fp*)w.prefix.p;
        A[h].rest = (fp*)w.rest.p;
        A[h].gtot = (fp*)w.gtot.p;
        A[h].buckets = (xyzz*)buckets;
        A[h].head = (xyzz*)head;
        A[h].tail = (xyzz*)tail;
        A[h].slice = 0;
        A[h].slices = S.count;
    }
    // The mixed additions of all entries, where there are too few for the rounds; an empty
    // launch otherwise.  (On the second stream instead: 2^20 points 5.53 -> 5.55 ms, and sparse
    // scalars up to 12% slower, behind the rounds' launches that leave at once.)
    if (least) {
        k_accumulate<<<div_up(chunks, 128), 128, 0, st>>>((const affine*)pts, sorted_pt, sorted_key, total, least, L,
                                                          (xyzz*)buckets, (xyzz*)head, (xyzz*)tail);
        ++*launches;
    }
    if (S.count > 1) CATMSM_CHECK(W.aux.begin(st));
    for (uint32_t s0 = 0; s0 < S.count; s0 += 2) {
        uint32_t nblk[2];
        for (uint32_t h = 0; h < 2; h++) {
            A[h].slice = s0 + h;
            nblk[h] = s0 + h < grid ? (grid - (s0 + h) + S.count - 1) / S.count : 0;
            if (!nblk[h]) continue;
            k_aff_first<<<nblk[h], kAffThreads, 0, sts[h]>>>(A[h]);
            ++*launches;
        }
        for (uint32_t r = 1; r <= rounds; r++) {
            const bool first = r == 1, last = r == rounds;
            for (uint32_t h = 0; h < 2; h++)
                if (nblk[h]) k_aff_invert<<<div_up(nblk[h] * kGroups, 32), 32, 0, sts[h]>>>(A[h], nblk[h] * kGroups);
            for (uint32_t h = 0; h < 2; h++) {
                if (!nblk[h]) continue;
                if (first && last) k_aff_round<true, true><<<nblk[h], kAffThreads, 0, sts[h]>>>(A[h], r);
                else if (first) k_aff_round<true, false><<<nblk[h], kAffThreads, 0, sts[h]>>>(A[h], r);
                else if (last) k_aff_round<false, true><<<nblk[h], kAffThreads, 0, sts[h]>>>(A[h], r);
                else k_aff_round<false, false><<<nblk[h], kAffThreads, 0, sts[h]>>>(A[h], r);
                *launches += 2;
            }
        }
    }
    CATMSM_CHECK(cudaGetLastError());
    return S.count > 1 ? W.aux.end(st) : cudaSuccess;
}

}  // namespace catmsm
