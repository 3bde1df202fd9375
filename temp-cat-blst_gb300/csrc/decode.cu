// Batched point decoding and validation on sm_103a.
//
// Each element follows the reference's single-point semantics exactly:
//   uncompress   blst_p1_uncompress  (blst/c_api.cpp:1633 -> scalar/curve/
//                point.cpp:909-1001): compressed flag required; infinity only
//                as 0xc0 followed by zeros; top 3 bits of x cleared, x < p,
//                y = sqrt(x^3 + 4) (p = 3 mod 4: a^((p+1)/4)), sign flag picks
//                y or -y by "y > (p-1)/2"; x == 0 is the order-2-coset point
//                (0, +/-2) -> POINT_NOT_IN_GROUP.
//   deserialize  blst_p1_deserialize (c_api.cpp:1643 -> point.cpp:1007-1103):
//                no flags -> big-endian x, y < p, on the curve, x != 0;
//                compressed flag -> uncompress; infinity flag alone with zeros
//                -> infinity; anything else -> BAD_ENCODING.
//   in_g1        blst_p1_affine_in_g1 (c_api.cpp:1257 -> point.cpp:1182-1244):
//                on the curve and phi^2(P) == -z^2 P (Scott's endomorphism
//                test, eprint 2021/1130, proof El Housni et al. 2022/352
//                Prop. 4), z = -0xd201000000010000; infinity is a member.
// Failed elements keep the caller's output bytes.  A decode can optionally be
// followed by the membership test (POINT_NOT_IN_GROUP on failure).
#include "common.cuh"
#include "glv_mult.cuh"
#include "catmsm_internal.h"
#include "catmsm_gpu.h"

#include <algorithm>

namespace catmsm {

enum { kOk = 0, kBadEncoding = 1, kNotOnCurve = 2, kNotInGroup = 3 };

__device__ __constant__ static const uint32_t FP_R2[12] = {
    0x1c341746u, 0xf4df1f34u, 0x09d104f1u, 0x0a76e6a6u, 0x4c95b6d5u, 0x8de5476cu,
    0x939d83c0u, 0x67eb88a9u, 0xb519952du, 0x9a793e85u, 0x92cae3aau, 0x11988fe5u};
__device__ __constant__ static const uint32_t FP_FOUR[12] = {   // 4 (Montgomery)
    0x000cfff3u, 0xaa270000u, 0xfc34000au, 0x53cc0032u, 0x6b0a807fu, 0x478fe97au,
    0xe6ba24d7u, 0xb1d37ebeu, 0xbf78ab2fu, 0x8ec9733bu, 0x3d83de7eu, 0x09d64551u};
__device__ __constant__ static const uint32_t FP_SQRT_E[12] = { // (p + 1) / 4
    0xffffeaabu, 0xee7fbfffu, 0xac54ffffu, 0x07aaffffu, 0x3dac3d89u, 0xd9cc34a8u,
    0x3ce144afu, 0xd91dd2e1u, 0x90d2eb35u, 0x92c6e9edu, 0x8e5ff9a6u, 0x0680447au};
__device__ __constant__ static const uint32_t FP_HALF[12] = {   // (p - 1) / 2
    0xffffd555u, 0xdcff7fffu, 0x58a9ffffu, 0x0f55ffffu, 0x7b587b12u, 0xb3986950u,
    0x79c2895fu, 0xb23ba5c2u, 0x21a5d66bu, 0x258dd3dbu, 0x1cbff34du, 0x0d0088f5u};

__device__ __forceinline__ void fp_from_be(fp& r, const uint8_t* b)
{
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const uint8_t* q = b + 44 - 4 * k;
        r.v[k] = ((uint32_t)q[0] << 24) | ((uint32_t)q[1] << 16) | ((uint32_t)q[2] << 8) | q[3];
    }
}

// a < b as 384-bit integers
__device__ __forceinline__ bool lt384(const fp& a, const uint32_t* b)
{
    for (int k = 11; k >= 0; k--)
        if (a.v[k] != b[k]) return a.v[k] < b[k];
    return false;
}

__device__ __forceinline__ bool eq_canon(const fp& a, const fp& b)
{
    fp x, y;
    fp_canon(x, a);
    fp_canon(y, b);
    uint32_t d = 0;
#pragma unroll
    for (int k = 0; k < 12; k++) d |= x.v[k] ^ y.v[k];
    return d == 0;
}

__device__ __forceinline__ void load_const(fp& r, const uint32_t* c)
{
#pragma unroll
    for (int k = 0; k < 12; k++) r.v[k] = c[k];
}

// y^2 == x^3 + 4 (Montgomery inputs)
__device__ __forceinline__ bool on_curve_xy(const fp& x, const fp& y)
{
    fp yy, xxx, four;
    fp_sqr(yy, y);
    fp_sqr(xxx, x);
    fp_mul(xxx, xxx, x);
    load_const(four, FP_FOUR);
    fp_add(xxx, xxx, four);
    return eq_canon(yy, xxx);
}

// canonical integer of a Montgomery value > (p - 1) / 2
__device__ __forceinline__ bool is_large(const fp& y)
{
    fp one, t;
    fp_zero(one);
    one.v[0] = 1;
    fp_mul(t, y, one);
    fp_canon(t, t);
    for (int k = 11; k >= 0; k--)
        if (t.v[k] != FP_HALF[k]) return t.v[k] > FP_HALF[k];
    return false;
}

__device__ int uncompress48(affine& out, const uint8_t* in)
{
    const uint8_t in0 = in[0];
    if ((in0 & 0x80) == 0) return kBadEncoding;
    if (in0 & 0x40) {
        uint32_t z = in0 & 0x3f;
        for (int i = 1; i < 48; i++) z |= in[i];
        if (z) return kBadEncoding;
        fp_zero(out.x);
        fp_zero(out.y);
        return kOk;
    }
    fp x;
    fp_from_be(x, in);
    x.v[11] &= 0x1fffffffu;                       // top 3 bits carry flags
    if (!lt384(x, FP_P)) return kBadEncoding;
    fp r2;
    load_const(r2, FP_R2);
    fp_mul(x, x, r2);
    fp a, four, y;
    fp_sqr(a, x);
    fp_mul(a, a, x);
    load_const(four, FP_FOUR);
    fp_add(a, a, four);
    fp_pow(y, a, FP_SQRT_E);
    fp yy;
    fp_sqr(yy, y);
    if (!eq_canon(yy, a)) return kNotOnCurve;
    const bool want = (in0 & 0x20) != 0;
    if (is_large(y) != want) fp_neg(y, y);
    fp_canon(x, x);
    fp_canon(y, y);
    if (fp_is_zero_raw(x)) return kNotInGroup;
    out.x = x;
    out.y = y;
    return kOk;
}

__device__ int deserialize96(affine& out, const uint8_t* in)
{
    const uint8_t in0 = in[0];
    if ((in0 & 0xe0) == 0) {
        fp x, y;
        fp_from_be(x, in);
        fp_from_be(y, in + 48);
        if (!lt384(x, FP_P) || !lt384(y, FP_P)) return kBadEncoding;
        fp r2;
        load_const(r2, FP_R2);
        fp_mul(x, x, r2);
        fp_mul(y, y, r2);
        fp_canon(x, x);
        fp_canon(y, y);
        const bool inf = fp_is_zero_raw(x) && fp_is_zero_raw(y);
        if (!inf && !on_curve_xy(x, y)) return kNotOnCurve;
        if (fp_is_zero_raw(x)) return kNotInGroup;
        out.x = x;
        out.y = y;
        return kOk;
    }
    if (in0 & 0x80) return uncompress48(out, in);
    if (in0 & 0x40) {
        uint32_t z = in0 & 0x3f;
        for (int i = 1; i < 96; i++) z |= in[i];
        if (z) return kBadEncoding;
        fp_zero(out.x);
        fp_zero(out.y);
        return kOk;
    }
    return kBadEncoding;
}

// Whether a point of the curve is in G1: phi^2(P) == -z^2 P.  Both products by |z|
// add an affine point: the second reads |z| P = (X, Y, Z) as the affine (X, Y) of
// the curve scaled by Z and multiplies its result's z by Z.  What bounds it: 126
// doublings, more than half of a checked decode's work.
__device__ __forceinline__ bool in_subgroup(const affine& a)
{
    if (fp_is_zero_raw(a.x) && fp_is_zero_raw(a.y)) return true;
    jac t0, t1;
    times_abs_z(t0, a.x, a.y);
    if (jac_is_inf(t0)) return false;                       // phi^2(P) is finite
    times_abs_z(t1, t0.x, t0.y);
    if (jac_is_inf(t1)) return false;
    fp_mul(t1.z, t1.z, t0.z);                               // z^2 P
    // phi^2(P) = (beta^2 x, y) vs -t1 = (X, -Y, Z): X == beta^2 x Z^2, -Y == y Z^3
    fp b2, zz, t;
    load_const(b2, FP_BETA2);
    fp_sqr(zz, t1.z);
    fp_mul(t, a.x, b2);
    fp_mul(t, t, zz);
    if (!eq_canon(t, t1.x)) return false;
    fp_mul(zz, zz, t1.z);
    fp_mul(t, a.y, zz);
    fp_neg(t1.y, t1.y);
    return eq_canon(t, t1.y);
}

// The same by a quad, every lane with the same point.
__device__ __forceinline__ bool in_subgroup_quad(const affine& a, const quad_lane& q)
{
    if (fp_is_zero_raw(a.x) && fp_is_zero_raw(a.y)) return true;
    const bool odd = (q.k & 1) != 0;
    fp t0, t1;
    qd_times_abs_z(t0, fp_sel(a.x, a.y, odd), q);
    if (qd_is_inf(t0, q)) return false;
    const fp base = fp_swap(t0, 2, q);                      // lanes 2, 3: X, Y
    qd_times_abs_z(t1, fp_sel(base, t0, q.k < 2), q);
    if (qd_is_inf(t1, q)) return false;
    fp b2, t;
    load_const(b2, FP_BETA2);
    fp_mul(b2, a.x, b2);
    t = fp_mul_call(t1, t0);                                // lanes 2, 3: zz, zzz of z^2 P
    t = fp_mul_call(fp_sel(b2, a.y, odd), t);               // beta^2 x ZZ, y ZZZ
    t = fp_swap(t, 2, q);
    if (q.k == 1) fp_neg(t, t);
    const bool eq = q.k >= 2 || eq_canon(t, t1);            // X, -Y
    return quad_flag(eq, 0, q) && quad_flag(eq, 1, q);
}

constexpr int kLaneThreads = 64, kLaneBlocks = 8;    // one lane an element: four warps per scheduler

// mode 0: uncompress (48-byte elements), 1: deserialize (96).  Points go to `pts`
// (which may be `in`, element over element) and codes to errs.  A kernel of its
// own, so that the squarings of the square root can be inlined in its loop
// without the membership test's code growing past the instruction cache: 300000
// checked elements 13.76 -> 13.57 ms (14.33 with the squarings inlined in both).
__global__ void __launch_bounds__(kLaneThreads, kLaneBlocks) k_decode(const uint8_t* in, uint32_t n, int mode,
                                                                      affine* pts, int32_t* __restrict__ errs)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    affine a;
    const int err = mode == 0 ? uncompress48(a, in + 48 * (size_t)i) : deserialize96(a, in + 96 * (size_t)i);
    if (err == kOk) pts[i] = a;
    errs[i] = err;
}

// Membership.  Decoded points (result false): the points of `pts` whose code is
// kOk go to `out` or change the code.  Otherwise errs is the result, 1 for a
// member, and a point may be off the curve.
// Quad: four lanes an element, for calls that do not fill the GPU: they last as
// long as one element's chain, whose doublings a quad does in half the time.
// 2111 checked elements: 1.50 -> 0.92 ms.  A full launch keeps one lane: 77824
// checked elements (one wave) 3.58 ms, the multiply pipe 88% busy.
template <bool Quad>
__global__ void __launch_bounds__(Quad ? 128 : kLaneThreads, Quad ? 2 : kLaneBlocks) k_members(const affine* __restrict__ pts, uint32_t n,
                                                                           bool result, affine* __restrict__ out,
                                                                           int32_t* __restrict__ errs)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t i = Quad ? t >> 2 : t;
    if (i >= n) return;
    const quad_lane q = quad_of(threadIdx.x & 31);
    if (!result && errs[i] != kOk) return;
    const affine a = pts[i];
    bool ok = true;
    if (result) ok = (fp_is_zero_raw(a.x) && fp_is_zero_raw(a.y)) || on_curve_xy(a.x, a.y);
    if (ok) ok = Quad ? in_subgroup_quad(a, q) : in_subgroup(a);
    if (Quad) __syncwarp(q.mask);
    if (Quad && q.k != 0) return;
    if (result) {
        errs[i] = ok ? 1 : 0;
        return;
    }
    if (ok) out[i] = a;
    else errs[i] = kNotInGroup;
}

// Elements up to which the membership test takes quads: one wave of them.
constexpr size_t kQuadBlocksPerSm = 2;

// Elements [lo, lo + m) of a call, on one stream.
struct DecodeSlice {
    const uint8_t* in;
    uint8_t* din;
    blst_p1_affine* out;
    affine *dout, *pts;
    int* errs;
    int32_t* derr;
    uint32_t m;
    cudaStream_t st;
};

static cudaError_t decode_upload(const DecodeSlice& s, size_t elem)
{
    if (s.din) CATMSM_CHECK(cudaMemcpyAsync(s.din, s.in, s.m * elem, cudaMemcpyHostToDevice, s.st));
    return cudaMemcpyAsync(s.dout, s.out, s.m * sizeof(affine), cudaMemcpyHostToDevice, s.st);
}

static cudaError_t decode_kernels(const DecodeSlice& s, int mode, bool check, bool quads)
{
    if (mode != 2) {
        k_decode<<<div_up(s.m, kLaneThreads), kLaneThreads, 0, s.st>>>(s.din, s.m, mode, s.pts, s.derr);
        g_stats.launches++;
        CATMSM_CHECK(cudaGetLastError());
    }
    if (check) {
        if (quads)
            k_members<true><<<div_up(4 * (size_t)s.m, 128), 128, 0, s.st>>>(s.pts, s.m, mode == 2, s.dout, s.derr);
        else
            k_members<false><<<div_up(s.m, kLaneThreads), kLaneThreads, 0, s.st>>>(s.pts, s.m, mode == 2, s.dout,
                                                                                   s.derr);
        g_stats.launches++;
        CATMSM_CHECK(cudaGetLastError());
    }
    return cudaSuccess;
}

static cudaError_t decode_download(const DecodeSlice& s, int mode)
{
    if (mode != 2) CATMSM_CHECK(cudaMemcpyAsync(s.out, s.dout, s.m * sizeof(affine), cudaMemcpyDeviceToHost, s.st));
    return cudaMemcpyAsync(s.errs, s.derr, s.m * sizeof(int32_t), cudaMemcpyDeviceToHost, s.st);
}

// More elements than one wave, with a square root or a membership test each, run as
// two halves on two streams: the kernels of
// one half fill the SMs that the last wave of the other's leave idle, and the
// second half's upload and the first one's download run beside kernels.  One
// stream -> two, checked uncompressing: 100003 elements 5.23 -> 4.95 ms, 200000
// 9.44 -> 9.02, 300000 13.59 -> 13.13.  Three or more slices queue behind their own
// streams' tails: 100003 elements 4.99 with three, 5.44 with four.  The caller's
// arrays are read to the end before any of them is written (they may overlap): the
// second stream starts after the first half's upload, and the first half's download
// waits for the second's upload.
static cudaError_t decode_halves(DecodeSlice* s, AuxStream& aux, size_t elem, int mode, bool check)
{
    CATMSM_CHECK(decode_upload(s[0], elem));
    CATMSM_CHECK(aux.begin(s[0].st));
    CATMSM_CHECK(decode_kernels(s[0], mode, check, false));
    CATMSM_CHECK(decode_upload(s[1], elem));
    CATMSM_CHECK(aux.end(s[0].st));
    CATMSM_CHECK(decode_kernels(s[1], mode, check, false));
    CATMSM_CHECK(decode_download(s[0], mode));
    return decode_download(s[1], mode);
}

static int decode_run(const uint8_t* in, size_t elem, int mode, size_t n, blst_p1_affine* out, int* errs,
                      int check_group)
{
    if (n == 0) return 0;
    if (!out || !errs || (mode != 2 && !in) || n > 0x7fffffffu) return (int)cudaErrorInvalidValue;
    Ctx* ctx = get_ctx();
    if (!ctx) return (int)cudaErrorInitializationError;
    cudaStream_t st = ctx->stream;
    AuxStream& aux = ctx->msm.aff.aux;
    const bool check = mode == 2 || check_group;
    uint8_t* din = mode == 2 ? nullptr : (uint8_t*)ctx->msm.scalars.get(n * elem);
    affine* dout = (affine*)ctx->msm.points.get(n * sizeof(affine));
    int32_t* derr = (int32_t*)ctx->msm.digits.get(n * 4);
    affine* pts = dout;                              // the decoded points, before the membership test:
    // without memory for all of them, the elements go through a smaller buffer in turn
    size_t piece = n;
    if (mode == 0 && check)
        while (!(pts = (affine*)ctx->msm.buckets.get(piece * sizeof(affine))) && piece > 4096) piece = (piece + 1) / 2;
    if (mode == 1 && check) pts = (affine*)din;      // each thread over its own 96 bytes
    if ((mode != 2 && !din) || !dout || !derr || !pts) return (int)cudaErrorMemoryAllocation;
    const size_t sms = (size_t)device_sms();
    // A deserialization without the membership test is its copies: 77825 elements
    // 184 us on one stream, 206 on two.
    const bool halves = n > kLaneThreads * kLaneBlocks * sms && (mode == 0 || check) && piece == n;
    const size_t cut = halves ? n / 2 / kLaneThreads * kLaneThreads : n;
    cudaError_t err = halves ? aux.ensure(st) : cudaSuccess;
    if (err == cudaSuccess) {
        DecodeSlice s[2];
        for (int k = 0; k < 2; k++) {
            const size_t lo = k ? cut : 0;
            s[k] = DecodeSlice{mode == 2 ? nullptr : in + lo * elem,
                               mode == 2 ? nullptr : din + lo * elem,
                               out + lo,
                               dout + lo,
                               pts + lo,
                               errs + lo,
                               derr + lo,
                               (uint32_t)(k ? n - cut : cut),
                               k ? aux.stream : st};
        }
        if (halves) {
            err = decode_halves(s, aux, elem, mode, check);
            const cudaError_t e = cudaStreamSynchronize(aux.stream);
            if (err == cudaSuccess) err = e;
        } else {
            err = decode_upload(s[0], elem);
            for (size_t lo = 0; lo < n && err == cudaSuccess; lo += piece) {
                DecodeSlice t = s[0];
                t.din = mode == 2 ? nullptr : t.din + lo * elem;
                t.dout += lo;
                t.derr += lo;
                t.m = (uint32_t)std::min(piece, n - lo);
                err = decode_kernels(t, mode, check, t.m <= kQuadBlocksPerSm * 32 * sms);
            }
            if (err == cudaSuccess) err = decode_download(s[0], mode);
        }
    }
    const cudaError_t e = cudaStreamSynchronize(st);
    return (int)(err == cudaSuccess ? e : err);
}

}  // namespace catmsm

using namespace catmsm;

extern "C" {

int catmsm_p1s_uncompress(blst_p1_affine* out, const blst_byte* in48, size_t n, int* errs, int check_group)
{
    return decode_run(in48, 48, 0, n, out, errs, check_group);
}

int catmsm_p1s_deserialize(blst_p1_affine* out, const blst_byte* in96, size_t n, int* errs, int check_group)
{
    return decode_run(in96, 96, 1, n, out, errs, check_group);
}

int catmsm_p1s_affine_in_g1(const blst_p1_affine* points, size_t n, int* results)
{
    return decode_run(nullptr, 96, 2, n, const_cast<blst_p1_affine*>(points), results, 0);
}

}  // extern "C"
