// G1 point arithmetic on sm_103a (y^2 = x^3 + 4 over Fp).
//
// Representations:
//   affine  {x, y}            96 B, all-zero = infinity (blst_p1_affine,
//                             bindings/blst_types.h:101)
//   jacobian{x, y, z}         144 B, z == 0 = infinity (blst_p1, :99)
//   xyzz    {x, y, zz, zzz}   x = X/ZZ, y = Y/ZZZ, ZZ^3 = ZZZ^2; zz == 0 =
//                             infinity.  Same coordinates the reference uses
//                             for its Pippenger buckets (scalar/curve/point.cpp
//                             :1939-2113).
// Formulas are the public explicit-formulas-database ones for a = 0:
//   xyzz madd-2008-s / mdbl-2008-s / add-2008-s / dbl-2008-s,
//   jacobian dbl-2009-l and add-2007-bl (with explicit special cases).
// Every addition handles infinity, doubling and opposite inputs, so the group
// law is complete and results are exact for any points on the curve.
#pragma once
#include "field.cuh"

namespace catmsm {

struct affine { fp x, y; };
struct jac { fp x, y, z; };
struct xyzz { fp x, y, zz, zzz; };

// Vectorised global loads and stores of points (16-byte aligned rows).
__device__ __forceinline__ void load_affine(fp& x, fp& y, const affine* p)
{
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 v[6];
#pragma unroll
    for (int k = 0; k < 6; k++) v[k] = __ldg(q + k);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        x.v[4 * k + 0] = v[k].x; x.v[4 * k + 1] = v[k].y;
        x.v[4 * k + 2] = v[k].z; x.v[4 * k + 3] = v[k].w;
        y.v[4 * k + 0] = v[k + 3].x; y.v[4 * k + 1] = v[k + 3].y;
        y.v[4 * k + 2] = v[k + 3].z; y.v[4 * k + 3] = v[k + 3].w;
    }
}

__device__ __forceinline__ void store_xyzz(xyzz* dst, const xyzz& p)
{
    uint4* q = reinterpret_cast<uint4*>(dst);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&p);
#pragma unroll
    for (int k = 0; k < 12; k++) q[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
}

__device__ __forceinline__ void store_affine(affine* dst, const affine& p)
{
    uint4* q = reinterpret_cast<uint4*>(dst);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&p);
#pragma unroll
    for (int k = 0; k < 6; k++) q[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
}

__device__ __forceinline__ void load_xyzz(xyzz& p, const xyzz* src)
{
    const uint4* q = reinterpret_cast<const uint4*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&p);
#pragma unroll
    for (int k = 0; k < 12; k++) {
        uint4 v = q[k];
        d[4 * k] = v.x; d[4 * k + 1] = v.y; d[4 * k + 2] = v.z; d[4 * k + 3] = v.w;
    }
}

__device__ __forceinline__ bool aff_is_inf(const affine& a)
{
    return fp_is_zero_raw(a.x) && fp_is_zero_raw(a.y);
}

__device__ __forceinline__ void xyzz_set_inf(xyzz& p)
{
    fp_zero(p.x); fp_zero(p.y); fp_zero(p.zz); fp_zero(p.zzz);
}

__device__ __forceinline__ bool xyzz_is_inf(const xyzz& p) { return fp_is_zero(p.zz); }

// p = 2 * (ax, ay) for an affine point (mdbl-2008-s)
__device__ __forceinline__ void xyzz_dbl_affine(xyzz& p, const fp& ax, const fp& ay)
{
    fp U, V, W, S, M, t;
    fp_dbl(U, ay);
    fp_sqr(V, U);
    fp_mul(W, V, U);
    fp_mul(S, ax, V);
    fp_sqr(M, ax);
    fp_dbl(t, M);
    fp_add(M, t, M);
    fp_sqr(t, M);
    fp_sub(t, t, S);
    fp_sub(p.x, t, S);
    fp_sub(t, S, p.x);
    fp_neg(S, ay);
    fp_mul2(p.y, M, t, W, S);     // Y3 = M (S - X3) - W y, one reduction
    p.zz = V;
    p.zzz = W;
}

// p += (ax, +/-ay)   (madd-2008-s, 8M + 2S); ay already carries the sign
__device__ __forceinline__ void xyzz_madd(xyzz& p, const fp& ax, const fp& ay)
{
    if (xyzz_is_inf(p)) {
        p.x = ax; p.y = ay;
        fp_set_one(p.zz); fp_set_one(p.zzz);
        return;
    }
    fp P, R;
    fp_mul(P, ax, p.zz);
    fp_sub(P, P, p.x);
    fp_mul(R, ay, p.zzz);
    fp_sub(R, R, p.y);
    if (fp_is_zero(P)) {
        if (fp_is_zero(R)) xyzz_dbl_affine(p, ax, ay);
        else xyzz_set_inf(p);
        return;
    }
    fp PP, PPP, Q;
    fp_sqr(PP, P);
    fp_mul(PPP, PP, P);
    fp_mul(p.zz, p.zz, PP);
    fp_mul(p.zzz, p.zzz, PPP);
    fp_mul(Q, p.x, PP);
    fp_sqr(P, R);                 // P := R^2
    fp_sub(P, P, PPP);
    fp_sub(P, P, Q);
    fp_sub(p.x, P, Q);            // X3 = R^2 - PPP - 2Q
    fp_sub(Q, Q, p.x);
    fp_neg(PPP, PPP);
    fp_mul2(p.y, Q, R, p.y, PPP); // Y3 = R (Q - X3) - Y1 PPP, one reduction
}

// p = 2p (dbl-2008-s)
__device__ __forceinline__ void xyzz_dbl(xyzz& p)
{
    if (xyzz_is_inf(p)) return;
    fp U, V, W, S, M, t;
    fp_dbl(U, p.y);
    fp_sqr(V, U);
    fp_mul(W, V, U);
    fp_mul(S, p.x, V);
    fp_sqr(M, p.x);
    fp_dbl(t, M);
    fp_add(M, t, M);
    fp_mul(p.zz, p.zz, V);
    fp_mul(p.zzz, p.zzz, W);
    fp_sqr(t, M);
    fp_sub(t, t, S);
    fp_sub(p.x, t, S);
    fp_sub(t, S, p.x);
    fp_neg(W, W);
    fp_mul2(p.y, M, t, W, p.y);   // Y3 = M (S - X3) - W Y1, one reduction
}

// p += q (add-2008-s, 12M + 2S)
__device__ __forceinline__ void xyzz_add(xyzz& p, const xyzz& q)
{
    if (xyzz_is_inf(q)) return;
    if (xyzz_is_inf(p)) { p = q; return; }
    fp U1, S1, P, R;
    fp_mul(U1, p.x, q.zz);
    fp_mul(P, q.x, p.zz);
    fp_sub(P, P, U1);
    fp_mul(S1, p.y, q.zzz);
    fp_mul(R, q.y, p.zzz);
    fp_sub(R, R, S1);
    if (fp_is_zero(P)) {
        if (fp_is_zero(R)) xyzz_dbl(p);
        else xyzz_set_inf(p);
        return;
    }
    fp PP, PPP;
    fp_sqr(PP, P);
    fp_mul(PPP, PP, P);
    fp_mul(p.zz, p.zz, q.zz);
    fp_mul(p.zz, p.zz, PP);
    fp_mul(p.zzz, p.zzz, q.zzz);
    fp_mul(p.zzz, p.zzz, PPP);
    fp_mul(U1, U1, PP);           // Q = U1 PP
    fp_sqr(P, R);
    fp_sub(P, P, PPP);
    fp_sub(P, P, U1);
    fp_sub(p.x, P, U1);
    fp_sub(U1, U1, p.x);
    fp_neg(PPP, PPP);
    fp_mul2(p.y, U1, R, S1, PPP); // Y3 = R (Q - X3) - S1 PPP, one reduction
}

// d = p - q, p += q, sharing everything but the two R's (12M + 3S for both
// against 24M + 4S); exceptional operands take the general additions.
__device__ __forceinline__ void xyzz_add_sub(xyzz& p, xyzz& d, const xyzz& q)
{
    fp U1, S1, P, S2;
    fp_mul(U1, p.x, q.zz);
    fp_mul(P, q.x, p.zz);
    fp_sub(P, P, U1);
    if (xyzz_is_inf(p) || xyzz_is_inf(q) || fp_is_zero(P)) {
        xyzz n = q;
        fp_neg(n.y, n.y);
        d = p;
        xyzz_add(d, n);
        xyzz_add(p, q);
        return;
    }
    fp_mul(S1, p.y, q.zzz);
    fp_mul(S2, q.y, p.zzz);
    fp PP, PPP, t, R;
    fp_sqr(PP, P);
    fp_mul(PPP, PP, P);
    fp_mul(t, p.zz, q.zz);
    fp_mul(p.zz, t, PP);
    fp_mul(t, p.zzz, q.zzz);
    fp_mul(p.zzz, t, PPP);
    d.zz = p.zz;
    d.zzz = p.zzz;
    fp_mul(U1, U1, PP);           // Q = U1 PP
    fp_neg(P, PPP);
    fp_sub(P, P, U1);
    fp_sub(P, P, U1);             // -PPP - 2Q
    fp_neg(PPP, PPP);
    fp_sub(R, S2, S1);
    fp_sqr(t, R);
    fp_add(p.x, t, P);
    fp_sub(t, U1, p.x);
    fp_mul2(p.y, t, R, S1, PPP);  // Y3 = R (Q - X3) - S1 PPP
    fp_add(R, S2, S1);
    fp_neg(R, R);
    fp_sqr(t, R);
    fp_add(d.x, t, P);
    fp_sub(t, U1, d.x);
    fp_mul2(d.y, t, R, S1, PPP);
}

// Jacobian (X, Y, Z) = (x*zz, y*zzz, zz); reference point.cpp:2109
__device__ __forceinline__ void xyzz_to_jac(jac& o, const xyzz& p)
{
    if (xyzz_is_inf(p)) {
        fp_zero(o.x); fp_zero(o.y); fp_zero(o.z);
        return;
    }
    fp_mul(o.x, p.x, p.zz);
    fp_mul(o.y, p.y, p.zzz);
    o.z = p.zz;
}

// xyzz from Jacobian: zz = Z^2, zzz = Z^3
__device__ __forceinline__ void jac_to_xyzz(xyzz& o, const jac& p)
{
    if (fp_is_zero(p.z)) { xyzz_set_inf(o); return; }
    o.x = p.x;
    o.y = p.y;
    fp_sqr(o.zz, p.z);
    fp_mul(o.zzz, o.zz, p.z);
}

// Affine normalisation of an xyzz point: x = X / ZZ, y = Y / ZZZ.
// 1/ZZ and 1/ZZZ come from one inversion of ZZZ*ZZ... via (ZZ*ZZZ)^-1.
__device__ __forceinline__ void xyzz_to_affine(affine& o, const xyzz& p)
{
    if (xyzz_is_inf(p)) { fp_zero(o.x); fp_zero(o.y); return; }
    fp t, inv;
    fp_mul(t, p.zz, p.zzz);
    fp_inv(inv, t);
    fp_mul(t, inv, p.zzz);        // 1/ZZ
    fp_mul(o.x, p.x, t);
    fp_mul(t, inv, p.zz);         // 1/ZZZ
    fp_mul(o.y, p.y, t);
    fp_canon(o.x, o.x);
    fp_canon(o.y, o.y);
}


// ---------------------------------------------------------------- Jacobian
__device__ __forceinline__ bool jac_is_inf(const jac& p) { return fp_is_zero(p.z); }

__device__ __forceinline__ void jac_set_inf(jac& p) { fp_zero(p.x); fp_zero(p.y); fp_zero(p.z); }

// dbl-2009-l (a = 0): 2M + 5S
__device__ __forceinline__ void jac_dbl(jac& p)
{
    if (jac_is_inf(p)) return;
    fp A, B, C, D, E, t;
    fp_sqr(A, p.x);
    fp_sqr(B, p.y);
    fp_sqr(C, B);
    fp_add(t, p.x, B);
    fp_sqr(t, t);
    fp_sub(t, t, A);
    fp_sub(t, t, C);
    fp_dbl(D, t);
    fp_dbl(E, A);
    fp_add(E, E, A);
    fp_mul(p.z, p.y, p.z);
    fp_dbl(p.z, p.z);
    fp_sqr(t, E);
    fp_sub(t, t, D);
    fp_sub(p.x, t, D);
    fp_sub(t, D, p.x);
    fp_mul(t, E, t);
    fp_dbl(C, C);
    fp_dbl(C, C);
    fp_dbl(C, C);
    fp_sub(p.y, t, C);
}

// GLV endomorphism of G1: phi(x, y) = (beta x, y) = lambda (x, y) for
// lambda = z^2 - 1 = 0xac45a4010001a40200000000ffffffff (lambda^2 + lambda + 1 = r)
// and the cube root of unity beta below (Montgomery form).
__device__ __constant__ static const uint32_t FP_BETA[12] = {
    0x8671f071u, 0xcd03c9e4u, 0x1fcda5d2u, 0x5dab2246u, 0xd3851b95u, 0x587042afu,
    0x01bacb9eu, 0x8eb60ebeu, 0x83d050d2u, 0x03f97d6eu, 0x54638741u, 0x18f02065u};

// ---------------------------------------------------------------------------
// Quad point operations: four consecutive lanes (a quad) perform one XYZZ
// addition or doubling together, lane k holding coordinate k of a point (x, y,
// zz, zzz).  At each step every lane computes one product through the same
// fp_mul_call, so an addition is 4 dependent multiplications instead of ~11.5 and
// a doubling 3 instead of ~8: for chains of few point operations in few threads
// (the reduction's upper levels, carry joins, small transforms) latency, not
// multiplier throughput, is what costs.  The coordinates meet by xor shuffles:
// in the first step of an addition each lane multiplies its own coordinate by
// the other operand's coordinate two lanes over (X1 ZZ2, Y1 ZZZ2, ZZ1 X2, ZZZ1
// Y2), and every later product has at least one factor in its lane, so an
// addition shuffles 6 field elements (and picks 9 operands) where lanes holding
// whole points broadcast 14 and picked 8 four-way ones.  What bounds it now is the
// 1.9k cycles of a multiplication by a warp alone (a wide multiply-add every 6
// cycles: the carry chains are not interleaved).  50021-point MSM 0.855 -> 0.840 ms,
// 2^12 FFT 6.8 -> 6.2 ms.  All control flow depends on shuffled flags, so the four
// lanes stay converged; callers keep a quad's lanes together.
struct quad_lane {
    uint32_t k;      // position in the quad
    uint32_t mask;   // the quad's four lanes
};

__device__ __forceinline__ quad_lane quad_of(uint32_t lane)
{
    return quad_lane{lane & 3u, 0xfu << (lane & 28u)};
}

__device__ __forceinline__ fp fp_bcast(const fp& v, int src, const quad_lane& q)
{
    fp r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = __shfl_sync(q.mask, v.v[i], src, 4);
    return r;
}

__device__ __forceinline__ fp fp_swap(const fp& v, int lanes, const quad_lane& q)
{
    fp r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = __shfl_xor_sync(q.mask, v.v[i], lanes, 4);
    return r;
}

// c ? b : a, word by word without a branch
__device__ __forceinline__ fp fp_sel(const fp& a, const fp& b, bool c)
{
    const uint32_t m = 0u - (uint32_t)c;
    fp r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = (a.v[i] & ~m) | (b.v[i] & m);
    return r;
}

// Lane `src`'s flag.
__device__ __forceinline__ bool quad_flag(bool f, int src, const quad_lane& q)
{
    return __shfl_sync(q.mask, (int)f, src, 4) != 0;
}

// Coordinate k of a point in memory (16-byte aligned), as its owner lane holds it.
__device__ __forceinline__ fp qd_load(const xyzz* p, uint32_t k)
{
    const uint4* s = reinterpret_cast<const uint4*>(p) + 3 * k;
    fp r;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const uint4 v = s[i];
        r.v[4 * i] = v.x; r.v[4 * i + 1] = v.y; r.v[4 * i + 2] = v.z; r.v[4 * i + 3] = v.w;
    }
    return r;
}

__device__ __forceinline__ void qd_store(xyzz* p, const fp& d, const quad_lane& q)
{
    uint4* s = reinterpret_cast<uint4*>(p) + 3 * q.k;
#pragma unroll
    for (int i = 0; i < 3; i++) s[i] = make_uint4(d.v[4 * i], d.v[4 * i + 1], d.v[4 * i + 2], d.v[4 * i + 3]);
}

// The point at infinity has zz = 0 (lane 2).
__device__ __forceinline__ bool qd_is_inf(const fp& d, const quad_lane& q) { return quad_flag(fp_is_zero(d), 2, q); }

// dbl-2008-s: X^2, U^2 | X V, U V, ZZ V, M^2 | M (S - X3), W Y, -, ZZZ W
__device__ __forceinline__ void qd_dbl(fp& d, const quad_lane& q)
{
    if (qd_is_inf(d, q)) return;
    fp U, M, t;
    fp_dbl(U, d);                                          // lane 1: U = 2Y
    const fp u = fp_sel(d, U, q.k == 1);
    fp r = fp_mul_call(u, u);                              // lane 0: X^2, lane 1: V
    fp_dbl(t, r);
    fp_add(M, t, r);                                       // lane 0: M
    const fp V = fp_bcast(r, 1, q);
    M = fp_bcast(M, 0, q);
    const bool l3 = q.k == 3;
    r = fp_mul_call(fp_sel(u, M, l3), fp_sel(V, M, l3));   // S, W, ZZ3, M^2
    const fp zz = r;
    const fp MM = fp_bcast(r, 3, q), W = fp_bcast(r, 1, q);
    fp X3;
    fp_sub(t, MM, r);
    fp_sub(X3, t, r);                                      // lane 0: M^2 - 2S
    fp_sub(t, r, X3);
    r = fp_mul_call(fp_sel(d, M, q.k == 0), fp_sel(W, t, q.k == 0));   // M (S - X3), Y W, -, ZZZ W
    fp_sub(t, fp_swap(r, 1, q), r);                        // lane 1: Y3
    d = fp_sel(fp_sel(fp_sel(r, X3, q.k == 0), t, q.k == 1), zz, q.k == 2);
}

// The last three steps of an addition.  PR: lanes 0, 2: P, lanes 1, 3: R; f: the
// first operand's U1, S1 (lanes 0, 1) and ZZ1 ZZ2, ZZZ1 ZZZ2 (lanes 2, 3: Mixed,
// the operands' own zz, zzz; otherwise d times e here):
//   P^2, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2 | U1 PP, P PP, ZZ PP, P PP | R (Q - X3), S1 PPP, -, ZZZ PPP
template <bool Mixed>
__device__ __forceinline__ fp qd_add_core(const fp& PR, const fp& f, const fp& d, const fp& e, const quad_lane& q)
{
    const bool lo = q.k < 2;
    fp r = Mixed ? fp_mul_call(PR, PR) : fp_mul_call(fp_sel(d, PR, lo), fp_sel(e, PR, lo));
    const fp PP = fp_bcast(r, 0, q), other = fp_swap(PR, 1, q);       // even lanes: R, odd lanes: P
    const fp T = Mixed ? f : fp_sel(r, f, lo);                        // U1, S1, ZZ1 ZZ2, ZZZ1 ZZZ2
    const fp s = fp_mul_call(fp_sel(T, other, (q.k & 1) != 0), PP);   // Q, PPP, ZZ3, PPP
    fp t, X3, v;
    fp_sub(t, r, s);                                                  // lane 1: RR - PPP
    v = fp_swap(t, 1, q);
    fp_sub(t, v, s);
    fp_sub(X3, t, s);                                                 // lane 0: RR - PPP - 2Q
    fp_sub(t, s, X3);                                                 // lane 0: Q - X3
    r = fp_mul_call(fp_sel(T, other, q.k == 0), fp_sel(s, t, q.k == 0));   // R (Q - X3), S1 PPP, -, ZZZ3
    fp_sub(t, fp_swap(r, 1, q), r);                                   // lane 1: Y3
    return fp_sel(fp_sel(fp_sel(r, X3, q.k == 0), t, q.k == 1), s, q.k == 2);
}

// d += e (add-2008-s)
__device__ __forceinline__ void qd_add(fp& d, const fp& e, const quad_lane& q)
{
    if (qd_is_inf(e, q)) return;
    if (qd_is_inf(d, q)) {
        d = e;
        return;
    }
    const fp r = fp_mul_call(d, fp_swap(e, 2, q));         // U1, S1, U2, S2
    const fp o = fp_swap(r, 2, q);
    const bool lo = q.k < 2;
    fp PR;
    fp_sub(PR, fp_sel(r, o, lo), fp_sel(o, r, lo));        // lanes 0, 2: U2 - U1, lanes 1, 3: S2 - S1
    const bool z = fp_is_zero(PR);
    if (quad_flag(z, 0, q)) {
        if (quad_flag(z, 1, q)) {
            qd_dbl(d, q);
        } else {
            fp_zero(d);
        }
        return;
    }
    d = qd_add_core<false>(PR, r, d, e, q);
}

// d = an affine point (not infinity): lane k passes coordinate k mod 2 of it.
__device__ __forceinline__ void qd_set_affine(fp& d, const fp& a, const quad_lane& q)
{
    fp one;
    fp_set_one(one);
    d = fp_sel(a, one, q.k >= 2);
}

// The differences P (even lanes: the ratio of the sum's z to d's) and R (odd lanes).
__device__ __forceinline__ fp qd_madd_diff(const fp& d, const fp& a, const quad_lane& q)
{
    const fp r = fp_sel(fp_mul_call(d, a), d, q.k < 2);    // X1, Y1, U2, S2
    const fp o = fp_swap(r, 2, q);
    fp PR;
    fp_sub(PR, fp_sel(r, o, q.k < 2), fp_sel(o, r, q.k < 2));
    return PR;
}

// d += an affine point, as above: madd-2008-s with the complete special cases.
__device__ __forceinline__ void qd_madd(fp& d, const fp& a, const quad_lane& q)
{
    if (qd_is_inf(d, q)) {
        qd_set_affine(d, a, q);
        return;
    }
    const fp PR = qd_madd_diff(d, a, q);
    const bool z = fp_is_zero(PR);
    if (quad_flag(z, 0, q)) {
        if (quad_flag(z, 1, q)) qd_dbl(d, q);
        else fp_zero(d);
        return;
    }
    d = qd_add_core<true>(PR, d, d, d, q);
}

}  // namespace catmsm
