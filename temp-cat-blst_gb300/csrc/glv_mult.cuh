// Scalar multiplication of a variable G1 point by a GLV-split scalar
// k = k1 + lambda k2 (k1, k2 < 2^128): k P = k1 P + k2 phi(P).
//
// Both halves walk one chain of ~128 doublings and add multiples of P and of
// phi(P) from an 8-entry table.  What bounds it: in a full launch the multiply
// pipe (additions were half of the work), in a small one the chain.  The table is
// "effective affine": P is read as the affine point (X, Y) of the isomorphic
// curve y^2 = x^3 + 4 Z^6 (the a = 0 formulas never use the constant), the
// multiples are built with mixed additions, and their z ratios bring all of
// them to one common z without an inversion.  The main loop's additions are then
// mixed (8M + 3S) instead of general Jacobian ones (12M + 4S, about a third more), and the
// common z is multiplied in once at the end.  Inverting to real affine tables
// instead cost as much as it saved (a serial chain per thread).
//
// Points are XYZZ in and out: the next pass adds them without a square per
// addition, and the quad form (below) keeps them so throughout.
#pragma once
#include "curve.cuh"

namespace catmsm {

// Signed fixed 4-bit windows of a value below 2^128: 33 digits in [-7, 8].
// Lanes of a warp on different scalars add at the same positions.  Against 5-bit
// windows: ~61 additions instead of ~50 for a table of 8 entries instead of
// 16 (seven mixed additions and a rescaling each), the same work in total
// and half the local memory.
__device__ __forceinline__ void booth4_128(int8_t* d, const uint32_t* k)
{
    uint32_t carry = 0;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        int v = (int)(((k[i >> 3] >> (4 * (i & 7))) & 15u) + carry);
        carry = v > 8 ? 1u : 0u;
        d[i] = (int8_t)(v - (int)(carry << 4));
    }
    d[32] = (int8_t)carry;
}

// Width-5 NAF of a value below 2^128 (4 little-endian words): digits d_i in
// {0, +-1, +-3, ..., +-15} with value = sum_i d_i 2^i and at most one nonzero
// digit in any five consecutive positions (density ~1/6).  Returns the number
// of digits, at most 129: subtracting a negative digit can carry the value
// past 2^128 once, after which every step halves it.
__device__ __forceinline__ int wnaf5_128(int8_t* d, const uint32_t* k)
{
    uint32_t w0 = k[0], w1 = k[1], w2 = k[2], w3 = k[3], w4 = 0;
    int len = 0;
#pragma unroll 1
    for (int i = 0; i < 130 && (w0 | w1 | w2 | w3 | w4); i++) {
        int v = 0;
        if (w0 & 1u) {
            v = (int)(w0 & 31u);
            if (v > 16) v -= 32;
            if (v > 0) {
                w0 -= (uint32_t)v;                   // the low five bits are v: no borrow
            } else {
                uint64_t s = (uint64_t)w0 + (uint32_t)(-v);
                w0 = (uint32_t)s;
                s = (s >> 32) + w1; w1 = (uint32_t)s;
                s = (s >> 32) + w2; w2 = (uint32_t)s;
                s = (s >> 32) + w3; w3 = (uint32_t)s;
                w4 += (uint32_t)(s >> 32);
            }
        }
        d[i] = (int8_t)v;
        len = i + 1;
        w0 = (w0 >> 1) | (w1 << 31);
        w1 = (w1 >> 1) | (w2 << 31);
        w2 = (w2 >> 1) | (w3 << 31);
        w3 = (w3 >> 1) | (w4 << 31);
        w4 >>= 1;
    }
    return len;
}

// p += (ax, ay), Jacobian + affine (madd with the a = 0 special cases)
__device__ __forceinline__ void jac_madd(jac& p, const fp& ax, const fp& ay)
{
    if (jac_is_inf(p)) {
        p.x = ax; p.y = ay;
        fp_set_one(p.z);
        return;
    }
    fp zz, h, r, t;
    fp_sqr(zz, p.z);
    fp_mul(h, ax, zz);
    fp_sub(h, h, p.x);
    fp_mul(zz, zz, p.z);
    fp_mul(r, ay, zz);
    fp_sub(r, r, p.y);
    if (fp_is_zero(h)) {
        if (fp_is_zero(r)) jac_dbl(p);
        else jac_set_inf(p);
        return;
    }
    fp_mul(p.z, p.z, h);
    fp_sqr(t, h);
    fp_mul(zz, p.x, t);           // V = X1 HH
    fp_mul(t, t, h);              // HHH
    fp_sqr(h, r);
    fp_sub(h, h, t);
    fp_sub(h, h, zz);
    fp_sub(p.x, h, zz);           // X3 = R^2 - HHH - 2V
    fp_sub(zz, zz, p.x);
    fp_neg(t, t);
    fp_mul2(p.y, zz, r, p.y, t);  // Y3 = R (V - X3) - Y1 HHH, one reduction
}

// Eight multiples of the point with Jacobian x, y (z read as 1) on a common z:
// (tx[i], ty[i]) = (2i + 1) P (Odd) or (i + 1) P, and bx[i] = beta tx[i], the x
// of phi.  zg: the common z, zero if a multiple met an exceptional case (a
// point of small order).
template <bool Odd>
__device__ __forceinline__ void glv_table(fp* tx, fp* ty, fp* bx, fp& zg, const fp& X, const fp& Y)
{
    fp rat[8];                    // z of entry i over z of entry i - 1
    fp ax, ay, z, V, W, S, M, t;
    // 2 (X, Y) as xyzz_dbl_affine: zz = U^2, z = U = 2Y
    fp_dbl(z, Y);
    fp_sqr(V, z);
    fp_mul(W, V, z);
    fp_mul(S, X, V);
    fp_sqr(M, X);
    fp_dbl(t, M);
    fp_add(M, t, M);
    fp_sqr(t, M);
    fp_sub(t, t, S);
    fp_sub(t, t, S);              // x of 2P
    fp_sub(V, S, t);
    fp_mul(M, M, V);
    fp_mul(W, W, Y);
    fp_sub(M, M, W);              // y of 2P
    zg = z;
    fp x, y;
    int i0;
    if (Odd) {
        // on the curve scaled by U, 2P is affine and P = (X U^2, Y U^3)
        ax = t; ay = M;
        x = S; y = W;
        fp_set_one(z);
        i0 = 1;
    } else {
        ax = X; ay = Y;
        tx[0] = X; ty[0] = Y;
        rat[1] = z;
        x = t; y = M;
        i0 = 2;
    }
    tx[i0 - 1] = x; ty[i0 - 1] = y;
#pragma unroll 1
    for (int i = i0; i < 8; i++) {
        fp zz, h, r;
        fp_sqr(zz, z);
        fp_mul(h, ax, zz);
        fp_sub(h, h, x);
        fp_mul(zz, zz, z);
        fp_mul(r, ay, zz);
        fp_sub(r, r, y);
        fp_mul(z, z, h);
        rat[i] = h;
        fp_sqr(t, h);
        fp_mul(zz, x, t);
        fp_mul(t, t, h);
        fp_sqr(h, r);
        fp_sub(h, h, t);
        fp_sub(h, h, zz);
        fp_sub(x, h, zz);
        fp_sub(zz, zz, x);
        fp_neg(t, t);
        fp_mul2(y, zz, r, y, t);
        tx[i] = x; ty[i] = y;
    }
    fp beta;
#pragma unroll
    for (int k = 0; k < 12; k++) beta.v[k] = FP_BETA[k];
    fp_mul(bx[7], tx[7], beta);
    fp s = rat[7];
#pragma unroll 1
    for (int i = 6; i >= 0; i--) {
        if (i < 6) fp_mul(s, s, rat[i + 1]);
        fp s2;
        fp_sqr(s2, s);
        fp_mul(t, tx[i], s2);
        tx[i] = t;
        fp_mul(bx[i], t, beta);
        fp_mul(s2, s2, s);
        fp_mul(ty[i], ty[i], s2);
    }
    if (Odd) fp_mul(zg, zg, s);
    else zg = s;
}

// k1 P + k2 phi(P) by double and add with the complete additions: points of small
// order only, whose table has no common z.
static __device__ __noinline__ void xyzz_mult_plain(xyzz& out, const xyzz& P, const uint32_t* k1, const uint32_t* k2)
{
    xyzz Q = P, acc;
    fp beta;
#pragma unroll
    for (int k = 0; k < 12; k++) beta.v[k] = FP_BETA[k];
    fp_mul(Q.x, Q.x, beta);
    xyzz_set_inf(acc);
#pragma unroll 1
    for (int i = 127; i >= 0; i--) {
        xyzz_dbl(acc);
        if ((k1[i >> 5] >> (i & 31)) & 1u) xyzz_add(acc, P);
        if ((k2[i >> 5] >> (i & 31)) & 1u) xyzz_add(acc, Q);
    }
    out = acc;
}

// acc on the table's curve -> out with P's own z and the table's common z
__device__ __forceinline__ void glv_finish(xyzz& out, const jac& acc, const fp& zg, const xyzz& P)
{
    if (jac_is_inf(acc)) {
        xyzz_set_inf(out);
        return;
    }
    fp z, zz;
    fp_mul(z, acc.z, zg);
    fp_sqr(zz, z);
    fp_mul(z, zz, z);
    const fp pzz = P.zz, pzzz = P.zzz;
    out.x = acc.x;
    out.y = acc.y;
    fp_mul(out.zz, zz, pzz);
    fp_mul(out.zzz, z, pzzz);
}

// Lanes with scalars of their own: fixed windows.
static __device__ __noinline__ void xyzz_mult_glv(xyzz& out, const xyzz& P, const uint32_t* k1, const uint32_t* k2)
{
    if (xyzz_is_inf(P)) {
        xyzz_set_inf(out);
        return;
    }
    fp tx[8], ty[8], bx[8], zg;
    glv_table<false>(tx, ty, bx, zg, P.x, P.y);
    if (fp_is_zero(zg)) {
        xyzz_mult_plain(out, P, k1, k2);
        return;
    }
    int8_t d1[33], d2[33];
    booth4_128(d1, k1);
    booth4_128(d2, k2);
    jac acc;
    jac_set_inf(acc);
#pragma unroll 1
    for (int i = 32; i >= 0; i--) {
#pragma unroll 1
        for (int k = 0; k < 4; k++) jac_dbl(acc);
#pragma unroll 1
        for (int hh = 0; hh < 2; hh++) {
            const int a = hh ? d2[i] : d1[i];
            if (a) {
                const int e = (a > 0 ? a : -a) - 1;
                fp y = ty[e];
                if (a < 0) fp_neg(y, y);
                jac_madd(acc, hh ? bx[e] : tx[e], y);
            }
        }
    }
    glv_finish(out, acc, zg, P);
}

// Lanes that all multiply by one scalar: width-5 NAF halves over the odd
// multiples (~43 additions against ~61); the digit positions depend on the scalar.
static __device__ __noinline__ void xyzz_mult_glv_shared(xyzz& out, const xyzz& P, const uint32_t* k1,
                                                         const uint32_t* k2)
{
    if (xyzz_is_inf(P)) {
        xyzz_set_inf(out);
        return;
    }
    fp tx[8], ty[8], bx[8], zg;
    glv_table<true>(tx, ty, bx, zg, P.x, P.y);
    if (fp_is_zero(zg)) {
        xyzz_mult_plain(out, P, k1, k2);
        return;
    }
    int8_t d1[130], d2[130];
    const int n1 = wnaf5_128(d1, k1), n2 = wnaf5_128(d2, k2);
    jac acc;
    jac_set_inf(acc);
#pragma unroll 1
    for (int i = max(n1, n2) - 1; i >= 0; i--) {
        jac_dbl(acc);
#pragma unroll 1
        for (int hh = 0; hh < 2; hh++) {
            const int a = hh ? (i < n2 ? d2[i] : 0) : (i < n1 ? d1[i] : 0);
            if (a) {
                const int e = (a > 0 ? a : -a) >> 1;
                fp y = ty[e];
                if (a < 0) fp_neg(y, y);
                jac_madd(acc, hh ? bx[e] : tx[e], y);
            }
        }
    }
    glv_finish(out, acc, zg, P);
}

// ---------------------------------------------------------------------------
// The quad form: four lanes on one multiplication (see the quad point
// operations), for launches whose time is the chain of one of them.  XYZZ
// throughout: a doubling is 3 dependent products and a mixed addition 4.  The
// table lives in shared memory, one copy per quad.
struct quad_table {
    fp x[8], y[8], bx[8], ny[8];  // ny: -y; while the table is built, the z ratios and their suffix products
};

// Every lane of the quad passes the same point and scalar; returns the product,
// distributed.  Half: k1 P only.
template <bool Half>
static __device__ __noinline__ fp qd_mult_glv(const xyzz& P, const uint32_t* k1, const uint32_t* k2, quad_table* tab,
                                              const quad_lane q)
{
    fp d;
    fp_zero(d);
    if (xyzz_is_inf(P)) return d;
    const bool odd = (q.k & 1) != 0;
    // multiples 1 .. 8 of the affine (X, Y), z ratios to tab->ny
    const fp a = fp_sel(P.x, P.y, odd);
    fp c, h;
    qd_set_affine(c, a, q);
    fp_dbl(h, P.y);               // z of 2 (X, Y)
    qd_dbl(c, q);
    if (q.k == 0) {
        tab->x[0] = a;
        tab->x[1] = c;
        tab->ny[1] = h;
    } else if (q.k == 1) {
        tab->y[0] = a;
        tab->y[1] = c;
    }
#pragma unroll 1
    for (int i = 2; i < 8; i++) {
        const fp PR = qd_madd_diff(c, a, q);
        c = qd_add_core<true>(PR, c, c, c, q);
        if (q.k == 0) {
            tab->x[i] = c;
            tab->ny[i] = PR;
        } else if (q.k == 1) {
            tab->y[i] = c;
        }
    }
    __syncwarp(q.mask);
    if (qd_is_inf(c, q)) {        // zz of 8 P: zero if any ratio is
        const uint32_t zero[4] = {0, 0, 0, 0};
        xyzz out;
        xyzz_mult_plain(out, P, k1, Half ? zero : k2);
        const fp lo = fp_sel(out.x, out.y, odd), hi = fp_sel(out.zz, out.zzz, odd);
        return fp_sel(lo, hi, q.k >= 2);
    }
    // suffix products: ny[i] = product of the ratios i + 1 .. 7 (i < 7)
    fp s = tab->ny[7];
#pragma unroll 1
    for (int i = 5; i >= 0; i--) {
        fp t;
        fp_mul(t, s, tab->ny[i + 1]);
        __syncwarp(q.mask);
        if (q.k == 0) tab->ny[i + 1] = s;
        s = t;
    }
    if (q.k == 0) tab->ny[0] = s;
    __syncwarp(q.mask);
    fp beta;
#pragma unroll
    for (int k = 0; k < 12; k++) beta.v[k] = FP_BETA[k];
    // lane k rescales entries k and k + 4 (entry 7 has the common z already)
#pragma unroll 1
    for (uint32_t i = q.k; i < 8; i += 4) {
        fp one;
        fp_set_one(one);
        const fp si = i < 7 ? tab->ny[i] : one;
        fp s2, x;
        fp_sqr(s2, si);
        fp_mul(x, tab->x[i], s2);
        tab->x[i] = x;
        fp_mul(x, x, beta);
        tab->bx[i] = x;
        fp_mul(s2, s2, si);
        fp_mul(x, tab->y[i], s2);
        tab->y[i] = x;
        fp_neg(x, x);
        tab->ny[i] = x;
    }
    __syncwarp(q.mask);
    int8_t d1[33], d2[33];
    booth4_128(d1, k1);
    if (!Half) booth4_128(d2, k2);
    bool started = false;
#pragma unroll 1
    for (int i = 32; i >= 0; i--) {
        if (started) {
#pragma unroll 1
            for (int k = 0; k < 4; k++) qd_dbl(d, q);
        }
#pragma unroll 1
        for (int hh = 0; hh < (Half ? 1 : 2); hh++) {
            const int g = hh ? d2[i] : d1[i];
            if (g) {
                const int e = (g > 0 ? g : -g) - 1;
                qd_madd(d, odd ? (g > 0 ? tab->y[e] : tab->ny[e]) : (hh ? tab->bx[e] : tab->x[e]), q);
                started = true;
            }
        }
    }
    // common z of the table (c's zz, zzz), then P's own
    const fp r = fp_mul_call(fp_mul_call(d, c), fp_sel(P.zz, P.zzz, odd));
    return fp_sel(d, r, q.k >= 2);
}

// ---------------------------------------------------------------------------
// The pair form: two lanes on one multiplication, between the quad (whose four
// lanes idle in a third of their products) and the single lane (whose chain of
// 7 and 11 products a doubling and an addition is twice as long).  Jacobian: lane
// 0 holds x, lane 1 holds y and z; a doubling is 4 dependent products (two of
// them squarings), a mixed addition 6.  5.4 k of them 0.98 ms (quads 1.03), 12 k
// 1.33 (lanes 1.65, quads two waves), from 20 k no faster than lanes: 2^12 FFT
// 6.2 -> 5.4 ms, 2^13 9.9 -> 8.1.
struct pair_table {
    fp x[8], y[8], bx[8];         // bx: while the table is built, the z ratios and their suffix products
};

struct pair_lane {
    bool odd;
    uint32_t mask;
};

struct pair_acc {
    fp c, z;                      // lane 0: x, -; lane 1: y, z
};

__device__ __forceinline__ fp pd_swap(const fp& v, const pair_lane& l)
{
    fp r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = __shfl_xor_sync(l.mask, v.v[i], 1, 2);
    return r;
}

__device__ __forceinline__ fp pd_bcast(const fp& v, int src, const pair_lane& l)
{
    fp r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = __shfl_sync(l.mask, v.v[i], src, 2);
    return r;
}

// dbl-2009-l: X^2, Y^2 | (X + B)^2, B^2 | E^2, Y Z | E (D - X3), -
__device__ __forceinline__ void pd_dbl(pair_acc& p, const pair_lane& l)
{
    fp s, w, t, E, X3;
    fp_sqr(s, p.c);                                       // A, B
    fp_add(t, p.c, pd_swap(s, l));                        // lane 0: X + B
    fp_sqr(w, fp_sel(t, s, l.odd));                       // (X + B)^2, C
    fp_dbl(E, s);
    fp_add(E, E, s);                                      // lane 0: E = 3A
    fp r, D;
    fp_mul(r, fp_sel(E, p.c, l.odd), fp_sel(E, p.z, l.odd));
    fp_sub(t, w, s);
    fp_sub(t, t, pd_swap(w, l));
    fp_dbl(D, t);
    fp_sub(t, r, D);
    fp_sub(X3, t, D);
    fp_sub(t, D, X3);
    fp_mul(t, E, t);                                      // lane 0: E (D - X3)
    fp_dbl(w, w);
    fp_dbl(w, w);
    fp_dbl(w, w);                                         // lane 1: 8C
    fp_sub(t, pd_swap(t, l), w);                          // lane 1: Y3
    p.c = fp_sel(X3, t, l.odd);
    fp_dbl(p.z, r);                                       // lane 1: 2YZ
}

// h = the difference H = U2 - X1 (both lanes), r = S2 - Y1 (lane 1), hh = H^2
// (lane 0) of (ax, ay) and p: Z^2 | U2, Z^3 | H^2, S2
__device__ __forceinline__ void pd_diff(fp& h, fp& r, fp& hh, const pair_acc& p, const fp& a, const pair_lane& l)
{
    fp t, u;
    fp_sqr(t, p.z);
    t = pd_bcast(t, 1, l);
    fp_mul(u, fp_sel(a, p.z, l.odd), t);
    fp_sub(t, u, p.c);
    h = pd_bcast(t, 0, l);
    fp_mul(hh, fp_sel(h, a, l.odd), fp_sel(h, u, l.odd));
    fp_sub(r, hh, p.c);
}

// The rest of the addition: H HH, Z H | X HH, R^2 | R (V - X3), Y HHH
__device__ __forceinline__ void pd_core(pair_acc& p, const fp& h, const fp& r, const fp& hh, const pair_lane& l)
{
    fp z, v, t, X3, u;
    fp_mul(z, fp_sel(hh, p.z, l.odd), h);                 // HHH, Z3
    fp_mul(v, fp_sel(p.c, r, l.odd), fp_sel(hh, r, l.odd));   // V, RR
    const fp R = pd_swap(r, l), o = pd_swap(fp_sel(z, v, l.odd), l);   // lane 0: R, RR; lane 1: -, HHH
    fp_sub(t, o, z);
    fp_sub(t, t, v);
    fp_sub(X3, t, v);                                     // lane 0: RR - HHH - 2V
    fp_sub(u, v, X3);
    fp_mul(t, fp_sel(R, p.c, l.odd), fp_sel(u, o, l.odd));
    fp_sub(t, pd_swap(t, l), t);                          // lane 1: R (V - X3) - Y HHH
    p.c = fp_sel(X3, t, l.odd);
    p.z = z;
}

__device__ __forceinline__ void pd_set(pair_acc& p, const fp& a)
{
    p.c = a;
    fp_set_one(p.z);
}

// Both lanes of the pair pass the same point and scalar; the product's x and zz
// in lane 0 (lo, hi), y and zzz in lane 1.
static __device__ __noinline__ void pd_mult_glv(fp& lo, fp& hi, const xyzz& P, const uint32_t* k1, const uint32_t* k2,
                                                pair_table* tab, const pair_lane l)
{
    fp_zero(lo);
    fp_zero(hi);
    if (xyzz_is_inf(P)) return;
    const fp a = fp_sel(P.x, P.y, l.odd);
    pair_acc p;
    pd_set(p, a);
    (l.odd ? tab->y : tab->x)[0] = a;
#pragma unroll 1
    for (int i = 1; i < 8; i++) {
        if (i == 1) {
            pd_dbl(p, l);
            if (l.odd) tab->bx[1] = p.z;                  // 2Y
        } else {
            fp h, r, hh;
            pd_diff(h, r, hh, p, a, l);
            pd_core(p, h, r, hh, l);
            if (l.odd) tab->bx[i] = h;
        }
        (l.odd ? tab->y : tab->x)[i] = p.c;
    }
    const fp zg = pd_bcast(p.z, 1, l);                    // z of 8 P: zero if any ratio is
    if (fp_is_zero(zg)) {
        xyzz out;
        xyzz_mult_plain(out, P, k1, k2);
        lo = fp_sel(out.x, out.y, l.odd);
        hi = fp_sel(out.zz, out.zzz, l.odd);
        return;
    }
    __syncwarp(l.mask);
    // suffix products: bx[i] = product of the ratios i + 1 .. 7 (i < 7)
    fp s = tab->bx[7];
#pragma unroll 1
    for (int i = 5; i >= 0; i--) {
        fp t;
        fp_mul(t, s, tab->bx[i + 1]);
        __syncwarp(l.mask);
        if (!l.odd) tab->bx[i + 1] = s;
        s = t;
    }
    if (!l.odd) tab->bx[0] = s;
    __syncwarp(l.mask);
    fp beta;
#pragma unroll
    for (int k = 0; k < 12; k++) beta.v[k] = FP_BETA[k];
    // a lane rescales every second entry (entry 7 has the common z already)
#pragma unroll 1
    for (int i = l.odd ? 1 : 0; i < 8; i += 2) {
        fp one;
        fp_set_one(one);
        const fp si = i < 7 ? tab->bx[i] : one;
        fp s2, x;
        fp_sqr(s2, si);
        fp_mul(x, tab->x[i], s2);
        tab->x[i] = x;
        fp_mul(x, x, beta);
        tab->bx[i] = x;
        fp_mul(s2, s2, si);
        fp_mul(x, tab->y[i], s2);
        tab->y[i] = x;
    }
    __syncwarp(l.mask);
    int8_t d1[33], d2[33];
    booth4_128(d1, k1);
    booth4_128(d2, k2);
    bool inf = true;
#pragma unroll 1
    for (int i = 32; i >= 0; i--) {
        if (!inf) {
#pragma unroll 1
            for (int k = 0; k < 4; k++) pd_dbl(p, l);
        }
#pragma unroll 1
        for (int w = 0; w < 2; w++) {
            const int g = w ? d2[i] : d1[i];
            if (!g) continue;
            const int e = (g > 0 ? g : -g) - 1;
            fp b = l.odd ? tab->y[e] : w ? tab->bx[e] : tab->x[e], n;
            fp_neg(n, b);
            b = fp_sel(b, n, l.odd && g < 0);
            if (inf) {
                pd_set(p, b);
                inf = false;
                continue;
            }
            fp h, r, hh;
            pd_diff(h, r, hh, p, b, l);
            if (fp_is_zero(h)) {
                const bool same = __shfl_sync(l.mask, (int)fp_is_zero(r), 1, 2) != 0;
                if (same) pd_dbl(p, l);
                else inf = true;
                continue;
            }
            pd_core(p, h, r, hh, l);
        }
    }
    if (inf) return;
    // Z zg, then its square (lane 0) and cube (lane 1), times P's own
    fp z, zz, t;
    fp_mul(z, p.z, zg);
    z = pd_bcast(z, 1, l);
    fp_sqr(zz, z);
    fp_mul(t, zz, z);
    fp_mul(hi, fp_sel(zz, t, l.odd), fp_sel(P.zz, P.zzz, l.odd));
    lo = p.c;
}

__device__ __constant__ static const uint32_t FP_BETA2[12] = {  // beta^2 (Montgomery)
    0x798a64e8u, 0x30f1361bu, 0x7ece5a2au, 0xf3b8ddabu, 0xc61577f7u, 0x16a8ca3au,
    0x74fd029bu, 0xc26a2ff8u, 0x60701c6eu, 0x3636b766u, 0x241b6160u, 0x051ba4abu};

// |z| = 0xd201000000010000 as runs of doublings, each but the last followed by
// one addition (the reference's addition chain)
__device__ __constant__ static const uint8_t Z_RUNS[6] = {1, 2, 3, 9, 32, 16};

// out = |z| (ax, ay)
__device__ __forceinline__ void times_abs_z(jac& out, const fp& ax, const fp& ay)
{
    out.x = ax;
    out.y = ay;
    fp_set_one(out.z);
#pragma unroll 1
    for (int r = 0; r < 6; r++) {
#pragma unroll 1
        for (int i = Z_RUNS[r]; i > 0; i--) jac_dbl(out);
        if (r < 5) jac_madd(out, ax, ay);
    }
}

// The same by a quad, distributed; lane k passes coordinate k mod 2.
__device__ __forceinline__ void qd_times_abs_z(fp& out, const fp& a, const quad_lane& q)
{
    qd_set_affine(out, a, q);
#pragma unroll 1
    for (int r = 0; r < 6; r++) {
#pragma unroll 1
        for (int i = Z_RUNS[r]; i > 0; i--) qd_dbl(out, q);
        if (r < 5) qd_madd(out, a, q);
    }
}

}  // namespace catmsm
