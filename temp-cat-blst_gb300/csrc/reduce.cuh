// The reduction's kernels of one lane per node.  Each translation unit that includes
// this takes them with its own setting of CATMSM_INLINE_SQR / _MUL2 (see field.cuh),
// and instantiates the Inlined value that says which: msm.cu true, reduce_calls.cu
// false.
#pragma once
#include "curve.cuh"

namespace catmsm {

// One level of fan-in F = 2^lgF (msm.cu, 6/7), a thread per node; inQ null: buckets, `first` weighs them j + 1.
template <bool Inlined>
__global__ void __launch_bounds__(128) k_reduce_level(const xyzz* __restrict__ inA, const xyzz* __restrict__ inQ,
                                                      uint32_t m_in, uint32_t F, uint32_t lgF, uint32_t D,
                                                      int first, xyzz* __restrict__ outA, xyzz* __restrict__ outQ)
{
    const uint32_t m_out = (m_in + F - 1) / F;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= D * m_out) return;
    const uint32_t w = t / m_out, u = t % m_out;
    const uint32_t c0 = u * F;
    const uint32_t cnt = min(F, m_in - c0);
    const xyzz* a = inA + (size_t)w * m_in + c0;
    xyzz r, tt, b;
    xyzz_set_inf(r);
    xyzz_set_inf(tt);
    for (int j = (int)cnt - 1; j >= 1; j--) {
        load_xyzz(b, a + j);
        xyzz_add(r, b);
        xyzz_add(tt, r);
    }
    load_xyzz(b, a);
    xyzz_add(r, b);
    if (first) xyzz_add(tt, r);
    if (inQ) {
        const xyzz* q = inQ + (size_t)w * m_in + c0;
        for (uint32_t j = 0; j < cnt; j++) {
            load_xyzz(b, q + j);
            xyzz_add(tt, b);
        }
    }
    if (m_out > 1) {
        for (uint32_t k = 0; k < lgF; k++) xyzz_dbl(r);
        store_xyzz(outA + (size_t)w * m_out + u, r);
    }
    store_xyzz(outQ + (size_t)w * m_out + u, tt);
}

// Thread g's node and role.  The role is uniform per warp (even warps Q, odd
// warps A): lanes of one warp taking different roles would run both paths one
// after the other.  A warp covers 32 nodes, or 8 with quads.
template <bool Quad>
__device__ __forceinline__ void pair_slot(uint32_t g, uint32_t& node, bool& q_role)
{
    node = Quad ? (g >> 6) * 8 + ((g >> 2) & 7) : (g >> 6) * 32 + (g & 31);
    q_role = ((g >> 5) & 1) == 0;
}

__device__ __forceinline__ void pair_node(xyzz& out, const xyzz* a, const xyzz* q, uint32_t cnt, bool q_role)
{
    xyzz b;
    if (q_role) {
        load_xyzz(out, q);
        if (cnt == 2) {
            load_xyzz(b, a + 1);
            xyzz_add(out, b);
            load_xyzz(b, q + 1);
            xyzz_add(out, b);
        }
    } else {
        load_xyzz(out, a);
        if (cnt == 2) {
            load_xyzz(b, a + 1);
            xyzz_add(out, b);
        }
        xyzz_dbl(out);
    }
}

// One binary level over D windows of m_in (A, Q) pairs, by lanes.
template <bool Inlined>
__global__ void __launch_bounds__(128) k_reduce_pair_lanes(const xyzz* __restrict__ inA,
                                                           const xyzz* __restrict__ inQ, uint32_t m_in, uint32_t D,
                                                           xyzz* __restrict__ outA, xyzz* __restrict__ outQ)
{
    const uint32_t m_out = (m_in + 1) / 2;
    uint32_t t;
    bool q_role;
    pair_slot<false>(blockIdx.x * blockDim.x + threadIdx.x, t, q_role);
    if (t >= D * m_out || (!q_role && m_out == 1)) return;
    const uint32_t w = t / m_out, u = t % m_out;
    const size_t base = (size_t)w * m_in + 2 * u;
    xyzz r;
    pair_node(r, inA + base, inQ + base, min(2u, m_in - 2 * u), q_role);
    store_xyzz((q_role ? outQ : outA) + (size_t)w * m_out + u, r);
}

}  // namespace catmsm
