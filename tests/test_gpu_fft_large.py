"""A transform too large for a pass's products to be kept (2^22 points: a level of
butterflies a pass throughout, the inverse's scale in the last level's roots), as a round
trip, with three of its forward outputs against sums in the exponent."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001


def test_round_trip_without_products(gpu, oracle, synth):
    import torch
    lg, m = 22, 4096
    n, L = 1 << lg, gpu.load()
    small = synth.scalars(101, m, 0)                         # the points repeat: x_i = k_(i mod m) G
    k = torch.frombuffer(bytearray(small), dtype=torch.uint8).cuda()
    aff = torch.empty(96 * m, dtype=torch.uint8, device="cuda")
    assert L.catmsm_p1_affines_from_scalars_device(aff.data_ptr(), k.data_ptr(), m) == 0
    one = torch.frombuffer(bytearray(((1 << 384) % int("1a0111ea397fe69a4b1ba7b6434bacd764774b84f38512bf6730d2a0f6b0f624"
                                                       "1eabfffeb153ffffb9feffffffffaaab", 16)).to_bytes(48, "little")),
                           dtype=torch.uint8).cuda()
    jac = torch.cat([aff.view(m, 96), one.expand(m, 48)], 1).repeat(n // m, 1).contiguous()
    start = jac[:m].cpu().numpy().tobytes()
    ok, dom = gpu.fr_fft_domain_init(n)
    assert ok
    d = torch.from_numpy(np.frombuffer(dom, dtype=np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    assert L.catmsm_p1_fft_device(C.c_void_p(jac.data_ptr()), n, C.c_void_p(d.data_ptr()), 0) == 0
    # a repeated input has outputs at multiples of n / m only: (n / m) sum_i k_i w^(i j n / m)
    w = int.from_bytes(dom[32:64], "little") * pow(1 << 256, -1, R) % R
    ks = [int.from_bytes(small[32 * i:32 * i + 32], "little") for i in range(m)]
    for j in (0, 1, 777):
        v = pow(w, j * (n // m), R)
        e, p = 0, 1
        for x in ks:
            e, p = (e + x * p) % R, p * v % R
        e = e * (n // m) % R
        got = jac[j * (n // m)].cpu().numpy().tobytes()
        want = gpu.points_from_scalars(e.to_bytes(32, "little"), 1)
        assert oracle.compress(got) == oracle.compress(want + one.cpu().numpy().tobytes())
    assert not jac[1, 96:].any() and not jac[n - 1, 96:].any()
    assert L.catmsm_p1_fft_device(C.c_void_p(jac.data_ptr()), n, C.c_void_p(d.data_ptr()), 1) == 0
    for i in list(range(0, m, 61)) + [m, n // 2 + 5, n - 1]:
        assert oracle.compress(jac[i].cpu().numpy().tobytes()) == oracle.compress(start[144 * (i % m):144 * (i % m) + 144])
