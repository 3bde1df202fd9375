"""Large MSMs whose size asks for affine rounds and whose scalars leave fewer entries
than they need (msm_affine_min_entries), on both sides of it, against the mixed
additions alone; and batches of sparse scalars against the plain MSM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kept", [(1 << 18, 0.0001), (1 << 18, 0.55), (1 << 18, 0.57), (1 << 19, 0.1), (1 << 19, 0.8),
                                    (1 << 19, 0.82), (1 << 20, 0.18), (1 << 20, 0.2)])
def test_sparse_large_msm(gpu, oracle, synth, n, kept):
    import torch
    k = torch.frombuffer(bytearray(synth.point_scalars(91, n)), dtype=torch.uint8).cuda()
    pts = torch.empty(96 * n, dtype=torch.uint8, device="cuda")
    assert gpu.load().catmsm_p1_affines_from_scalars_device(pts.data_ptr(), k.data_ptr(), n) == 0
    sc = np.frombuffer(synth.scalars(92, n, 0), dtype=np.uint8).reshape(n, 32).copy()
    sc[synth.splitmix64(93, n) > np.uint64(min(int(kept * 2 ** 64), 2 ** 64 - 1))] = 0
    d = torch.from_numpy(sc).cuda()
    torch.cuda.synchronize()
    got = gpu.msm_device(pts.data_ptr(), d.data_ptr(), 32, n, 255)
    prev = gpu.msm_affine_rounds(0)
    try:
        want = gpu.msm_device(pts.data_ptr(), d.data_ptr(), 32, n, 255)
    finally:
        gpu.msm_affine_rounds(prev)
    assert oracle.compress(got) == oracle.compress(want)


@pytest.mark.parametrize("graph", [False, True])
def test_sparse_batch(gpu, oracle, synth, graph):
    n, nmsm = 4096, 64
    pts = gpu.points_from_scalars(synth.point_scalars(94, n), n)
    b = gpu.Basis(pts, n, 11)
    for kept in (0.05, 1.0, 0.6):
        sc = np.frombuffer(synth.scalars(95, n * nmsm, 0), dtype=np.uint8).reshape(n * nmsm, 32).copy()
        sc[synth.splitmix64(96, n * nmsm) > np.uint64(min(int(kept * 2 ** 64), 2 ** 64 - 1))] = 0
        out = b.msm_batch([n] * nmsm, sc.tobytes(), graph)
        for j in range(0, nmsm, 9):
            ref = gpu.p1s_mult_pippenger(pts, sc[n * j:n * (j + 1)].tobytes(), n, 256)
            assert oracle.compress(out[144 * j:144 * j + 144]) == oracle.compress(ref)
    b.close()
