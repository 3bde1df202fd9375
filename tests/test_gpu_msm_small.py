"""The MSM of few points (msm_small.cu): every scalar width the windows treat
differently, sizes at the ends of its ranges and one past them, one hot bucket,
edge scalars, repeated, opposite and identity points, against the oracle."""
import pytest

pytestmark = pytest.mark.gpu

R = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001
LAMBDA = 0xac45a4010001a40200000000ffffffff
P = 0x1a0111ea397fe69a4b1ba7b6434bacd764774b84f38512bf6730d2a0f6b0f6241eabfffeb153ffffb9feffffffffaaab


def _scalars(vals, nbits):
    return b"".join((v % (1 << nbits)).to_bytes((nbits + 7) // 8, "little") for v in vals)


@pytest.mark.parametrize("nbits", [1, 3, 4, 5, 7, 8, 31, 63, 64, 127, 128, 129, 255, 256])
@pytest.mark.parametrize("n", [1, 2, 33, 1025])
def test_small_widths(gpu, oracle, synth, n, nbits):
    import random
    rnd = random.Random(n * 1000 + nbits)
    pts = oracle.gen_points(17, n)
    vals = [rnd.randrange(1 << nbits) for _ in range(n)]
    for i, v in enumerate([(1 << nbits) - 1, 0, 1, 1 << (nbits - 1), 0x88888888888888888888888888888888,
                           0x80808080808080808080808080808080, 0x7f7f7f7f7f7f7f7f7f7f7f7f7f7f7f7f, R - 1, R, LAMBDA,
                           (LAMBDA + 1) // 2, (LAMBDA + 1) // 2 * (LAMBDA + 1)]):
        if 2 * i < n:
            vals[2 * i] = v
    sc = _scalars(vals, nbits)
    assert oracle.compress(gpu.p1s_mult_pippenger(pts, sc, n, nbits)) == oracle.msm(pts, sc, n, nbits)


@pytest.mark.parametrize("n,nbits", [(255, 255), (256, 255), (257, 255), (512, 64), (513, 64), (3072, 64), (3073, 64),
                                     (12287, 255), (12288, 255), (12289, 255)])
def test_small_sizes(gpu, oracle, synth, n, nbits):
    """4- and 8-bit windows up to / from 512 pipeline points; the general pipeline from 3073 unsplit or 24578 split ones."""
    pts = gpu.points_from_scalars(synth.point_scalars(23, n), n)
    sc = synth.scalars(24, n, 2 if nbits == 255 else 1)
    if nbits == 64:
        sc = b"".join(sc[32 * i:32 * i + 8] for i in range(n))
    assert oracle.compress(gpu.p1s_mult_pippenger(pts, sc, n, nbits)) == oracle.msm(pts, sc, n, nbits)


@pytest.mark.parametrize("n", [100, 4096, 12288])
def test_small_hot_buckets_and_special_points(gpu, oracle, synth, n):
    pts = bytearray(gpu.points_from_scalars(synth.point_scalars(29, n), n))
    for scalar in (1, 8, 128, R - 1):                            # every entry of a window in one bucket
        sc = scalar.to_bytes(32, "little") * n
        assert oracle.compress(gpu.p1s_mult_pippenger(bytes(pts), sc, n, 255)) == oracle.msm(bytes(pts), sc, n, 255)
    one = bytes(pts[:96])
    for i in range(0, n, 3):                                     # equal, opposite and identity points
        src = bytearray(one)
        if i % 2:
            y = int.from_bytes(src[48:], "little")
            src[48:] = (P - y).to_bytes(48, "little")
        pts[96 * i:96 * i + 96] = src if i % 5 else bytes(96)
    for sc in (synth.scalars(31, n, 0), (5).to_bytes(32, "little") * n):
        assert oracle.compress(gpu.p1s_mult_pippenger(bytes(pts), sc, n, 255)) == oracle.msm(bytes(pts), sc, n, 255)
    sc = synth.scalars(33, n, 0)
    assert gpu.msm_affine_rounds(0) == -1                        # the general pipeline gives the same point
    try:
        general = gpu.p1s_mult_pippenger(bytes(pts), sc, n, 255)
    finally:
        gpu.msm_affine_rounds(-1)
    assert general == gpu.p1s_mult_pippenger(bytes(pts), sc, n, 255)
