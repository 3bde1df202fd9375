"""Small MSMs whose scalars fill the buckets unevenly, at both sides of what one
block of the small kernel takes (2048 entries, 7/4 of its share, 2560 of one
bucket): the result equals the oracle's whichever path runs."""
import pytest

pytestmark = pytest.mark.gpu

N = 12288


@pytest.fixture(scope="module")
def points(gpu, synth):
    return gpu.points_from_scalars(synth.point_scalars(81, N), N)


def _scalars(synth, kind, n):
    rnd = synth.scalars(82, n, 0)
    one = (1).to_bytes(32, "little")
    if kind == "equal":
        return rnd[:32] * n
    if kind == "eight":
        return b"".join(rnd[32 * (i % 8):32 * (i % 8) + 32] for i in range(n))
    if kind.startswith("ones"):                                  # that many in a hundred are 1, the others 0
        k = int(kind[4:])
        return b"".join(one if i % 100 < k else bytes(32) for i in range(n))
    if kind.startswith("mixed"):                                 # the others random
        k = int(kind[5:])
        return b"".join(one if i % 100 < k else rnd[32 * i:32 * i + 32] for i in range(n))
    bits = int(kind[4:])
    return b"".join((int.from_bytes(rnd[32 * i:32 * i + 32], "little") & ((1 << bits) - 1)).to_bytes(32, "little")
                    for i in range(n))


@pytest.mark.parametrize("kind", ["equal", "eight", "ones50", "ones99", "mixed20", "mixed43", "bits64", "bits129", "bits160"])
@pytest.mark.parametrize("n", [1024, 1025, 2048, 2100, 4700, 12288])
def test_uneven_small_msm(gpu, oracle, synth, points, kind, n):
    sc = _scalars(synth, kind, n)
    assert oracle.compress(gpu.p1s_mult_pippenger(points[:96 * n], sc, n, 255)) == oracle.msm(points[:96 * n], sc, n, 255)


@pytest.mark.parametrize("nbits", [97, 100, 121])
@pytest.mark.parametrize("n", [2184, 2185, 3072])
def test_narrow_top_window(gpu, oracle, synth, points, nbits, n):
    nb = (nbits + 7) // 8
    rnd = synth.scalars(83, n, 0)
    sc = b"".join((int.from_bytes(rnd[32 * i:32 * i + 32], "little") & ((1 << nbits) - 1)).to_bytes(nb, "little")
                  for i in range(n))
    assert oracle.compress(gpu.p1s_mult_pippenger(points[:96 * n], sc, n, nbits)) == \
        oracle.msm(points[:96 * n], sc, n, nbits)
