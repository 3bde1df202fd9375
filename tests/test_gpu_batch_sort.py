"""The batched commitments' bucket sort (batch.cu): MSM lengths at the edges of
a part (1024 pairs), windows on both sides of the part sort's limits, one
bucket holding a whole MSM, zero scalars, and scalars in page-locked and in
pageable memory, each against the plain MSM over the same prefix."""
import pytest

pytestmark = pytest.mark.gpu

N = 2500
COUNTS = [0, 1, 2, 1023, 1024, 1025, 2047, 2049, N, 700, 700]


@pytest.fixture(scope="module")
def batch(gpu, oracle, synth):
    pts = gpu.points_from_scalars(synth.point_scalars(61, N), N)
    sc = [synth.scalars(100 + j, k, 2 if j % 2 else 0) if k else b"" for j, k in enumerate(COUNTS)]
    sc[-2] = synth.scalars(7, 1, 0) * 700                       # every window of the MSM in one bucket
    sc[-1] = bytes(32 * 700)
    want = [oracle.compress(gpu.p1s_mult_pippenger(pts[:96 * k], s, k, 256)) if k else oracle.compress(bytes(144))
            for k, s in zip(COUNTS, sc)]
    return pts, b"".join(sc), want


@pytest.mark.parametrize("window", [2, 5, 11, 13, 14])
@pytest.mark.parametrize("chunk", [16, 96])
def test_batch_sort(gpu, oracle, batch, window, chunk):
    import torch
    pts, sc, want = batch
    b = gpu.Basis(pts, N, window)
    b.set_config(window, chunk)
    pinned = torch.frombuffer(bytearray(sc), dtype=torch.uint8).pin_memory()
    for scalars, graph in ((sc, True), (pinned.data_ptr(), True), (pinned.data_ptr(), False)):
        out = b.msm_batch(COUNTS, scalars, graph)
        got = [oracle.compress(out[144 * i:144 * i + 144]) for i in range(len(COUNTS))]
        assert got == want
    # another batch of the same size: fewer pairs (the captured graph's capacity), then more
    for counts in ([1] * len(COUNTS), COUNTS[::-1]):
        full = {k: sc[32 * sum(COUNTS[:i]):32 * sum(COUNTS[:i + 1])] for i, k in enumerate(COUNTS)}
        cat = b"".join(full[k] for k in counts)
        out = b.msm_batch(counts, cat)
        for i, k in enumerate(counts):
            ref = gpu.p1s_mult_pippenger(pts[:96 * k], full[k], k, 256) if k else bytes(144)
            assert oracle.compress(out[144 * i:144 * i + 144]) == oracle.compress(ref)
    b.close()
