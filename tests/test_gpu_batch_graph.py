"""Batches of one basis whose workspaces move between two uses of the captured
graph (more pairs, more MSMs, another chunk length), each against the plain MSM
over the same prefix."""
import pytest

pytestmark = pytest.mark.gpu

N = 600


@pytest.mark.parametrize("between", ["more_pairs", "more_msms", "chunk"])
def test_graph_after_buffers_moved(gpu, oracle, synth, between):
    pts = gpu.points_from_scalars(synth.point_scalars(71, N), N)
    b = gpu.Basis(pts, N, 9)
    b.set_config(9, 64)

    def check(counts, seed, graph):
        sc = synth.scalars(seed, sum(counts), 0)
        out, off = b.msm_batch(counts, sc, graph), 0
        for j, k in enumerate(counts):
            ref = gpu.p1s_mult_pippenger(pts[:96 * k], sc[32 * off:32 * (off + k)], k, 256)
            assert oracle.compress(out[144 * j:144 * j + 144]) == oracle.compress(ref)
            off += k

    check([3, 40, 1, 17], 1, True)
    if between == "more_pairs":
        check([N] * 4, 2, False)
    elif between == "more_msms":
        check([9] * 70, 2, False)
    else:
        b.set_config(9, 2)
        check([N] * 4, 2, False)
        b.set_config(9, 64)
    check([3, 40, 1, 17], 3, True)
    check([5, 1, 30, 2], 4, True)
    b.close()
