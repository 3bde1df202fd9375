"""CPU checks of the MSM's window choice (host arithmetic only)."""
import pytest


@pytest.mark.parametrize("n", [1, 2, 100, 512, 513, 3000, 3072, 3073, 5000, 1 << 16, (1 << 18) - 1, 1 << 18, 300007, 1 << 20])
def test_window_query_is_the_plan_for_128_bits(gpu_binding, n):
    """catmsm_msm_window answers with the width that the MSM takes: the small
    kernel's up to 3072 points, the cost model's from 2^18 on."""
    assert gpu_binding.msm_window(n) == gpu_binding.msm_plan_detail(n, 128)[0]
    if n < 1 << 18:
        assert {gpu_binding.msm_plan_detail(n, b)[0] for b in (1, 17, 64, 100, 128)} == {gpu_binding.msm_window(n)}


@pytest.mark.parametrize("nbits", [63, 64, 127])
@pytest.mark.parametrize("rounds", [-1, 0, 2])
def test_plan_is_what_runs(gpu_binding, nbits, rounds):
    """catmsm_msm_plan against the windows that are reduced, with the affine
    rounds chosen by size (small kernel) and set by the caller (general pipeline)."""
    import fake_cuda
    gpu_binding.load()
    windows, reduced = fake_cuda.run(gpu_binding.LIB_PATH, """
n, nbits, rounds = 1000, %d, %d
L.catmsm_msm_affine_rounds(rounds)
out = sizes([0, 0, 0])
assert L.catmsm_msm_plan(S(n), S(nbits), C.byref(out, 0), C.byref(out, 8), C.byref(out, 16)) == 0
clear()
assert L.catmsm_p1s_mult_pippenger_device(buf(144), aligned(96 * n), buf(32 * n), S(32), S(n), S(nbits), S(0)) == 0
done([out[1], [int(l[3]) for l in log() if l[0] == "launch" and "k_reduce_tail" in l[2]]])
""" % (nbits, rounds))
    assert reduced == [windows]
