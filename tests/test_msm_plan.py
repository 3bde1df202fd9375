"""CPU checks of the MSM's window choice (host arithmetic only)."""
import pytest


@pytest.mark.parametrize("n", [1, 2, 100, 512, 513, 3000, 3072, 3073, 5000, 1 << 16, (1 << 18) - 1, 1 << 18, 300007, 1 << 20])
def test_window_query_is_the_plan_for_128_bits(gpu_binding, n):
    """catmsm_msm_window answers with the width that the MSM takes: the small
    kernel's up to 3072 points, the cost model's from 2^18 on."""
    assert gpu_binding.msm_window(n) == gpu_binding.msm_plan_detail(n, 128)[0]
    if n < 1 << 18:
        assert {gpu_binding.msm_plan_detail(n, b)[0] for b in (1, 17, 64, 100, 128)} == {gpu_binding.msm_window(n)}
