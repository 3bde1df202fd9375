"""CPU checks of what the library's host code does when a CUDA call fails or memory
runs out, over a fake CUDA runtime (see fake_cuda)."""
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def host(gpu_binding):
    gpu_binding.load()
    return lambda body: fake_cuda.run(gpu_binding.LIB_PATH, body)


def test_a_failed_allocation_fails_one_call(host):
    """The error of an allocation that failed is reported by that call alone."""
    first, second = host("""
def call(n):
    return L.catmsm_p1s_deserialize(buf(96 * n), buf(96 * n), S(n), buf(4 * n), 0)
limit(1 << 20)
first = call(1 << 16)
limit(0)
done([first, call(1 << 16)])
""")
    assert first != 0 and second == 0
