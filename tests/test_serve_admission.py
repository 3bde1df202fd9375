"""CPU check of the serving engine's admission by its memory budget, over a fake
CUDA runtime (see fake_cuda)."""
import pytest

import fake_cuda


@pytest.mark.parametrize("budget_mb,admitted,rounds", [(1150, 4, False), (4096, 4, True), (600, 2, False)])
def test_batch_is_admitted_by_what_it_cannot_do_without(gpu_binding, budget_mb, admitted, rounds):
    """MSMs of 60000 points over 8-bit tables take 271 MB each.  The affine rounds of a
    batch of four take 1.84 GB more: within the budget they run, without room for
    them the batch is as large and runs without."""
    gpu_binding.load()
    most, kinds = fake_cuda.run(gpu_binding.LIB_PATH, """
import time
n = 60000
b = Basis(n, 8)
s = P(L.catmsm_server_create(b.h, S(1), S(%d << 20)))
sc = buf(32 * n)
F.fake_hold(1)
first = L.catmsm_server_submit_msm(s, sc, S(16))
while ["sync"] not in [l[:1] for l in log()[-1:]]:
    time.sleep(0.01)
clear()
tickets = [L.catmsm_server_submit_msm(s, sc, S(n)) for _ in range(4)]
F.fake_hold(0)
for t in [first] + tickets:
    assert L.catmsm_server_wait(s, C.c_int64(t), buf(144), None) == 0
st = [C.c_long() for _ in range(4)]
L.catmsm_server_stats(s, *[C.byref(x) for x in st])
done([st[2].value, sorted(set(k.split("<")[0] for k in kernels()))])
L.catmsm_server_destroy(s)
""" % budget_mb)
    assert most == admitted
    assert ("k_aff_first" in kinds) == rounds
