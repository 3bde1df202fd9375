"""Which kernels the G1 FFT's pass planner takes, on the CPU over a fake CUDA runtime
(see fake_cuda), and transforms of every form against the oracle with root tables in
which only some entries are powers of one root."""
import json
import math
import random

import pytest

R = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001
WAVE = 152 * 4 * 16             # quads that are resident at once


def _launches(gpu_binding, shapes, mode):
    """Per shape (log sizes of a batch), per stream: (kernel, threads) of the passes."""
    import fake_cuda
    gpu_binding.load()
    ops = fake_cuda.run(gpu_binding.LIB_PATH, """
out = []
for logs in json.loads(%r):
    ns = [1 << k for k in logs]
    dom = {n: domain(n) for n in set(ns)}
    vals = (P * len(ns))(*[buf(144 * n).value for n in ns])
    doms = (P * len(ns))(*[dom[n].value for n in ns])
    clear()
    assert L.catmsm_p1_fft_batch(vals, sizes(ns), doms, (C.c_int * len(ns))(*[%d] * len(ns)), S(len(ns))) == 0
    out.append([(l[1], l[2], int(l[3]) * int(l[4])) for l in log() if l[0] == "launch"])
    _keep.clear()
done(out)
""" % (json.dumps(shapes), mode))
    res = []
    for launches in ops:
        streams = {}
        for st, k, threads in launches:
            if "items" in k or "quarter" in k or "combine" in k or "stage" in k:
                streams.setdefault(st, []).append((k, threads))
        res.append(streams)
    return res


@pytest.mark.parametrize("mode", [0, 1])
def test_turns_run_in_the_form_that_was_priced(gpu_binding, mode):
    """Quarter turns by quads up to a wave of turns, by lanes above, for every number of
    levels a pass has."""
    shapes = [[15, 6, 2], [15, 3], [15, 11], [14, 14, 10, 9, 5], [12] * 3, [13], [16], [16] * 4]
    seen = set()
    for streams in _launches(gpu_binding, shapes, mode):
        for seq in streams.values():
            for i, (k, threads) in enumerate(seq):
                if "quarter" not in k:
                    continue
                quads = "true" in k
                slots = threads // (4 if quads else 1)               # two outputs each
                split = "true" in seq[i - 1][0]
                q = round(math.log2(seq[i + 1][1] / (2 * slots))) - 1 - split
                turns = slots - 2 * slots // 2 ** q
                seen.add((q, quads))
                assert quads == (turns <= WAVE), (q, slots, turns)
    assert {(2, True), (2, False)} <= seen and any(q > 2 for q, _ in seen)


# Batches of the same transform that take every form with turns (the small sizes' forms
# meet such tables in test_fft_passes.py).
BATCHES = {"pairs": [12], "lanes": [12] * 3, "lane_turns_two_groups": [12] * 32, "stages": [10] * 3 + [15]}


def test_batches_reach_every_form(gpu_binding):
    """The batches below and the golden sizes take, between them, every kind of pass."""
    shapes = list(BATCHES.values()) + [[3], [9], [17]]
    seen, streams = set(), {}
    for mode in (0, 1):
        for name, s in zip(list(BATCHES) + [None] * 3, _launches(gpu_binding, shapes, mode)):
            seen |= {k.replace("_", "") for seq in s.values() for k, _ in seq}
            streams[name] = len(s)
    want = {"kfftitems<1,false>", "kfftitems<2,false>", "kfftitems<4,false>", "kfftitems<4,true>",
            "kfftquarter<true>", "kfftquarter<false>", "kfftstagemulti<4>", "kfftstagemulti<6>", "kfftcombine"}
    assert want <= seen, want - seen
    assert streams["lane_turns_two_groups"] == 2 and streams["pairs"] == 1


@pytest.fixture(scope="module")
def broken(gpu, oracle):
    """2^12 points, a root table with a tenth of its entries replaced, and the oracle's
    forward and inverse transforms over it."""
    n = 1 << 12
    rnd = random.Random(12)
    jac = oracle.jacobian_randomize(5, n, oracle.gen_points(5, n))
    ok, d = gpu.fr_fft_domain_init(n)
    assert ok
    d = bytearray(d)
    for i in range(1, n):
        if rnd.random() < 0.1:
            d[32 * i:32 * i + 32] = (rnd.randrange(R) * (1 << 256) % R).to_bytes(32, "little")
    d, want = bytes(d), []
    for inverse in (False, True):
        ok, out = oracle.p1_fft_with_domain(jac, n, d, n + 2, inverse)
        assert ok
        want.append([oracle.serialize(out[144 * i:144 * i + 144]) for i in range(n)])
    return n, jac, d, want


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("batch", ["pairs", "lanes", "lane_turns_two_groups"])
def test_partly_broken_tables(gpu, oracle, broken, batch, mode):
    n, jac, d, want = broken
    count = len(BATCHES[batch])
    rc, out = gpu.p1_fft_batch([jac] * count, [n] * count, [d] * count, [mode] * count)
    assert rc == 0
    first = bytes(out[0])
    assert [oracle.serialize(first[144 * i:144 * i + 144]) for i in range(n)] == want[mode]
    for other in out[1:]:
        for i in range(0, n, 37 if count > 4 else 1):
            assert oracle.serialize(bytes(other[144 * i:144 * i + 144])) == want[mode][i]


@pytest.mark.parametrize("n,xn,turns", [(4, 1, 0), (64, 1, 0), (4, 2, 1)])
def test_passes_without_products_are_not_priced_as_products(gpu_binding, n, xn, turns):
    """Where every block of a pass has one non-identity input (a truncated prefix) there is
    nothing to multiply: no quarter turns are launched for it."""
    import fake_cuda
    gpu_binding.load()
    names = fake_cuda.run(gpu_binding.LIB_PATH, """
n, xn = %d, %d
v, d = buf(144 * n), domain(n)
for i in range(xn):
    C.memset(v.value + 144 * i, 1, 144)
L.catmsm_p1_fft_truncated_prefix.restype = C.c_bool
assert L.catmsm_p1_fft_truncated_prefix(v, S(n), S(xn), d, S(n + 2))
done(kernels())
""" % (n, xn))
    assert any("k_fft_items" in k or "k_fft_stage" in k for k in names)
    assert sum("quarter" in k for k in names) == turns
