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


@pytest.mark.parametrize("name,nth", [("cudaMemcpyAsync", 2), ("cudaMemcpyAsync", 3), ("cudaStreamBeginCapture", 1),
                                      ("cudaStreamEndCapture", 1), ("cudaGraphInstantiate", 1),
                                      ("cudaGraphLaunch", 1), ("cudaEventRecord", 1), ("cudaEventRecord", 2)])
def test_failed_batch_reads_nothing_after_return(host, name, nth):
    """A batch whose scalars are page-locked (read in place) and that fails after
    their copy was queued: the stream is waited for before the call returns, no
    capture stays open, and the next batch works."""
    rc, ops, again = host("""
b = Basis(4096, 10)
counts = [4096] * 60                       # 60 x 4096 pairs: affine rounds, on two streams
sc = pin(buf(32 * sum(counts)), 32 * sum(counts))
clear()
fail(%r, %d)
rc = b.batch(counts, True, sc)
ops = log()
done([rc, ops, b.batch(counts, True, sc)])
""" % (name, nth))
    assert rc != 0 and again == 0 and ["failed", name] in ops
    copies = [i for i, o in enumerate(ops) if o[0] == "copy"]
    stream = ops[copies[0]][1]
    assert ["sync", stream] in ops[copies[-1]:]
    begun = [o for o in ops if o[0] == "begin"]
    assert len(begun) == len([o for o in ops if o[0] == "end"])


@pytest.mark.parametrize("n", [64, 4096, 20000])
@pytest.mark.parametrize("nth", [3, 4])
def test_failed_msm_reads_nothing_after_return(host, n, nth):
    """A host MSM whose workspaces cannot be had after its inputs' copies were
    queued (the first two allocations are the inputs') waits for them."""
    ops = host("""
n = %d
ptr = (P * 2)(buf(96 * n).value, None), (P * 2)(buf(32 * n).value, None)
fail("cudaMalloc", %d)
L.blst_p1s_mult_pippenger(buf(144), ptr[0], S(n), ptr[1], S(255), buf(64))
done(log())
""" % (n, nth))
    assert ["failed", "cudaMalloc"] in ops
    at = {o[1]: i for i, o in enumerate(ops) if o[0] == "copy"}
    assert at and all(["sync", stream] in ops[i:] for stream, i in at.items())


def test_msm_without_memory_for_the_affine_rounds(host):
    """An MSM that would run affine rounds and has memory for everything but their
    lists runs without them, keeps none of the lists, and runs them again later."""
    full, kept, rc, ran, later = host("""
n = 1 << 18
pts, sc = aligned(96 * n), buf(32 * n)
def call():
    clear()
    rc = L.catmsm_p1s_mult_pippenger_device(buf(144), pts, sc, S(32), S(n), S(255), S(0))
    return rc, ["k_aff_first" in kernels(), "k_accumulate" in kernels()]
L.catmsm_msm_affine_rounds(0)
call()
base = F.fake_used()
limit(base + (256 << 20))
L.catmsm_msm_affine_rounds(-1)
rc, ran = call()
kept = F.fake_used() - base
limit(0)
done([F.fake_used(), kept, rc, ran, call()])
""")
    assert rc == 0 and ran == [False, True] and kept == 0
    assert later == [0, [True, True]]                    # (k_accumulate: for sparse scalars)


@pytest.mark.parametrize("ns", [[1 << 12], [1 << 17], [1 << 15] * 3, [4, 1 << 10, 1 << 14]])
def test_fft_without_memory_for_products(host, ns):
    """Transforms that have memory for everything but a pass's products run a level
    of butterflies a pass, and several levels again later."""
    rc, ran, stages, later = host("""
ns = %r
dom = {n: domain(n) for n in set(ns)}
vals = (P * len(ns))(*[buf(144 * n).value for n in ns])
doms = (P * len(ns))(*[dom[n].value for n in ns])
modes = (C.c_int * len(ns))(*[i %% 3 for i in range(len(ns))])
def call():
    clear()
    rc = L.catmsm_p1_fft_batch(vals, sizes(ns), doms, modes, S(len(ns)))
    return rc, log()
total = sum(ns)
limit(total * (144 + 192 + 32 + 48) + 200 * 1024)
rc, ops = call()
names = [o[2] for o in ops if o[0] == "launch"]
limit(0)
rc2, ops2 = call()
done([rc, any("k_fft_items" in k for k in names), sum("k_fft_stage" in k for k in names),
      rc2 == 0 and any("k_fft_items" in o[2] for o in ops2 if o[0] == "launch")])
""" % ns)
    assert rc == 0 and not ran and later
    assert stages >= max(ns).bit_length() - 1


@pytest.mark.parametrize("n", [9000, 100003])
def test_checked_decode_without_memory_for_the_points(host, n):
    """Checked uncompressing with memory for its inputs and results but not for all
    the points between its two kernels: every element goes through both, in pieces."""
    rc, ops = host("""
n = %d
limit(n * (48 + 96 + 4) + (1 << 19))
rc = L.catmsm_p1s_uncompress(buf(96 * n), buf(48 * n), S(n), buf(4 * n), 1)
done([rc, log()])
""" % n)
    run = [o for o in ops if o[0] == "launch"]
    assert rc == 0 and len({o[1] for o in run}) == 1
    assert [o[2].split("<")[0] for o in run] == ["k_decode", "k_members"] * (len(run) // 2) and len(run) > 2
    assert sum(int(o[3]) for o in run if o[2].startswith("k_decode")) * 64 >= n


@pytest.mark.parametrize("name,nth", [("cudaEventRecord", 2), ("cudaStreamWaitEvent", 2)])
@pytest.mark.parametrize("call", ["msm", "fft"])
def test_failed_join_waits_for_the_second_stream(host, call, name, nth):
    """A call that forked a second stream and cannot join it waits for it: its buffers are
    the next call's."""
    rc, ops = host("""
if %r == "msm":
    n = 1 << 18
    pts, sc = aligned(96 * n), buf(32 * n)
    call = lambda: L.catmsm_p1s_mult_pippenger_device(buf(144), pts, sc, S(32), S(n), S(255), S(0))
else:
    n, k = 1 << 14, 6
    v, d = (P * k)(*[buf(144 * n).value for _ in range(k)]), domain(n)
    call = lambda: L.catmsm_p1_fft_batch(v, sizes([n] * k), (P * k)(*[d.value] * k), (C.c_int * k)(*[0] * k), S(k))
assert call() == 0
clear()
fail(%r, %d)
rc = call()
done([rc, log()])
""" % (call, name, nth))
    assert rc != 0 and ["failed", name] in ops
    launches = [(i, o[1]) for i, o in enumerate(ops) if o[0] == "launch"]
    assert len({st for _, st in launches}) == 2
    for st in {st for _, st in launches}:
        last = max(i for i, s in launches if s == st)
        if st != launches[0][1]:                              # the forked one
            assert ["sync", st] in ops[last:]


ENTRIES = {
    "fft": "L.blst_p1_fft_with_domain(buf(144 * n), S(n), domain(n), S(n + 2), C.c_bool(False))",
    "fft_oneshot": "L.blst_p1_fft(buf(144 * n), S(n), C.c_bool(True))",
    "fft_batch": "L.catmsm_p1_fft_batch((P * 1)(buf(144 * n).value), sizes([n]), (P * 1)(domain(n).value), "
                 "(C.c_int * 1)(1), S(1))",
    "fr_fft": "L.blst_fr_fft_with_domain(buf(32 * n), S(n), domain(n), S(n + 2), C.c_bool(False))",
    "tile": "L.blst_p1s_tile_pippenger(buf(144), (P * 2)(buf(96 * n).value, None), S(n), (P * 2)(buf(32 * n).value, None), "
            "S(255), buf(64), S(8), S(8))",
    "mult_fr": "L.blst_p1s_mult_pippenger_fr(buf(144), aligned(96 * n), buf(32 * n), S(n), buf(1 << 20), S(1 << 20))",
    "wbits": "L.blst_p1s_mult_wbits(buf(144), buf(96 * 8 * n), S(4), S(n), (P * 2)(buf(32 * n).value, None), S(255), buf(64))",
}


@pytest.mark.parametrize("name,nth", [("cudaMemcpyAsync", 2), ("cudaMalloc", 3)])
@pytest.mark.parametrize("entry", sorted(ENTRIES))
def test_failed_call_uses_nothing_after_return(host, entry, name, nth):
    """Every host entry that fails after a copy was queued waits for it."""
    ops = host("n = 1024\nfail(%r, %d)\n%s\ndone(log())" % (name, nth, ENTRIES[entry]))
    if ["failed", name] not in ops:
        pytest.skip("the call makes fewer of them")
    at = {o[1]: i for i, o in enumerate(ops) if o[0] == "copy"}
    assert all(["sync", stream] in ops[i:] for stream, i in at.items())
