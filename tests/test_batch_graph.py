"""CPU check of the batched commitments' captured graph against its buffers.

A captured graph holds device addresses, so it may be replayed only while no
buffer that existed at its capture has been freed.  The library's host code
runs over a fake CUDA runtime that logs allocations, frees and replays (see
fake_cuda); the sequences are the ones in which a workspace moves between two
batches that would use the same graph.
"""
import pytest

import fake_cuda

SEQUENCES = {
    # a larger batch of the same number of MSMs, without the graph
    "more_pairs": """
b.batch([300] * 8, True)
b.batch([4096] * 8, False)
b.batch([300] * 8, True)
""",
    # more MSMs
    "more_msms": """
b.batch([300] * 8, True)
b.batch([300] * 64, False)
b.batch([300] * 8, True)
""",
    # a shorter chunk (more chunk carries), and back
    "chunk": """
b.batch([300] * 8, True)
b.config(10, 4)
b.batch([300] * 8, False)
b.config(10, 96)
b.batch([300] * 8, True)
""",
    # the affine rounds' lists: 64 x 4096 pairs run rounds
    "rounds": """
b.batch([4096] * 60 + [1] * 4, True)
b.config(10, 16)
b.batch([4096] * 64, False)
b.config(10, 96)
b.batch([4096] * 60 + [1] * 4, True)
""",
    # a larger batch that runs out of memory half-way
    "no_memory": """
b.batch([300] * 8, True)
limit(F.fake_used() + (1 << 22))
assert b.batch([4096] * 8, False) != 0
limit(0)
b.batch([300] * 8, True)
""",
}

PRELUDE = "b = Basis(4096, 10)\nclear()\n"


@pytest.mark.parametrize("name", sorted(SEQUENCES))
def test_no_replay_over_freed_buffers(gpu_binding, name):
    gpu_binding.load()
    ops = fake_cuda.run(gpu_binding.LIB_PATH, PRELUDE + SEQUENCES[name] + "done(log())")
    stale, replays = {}, 0
    for op in ops:
        if op[0] == "instantiate":
            stale[op[1]] = None
        elif op[0] == "free":
            for g in stale:
                stale[g] = stale[g] or op[1]
        elif op[0] == "destroy":
            stale.pop(op[1])
        elif op[0] == "replay":
            replays += 1
            assert stale[op[2]] is None, "graph replayed after a buffer was freed"
    assert replays == 2


def test_graph_is_kept_while_nothing_moves(gpu_binding):
    gpu_binding.load()
    ops = fake_cuda.run(gpu_binding.LIB_PATH, PRELUDE + """
for k in (300, 280, 300, 150, 299):
    b.batch([k] * 8, True)
done(log())
""")
    assert [o[0] for o in ops].count("instantiate") == 1 and [o[0] for o in ops].count("replay") == 5


def test_no_batch_over_freed_tables(gpu_binding):
    """A reconfiguration that runs out of memory has given up the old tables:
    batches fail until a configuration succeeds, whichever window it asks for."""
    gpu_binding.load()
    got = fake_cuda.run(gpu_binding.LIB_PATH, """
b = Basis(4096, 13)
b.batch([300] * 8, True)
limit(F.fake_used() + (1 << 20))
bad = [b.config(4, 96), b.batch([300] * 8, True), b.batch([300] * 8, False), b.config(4, 96)]
limit(0)
again = b.config(13, 96)
clear()
done([bad, again, b.batch([300] * 8, True), [l[0] for l in log()].count("instantiate")])
""")
    bad, again, ok, captures = got
    assert all(bad) and again == 0 and ok == 0 and captures == 1


def test_batches_around_a_rounds_threshold_share_the_captures(gpu_binding):
    """48 x 4096 pairs of 26 windows run one affine round, 30 x fewer none: batches of
    one size that alternate between the two are captured once each."""
    gpu_binding.load()
    ops = fake_cuda.run(gpu_binding.LIB_PATH, PRELUDE + """
for i in range(6):
    b.batch([4096] * 48 if i % 2 == 0 else [4096] * 30 + [1] * 18, True)
done(log())
""")
    kinds = [o[0] for o in ops]
    assert any("k_aff_first" in o[2] for o in ops if o[0] == "launch")
    assert any("k_accumulate" in o[2] for o in ops if o[0] == "launch")
    assert kinds.count("instantiate") == 2 and kinds.count("replay") == 6


@pytest.mark.parametrize("window,pairs,parts", [(13, 4096 * 29, False), (13, 4096 * 32, True), (11, 25599, False),
                                                (11, 25600, True), (12, 55855, True), (12, 55854, False),
                                                (14, 4096 * 32, False)])
def test_sort_follows_the_entries(gpu_binding, window, pairs, parts):
    """The sort by parts runs from 600 entries per bucket of an MSM on, for windows of 11
    to 13 bits, with and without the graph, whatever ran before."""
    gpu_binding.load()
    got = fake_cuda.run(gpu_binding.LIB_PATH, """
b = Basis(4096, %d)
counts = [%d // 64] * 63 + [%d - %d // 64 * 63]
seen = []
for graph in (False, True):
    for c in (counts, [1] * 64, counts, [1] * 64, counts):
        clear()
        assert b.batch(c, graph) == 0
        seen.append(["k_part_scatter" in kernels(), "k_scatter_batch" in kernels(), any(l[0] == "replay" for l in log())])
done(seen)
""" % (window, pairs, pairs, pairs))
    assert got[0] == got[2] == got[4] == [parts, not parts, False] and got[1] == got[3] == [False, True, False]
    assert got[5] == [parts, not parts, True]
    # both routes' graphs are kept (the second route's buffers may move once)
    assert got[8] == got[9] == [False, False, True]


@pytest.mark.parametrize("nmsm,pairs,inlined", [(256, 4, False), (256, 399, False), (256, 410, True), (32, 4096, False)])
def test_level_form_follows_the_fill(gpu_binding, nmsm, pairs, inlined):
    """The reduction's first level: inlined field operations in full launches over at
    least two entries a bucket, calls elsewhere."""
    gpu_binding.load()
    got = fake_cuda.run(gpu_binding.LIB_PATH, """
b = Basis(4096, 13)
clear()
b.batch([%d] * %d, False)
done([k for k in kernels() if k.startswith("k_reduce_level")])
""" % (pairs, nmsm))
    assert len(got) == 1 and ("true" in got[0]) == inlined


@pytest.mark.parametrize("window", [2, 8, 10])
def test_narrow_windows_sort_by_parts(gpu_binding, window):
    """Up to 512 buckets an MSM, where its parts fit shared memory (not 2 bits), always."""
    gpu_binding.load()
    got = fake_cuda.run(gpu_binding.LIB_PATH, """
b = Basis(4096, %d)
clear()
b.batch([1] * 8, False)
b.batch([4096] * 8, False)
done([k for k in kernels() if "scatter" in k])
""" % window)
    assert got == [("k_part_scatter" if window > 2 else "k_scatter_batch")] * 2
