"""CPU checks of the batched decoding's copies: which are ordered before which,
over a fake CUDA runtime (see fake_cuda)."""
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def host(gpu_binding):
    gpu_binding.load()
    return lambda body: fake_cuda.run(gpu_binding.LIB_PATH, body)


def _before(ops):
    """before(i, j): operation i is complete when operation j starts, by stream order,
    events and host waits alone."""
    clock, events, done = {}, {}, {}          # stream -> operations known complete or in order before its next one
    host = set()
    for i, o in enumerate(ops):
        if o[0] in ("copy", "set", "launch"):
            seen = clock.setdefault(o[1], set())
            seen |= host
            done[i] = set(seen)
            seen.add(i)
        elif o[0] == "record":
            events[o[2]] = set(clock.get(o[1], set())) | host
        elif o[0] == "wait":
            clock.setdefault(o[1], set()).update(events.get(o[2], set()))
        elif o[0] == "sync":
            host |= clock.get(o[1], set())
    return lambda i, j: i in done[j]


DECODES = {
    "uncompress": "L.catmsm_p1s_uncompress(buf(96 * n), buf(48 * n), S(n), buf(4 * n), %d)",
    "deserialize": "L.catmsm_p1s_deserialize(buf(96 * n), buf(96 * n), S(n), buf(4 * n), %d)",
}


@pytest.mark.parametrize("n", [5, 77824, 77825, 200001])
@pytest.mark.parametrize("check", [0, 1])
@pytest.mark.parametrize("call", sorted(DECODES))
def test_arrays_are_read_before_they_are_written(host, call, check, n):
    """The caller's arrays may overlap: every upload precedes every download."""
    ops = host("n = %d\nassert %s == 0\ndone(log())" % (n, DECODES[call] % check))
    before = _before(ops)
    up = [i for i, o in enumerate(ops) if o[0] == "copy" and o[5] == "1"]
    down = [i for i, o in enumerate(ops) if o[0] == "copy" and o[5] == "2"]
    assert up and down
    assert all(before(i, j) for i in up for j in down)


@pytest.mark.parametrize("call,check,streams", [("deserialize", 0, 1), ("deserialize", 1, 2), ("uncompress", 0, 2)])
def test_two_streams_only_with_work(host, call, check, streams):
    """A large deserialization without the membership test is its copies: one stream."""
    ops = host("n = 100003\nassert %s == 0\ndone(log())" % (DECODES[call] % check))
    assert len({o[1] for o in ops if o[0] == "launch"}) == streams
