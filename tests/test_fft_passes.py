"""The multi-level passes of the G1 FFT (fft.cu k_fft_items / k_fft_combine).

CPU: the item numbering restated in Python is a bijection, and the sums over
items equal the radix-2 network level by level, over the integers mod r, for
an arbitrary root table.  GPU: transforms whose passes take every q, with
identity and repeated points and a root table that is no group, against the
oracle's radix-2 transform."""
import random

import pytest

R = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001


def items_of(q):
    return 1 + (4 ** q - 1) // 3


def decode(it):
    """Item index -> (m, k mod 2^t), as k_fft_items decodes it."""
    if it == 0:
        return 0, 0
    top, rem = 1, it - 1
    while rem >= top * top:
        rem -= top * top
        top *= 2
    return top + rem // top, rem % top


def item_of(m, k):
    if m == 0:
        return 0
    t = m.bit_length() - 1
    top = 1 << t
    return 1 + (top * top - 1) // 3 + (m - top) * top + (k & (top - 1))


@pytest.mark.parametrize("q", [1, 2, 3, 4])
def test_item_numbering(q):
    seen = set()
    for it in range(items_of(q)):
        m, k = decode(it)
        assert 0 <= m < 1 << q and item_of(m, k) == it
        seen.add((m, k))
    assert len(seen) == items_of(q)
    assert {item_of(m, k) for m in range(1 << q) for k in range(1 << q)} == set(range(items_of(q)))


@pytest.mark.parametrize("n,split", [(16, (4,)), (16, (1, 3)), (32, (2, 3)), (64, (3, 1, 2))])
@pytest.mark.parametrize("inverse", [False, True])
def test_passes_equal_radix2(n, split, inverse):
    rnd = random.Random(n)
    roots = [rnd.randrange(R) for _ in range(n)]
    x = [rnd.randrange(R) for _ in range(n)]

    def root(pos, length):
        idx = pos * (n // length)
        return 1 if pos == 0 else roots[n - idx if inverse else idx]

    ref, length = list(x), 2
    while length <= n:
        h = length // 2
        for g in range(0, n, length):
            for j in range(h):
                u, v = ref[g + j], ref[g + j + h] * root(j, length)
                ref[g + j], ref[g + j + h] = (u + v) % R, (u - v) % R
        length *= 2
    a, s0 = list(x), 0
    for q in split:
        h, out = 1 << s0, list(a)
        for g in range(0, n, h << q):
            for j in range(h):
                prod = []
                for it in range(items_of(q)):
                    m, k = decode(it)
                    c = 1
                    for i in range(q):
                        if m >> i & 1:
                            c = c * root(j + h * (k & ((1 << i) - 1)), 2 * h << i) % R
                    prod.append(c * a[g + j + m * h] % R)
                for k in range(1 << q):
                    out[g + j + k * h] = sum((-1) ** bin(m & k).count("1") * prod[item_of(m, k)]
                                             for m in range(1 << q)) % R
        a, s0 = out, s0 + q
    assert a == ref


def booth4(k):
    d, carry = [], 0
    for i in range(32):
        v = (k >> (4 * i) & 15) + carry
        carry = 1 if v > 8 else 0
        d.append(v - 16 * carry)
    return d + [carry]


def test_booth4_digits():
    rnd = random.Random(4)
    for k in [0, 1, 8, 9, (1 << 128) - 1, 0x8888 << 100, 0x99999999999999999999999999999999] + \
            [rnd.randrange(1 << 128) for _ in range(5000)]:
        d = booth4(k)
        assert sum(x << (4 * i) for i, x in enumerate(d)) == k and all(-7 <= x <= 8 for x in d)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 4, 8, 32, 256])
@pytest.mark.parametrize("mode", ["fwd", "inv", "unscaled"])
def test_passes_match_oracle(gpu, oracle, n, mode):
    rnd = random.Random(100 + n)
    jac = bytearray(oracle.jacobian_randomize(n, n, oracle.gen_points(n, n)))
    for i in range(1, n, 5):
        jac[144 * i:144 * i + 144] = bytes(144)               # the identity
    for i in range(3, n, 7):
        jac[144 * i:144 * i + 144] = jac[:144]                # a repeated point
    ok, d = gpu.fr_fft_domain_init(n)
    assert ok
    d = bytearray(d)
    for i in range(1, n):                                     # roots that form no group, some zero and one
        v = rnd.choice([0, 1, R - 1, rnd.randrange(R), rnd.randrange(R), rnd.randrange(1 << 64)])
        d[32 * i:32 * i + 32] = (v * (1 << 256) % R).to_bytes(32, "little")
    d = bytes(d)
    if mode == "unscaled":
        got, ref = (x.p1_ifft_unscaled_with_domain(bytes(jac), n, d, n + 2) for x in (gpu, oracle))
    else:
        got, ref = (x.p1_fft_with_domain(bytes(jac), n, d, n + 2, mode == "inv") for x in (gpu, oracle))
    assert got[0] and ref[0]
    for i in range(n):
        s = slice(144 * i, 144 * i + 144)
        assert oracle.serialize(got[1][s]) == oracle.serialize(ref[1][s]), i
