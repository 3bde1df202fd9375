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


def item_order(it, items, turns):
    """Started `it`-th -> (m, k mod 2^t), as k_fft_items numbers them."""
    x0 = items // 2 if turns else items - 1
    if it == x0:
        return 0, 0
    late, top, wide = it > x0, 1, 1
    rem = it - x0 if late else it
    while rem >= top * wide:
        rem -= top * wide
        top *= 2
        wide = top // 2 if turns else top
    return top + rem // wide, rem % wide + (wide if late else 0)


Z3 = pow(-0xd201000000010000, 3, R)


@pytest.mark.parametrize("n,q", [(4, 2), (16, 2), (16, 4), (64, 3), (64, 2)])
@pytest.mark.parametrize("broken", [False, True])
def test_quarter_turns_equal_the_products(n, q, broken):
    # per butterfly: the items a turn stands for against the sum that replaces them
    assert Z3 * Z3 % R == R - 1
    assert {item_order(i, items_of(q), t) for i in range(items_of(q)) for t in (0, 1)} == \
        {decode(i) for i in range(items_of(q))}
    w = pow(7, (R - 1) // n, R)
    rnd = random.Random(n + q)
    roots = [pow(w, i, R) for i in range(n)]
    if broken:
        for i in range(1, n, 3):
            roots[i] = rnd.randrange(R)
    turned = 0
    for s0 in range(0, n.bit_length() - q):
        h = 1 << s0
        for j in range(h):
            def root(t, pos):
                return roots[pos * (n >> (s0 + t + 1))] if pos else 1

            def coeff(m, k):
                c = 1
                for i in range(q):
                    if m >> i & 1:
                        c = c * root(i, j + h * (k & ((1 << i) - 1))) % R
                return c
            x = [rnd.randrange(R) for _ in range(1 << q)]
            for u in range(1, 1 << (q - 1)):
                t = u.bit_length()
                turn = 1 << (t - 1)
                k = u - turn
                e = Z3 * root(t, j + h * k) % R
                r3 = roots[(j + h * k) * (n >> (s0 + t + 1)) + n // 4]
                assert r3 == root(t, j + h * u)
                if r3 not in (e, R - e):
                    assert broken
                    continue
                turned += 1
                sign = 1 if r3 == e else -1
                ms = range(1 << t, 2 << t)
                want = sum((-1) ** bin(m & u).count("1") * coeff(m, u) * x[m] for m in ms) % R
                got = sign * Z3 * sum((-1) ** bin(m & u).count("1") * coeff(m, k) * x[m] for m in ms) % R
                assert want == got
    assert turned or broken


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 16, 64, 256])
@pytest.mark.parametrize("mode", ["fwd", "inv"])
def test_turns_where_only_some_roots_are_powers(gpu, oracle, n, mode):
    rnd = random.Random(7 + n)
    jac = oracle.jacobian_randomize(n, n, oracle.gen_points(n, n))
    ok, d = gpu.fr_fft_domain_init(n)
    assert ok
    d = bytearray(d)
    for i in range(1, n):
        if i > n // 4 and rnd.random() < 0.3:
            d[32 * i:32 * i + 32] = (rnd.randrange(R) * (1 << 256) % R).to_bytes(32, "little")
    got, ref = (x.p1_fft_with_domain(bytes(jac), n, bytes(d), n + 2, mode == "inv") for x in (gpu, oracle))
    assert got[0] and ref[0]
    for i in range(n):
        s = slice(144 * i, 144 * i + 144)
        assert oracle.serialize(got[1][s]) == oracle.serialize(ref[1][s]), i
