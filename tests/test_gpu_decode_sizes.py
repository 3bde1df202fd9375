"""Decoding and membership at the line between the quad and the lane form
(one wave of quads: 64 elements per SM) and at ragged ends: every element of
a mixed batch gets the same code and bytes at every batch size."""
import pytest

pytestmark = pytest.mark.gpu

P = 0x1a0111ea397fe69a4b1ba7b6434bacd764774b84f38512bf6730d2a0f6b0f6241eabfffeb153ffffb9feffffffffaaab


def test_decode_same_at_every_size(gpu, oracle, synth):
    import torch
    line = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    base = 61
    pts = gpu.points_from_scalars(synth.point_scalars(9, base), base)
    one = ((1 << 384) % P).to_bytes(48, "little")
    enc = bytearray(b"".join(oracle.compress(pts[96 * i:96 * i + 96] + one) for i in range(base)))
    for i in range(0, base, 4):
        enc[48 * i + 7] ^= 0x3c                                # mostly not on the curve or not in the group
    enc[48:96] = bytes([0xc0]) + bytes(47)                     # the identity
    enc[96:144] = bytes([0x80]) + bytes(47)                    # x = 0: a point of order 3
    enc[144] &= 0x7f                                           # no compression flag
    rc, ref, aff = gpu.p1s_decode(bytes(enc), base, True, check_group=True)
    assert rc == 0 and set(ref) >= {0, 1, 2, 3}
    ok = [i for i in range(base) if ref[i] == 0]
    assert len(ok) > base // 2 and ref[0] in (2, 3) and ref[1] == 0 and ref[2] == 3 and ref[3] == 1
    for n in (1, 3, 33, line - 1, line, line + 1, line + 129):
        reps = n // base + 1
        rc, errs, out = gpu.p1s_decode((bytes(enc) * reps)[:48 * n], n, True, check_group=True)
        assert rc == 0 and errs == (ref * reps)[:n]
        assert out == (aff * reps)[:96 * n]
        rc, member = gpu.p1s_affine_in_g1(out, n)
        assert rc == 0 and all(member)                         # failed elements keep the zero bytes: the identity


@pytest.mark.parametrize("extra", [0, 1, 64, 65])
def test_decode_halves_same_codes_and_bytes(gpu, oracle, synth, extra):
    # one wave of lanes (512 elements per SM) is the line to two halves; every entry point
    import torch
    n = 512 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    base = 61
    pts = gpu.points_from_scalars(synth.point_scalars(9, base), base)
    one = ((1 << 384) % P).to_bytes(48, "little")
    comp = bytearray(b"".join(oracle.compress(pts[96 * i:96 * i + 96] + one) for i in range(base)))
    for i in range(0, base, 4):
        comp[48 * i + 7] ^= 0x3c
    flat = bytearray()
    for i in range(base):                                      # big-endian x, y; every fifth y changed
        c = [int.from_bytes(pts[96 * i + 48 * k:96 * i + 48 * k + 48], "little") * pow(1 << 384, -1, P) % P
             for k in (0, 1)]
        flat += c[0].to_bytes(48, "big") + ((c[1] + (i % 5 == 0)) % P).to_bytes(48, "big")
    reps = n // base + 1
    for data, elem, compressed in ((bytes(comp), 48, True), (bytes(flat), 96, False)):
        for check in (True, False):
            rc, ref, aff = gpu.p1s_decode(data, base, compressed, check_group=check)
            assert rc == 0 and len(set(ref)) > 1 and ref[1] == 0
            rc, errs, out = gpu.p1s_decode((data * reps)[:elem * n], n, compressed, check_group=check)
            assert rc == 0 and errs == (ref * reps)[:n] and out == (aff * reps)[:96 * n]
    rc, ref = gpu.p1s_affine_in_g1(aff, base)
    rc, member = gpu.p1s_affine_in_g1((aff * reps)[:96 * n], n)
    assert rc == 0 and list(member) == (list(ref) * reps)[:n]
