"""Generator of fp_sqr_impl (csrc/field.cuh): the unrolled 12-limb Montgomery
squaring.

Row i adds a_i * V_i with
    V_i = a_i 2^(32 i) + 2 sum_{j > i} a_j 2^(32 j),
whose limb j is a_i (j = i), a_{i+1} << 1 (j = i + 1; the bit shifted out
goes to the next limb) or (2a)_j = d[j] (j >= i + 2), and 0 below i.  The
accumulators are fp_mul_impl's: the product of limb j goes to the 64-bit slot at
word i + j, of e for even words and of o for odd ones; the even-j products of a
row form one carry chain into A (e for even i) with the carry in word i + 12,
the odd-j products one chain into B whose top word is fresh.  The Montgomery
rows and the final merge are fp_mul_impl's.

Run `python gen_fp_sqr.py` to print the function; the CPU test
tests/test_field_gen.py checks that field.cuh holds exactly this text.
"""

LO = ("mad.lo.cc.u32  ", "madc.lo.cc.u32 ")


def operand(i: int, j: int) -> str:
    """Limb j of V_i (j >= i)."""
    if j == i:
        return "a.v[%d]" % j
    if j == i + 1:
        return "(a.v[%d] << 1)" % j
    return "d[%d]" % j


def chain(acc: str, i: int, limbs: list, carry: bool) -> list:
    """acc += bi * (limbs of V_i) as one carry chain from word i + limbs[0];
    carry: assign the carry word, else assign the fresh top word."""
    m = len(limbs)
    w0 = i + limbs[0]
    b = "%%%d" % (3 * m + carry)
    body = []
    for k in range(m):
        src = "%%%d" % (2 * m + carry + k)
        top = k == m - 1 and not carry
        body.append("%s%%%d, %s, %s, %%%d;" % (LO[k > 0], 2 * k, src, b, 2 * k))
        body.append("%s%%%d, %s, %s, %s;" % ("madc.hi.u32    " if top else "madc.hi.cc.u32 ", 2 * k + 1, src, b,
                                             "0" if top else "%%%d" % (2 * k + 1)))
    if carry:
        body.append("addc.u32       %%%d, 0, 0;" % (2 * m))
    out = ['"%s"(%s[%d])' % ("=&r" if (k == 2 * m - 1 and not carry) else "+r", acc, w0 + k) for k in range(2 * m)]
    if carry:
        out.append('"=&r"(%s[%d])' % (acc, w0 + 2 * m))
    ins = ['"r"(%s)' % operand(i, j) for j in limbs] + ['"r"(bi)']
    lines = ['        asm("%s"' % (body[0] + ("\\n\\t" if len(body) > 1 else ""))]
    lines += ['            "%s"' % (x + ("\\n\\t" if n < len(body) - 2 else "")) for n, x in enumerate(body[1:])]
    lines.append("            : %s" % ", ".join(out))
    lines.append("            : %s);" % ", ".join(ins))
    return lines


def generate() -> str:
    L = ["__device__ __forceinline__ void fp_sqr_impl(fp& r, const fp& a)",
         "{",
         "    uint32_t e[26], o[26], d[12];",
         "#pragma unroll",
         "    for (int j = 1; j < 12; j++) d[j] = __funnelshift_l(a.v[j - 1], a.v[j], 1);   // (2a)_j"]
    for i in range(12):
        even = [j for j in range(i, 12) if j % 2 == 0]
        odd = [j for j in range(i, 12) if j % 2 == 1]
        A, B = ("e", "o") if i % 2 == 0 else ("o", "e")
        L.append("    {   // row %d" % i)
        L.append("        const uint32_t bi = a.v[%d];" % i)
        if i == 0:
            for j in even:
                L.append("        e[%d] = %s * bi;" % (j, operand(i, j)))
                L.append("        e[%d] = __umulhi(%s, bi);" % (j + 1, operand(i, j)))
            for j in odd:
                L.append("        o[%d] = %s * bi;" % (j, operand(i, j)))
                L.append("        o[%d] = __umulhi(%s, bi);" % (j + 1, operand(i, j)))
            L.append("        e[12] = 0;")
        else:
            if even:
                L += chain(A, i, even, True)
            else:
                L.append("        %s[%d] = 0;" % (A, i + 12))
            for j in odd:
                L.append("        // %s[%d..%d] += %s * bi;" % (B, i + j, i + j + 1, operand(i, j)))
            L += chain(B, i, odd, False)
        L.append("        mont_row(%s, %s, %d);" % (A, B, i))
        L.append("    }")
    L += ["    mont_merge(r, e, o);", "}"]
    return "\n".join(L) + "\n"


if __name__ == "__main__":
    print(generate(), end="")
