"""The multiply-pair chains of zyklop_b200/csrc/field.cuh (fe_mul_wide,
fe_sqr_wide, fe_redc_lazy), restated word by word with carry-flag semantics and
checked against Python integers (CPU only).

A chain that the code ends without a carry (mac*_top, the odd-limb chain of a
reduction row, the last word of a sum) asserts here that none is lost, and a
word that takes a chain's carry must not overflow."""
import random

import pytest

P = 21888242871839275222246405745257275088696311157297823662689037894645226208583
R = 21888242871839275222246405745257275088548364400416034343698204186575808495617
M32 = (1 << 32) - 1


def limbs(x, n=8):
    return [(x >> (32 * i)) & M32 for i in range(n)]


def val(ws):
    return sum(w << (32 * i) for i, w in enumerate(ws))


def mac(e, at, xs, y, carry_to=None, cin=0):
    """e[at..] += xs (every second word) * y; the carry joins e[carry_to]"""
    c = cin
    for k, x in enumerate(xs):
        v = (x * y & M32) + e[at + 2 * k] + c
        e[at + 2 * k], c = v & M32, v >> 32
        v = (x * y >> 32) + e[at + 2 * k + 1] + c
        e[at + 2 * k + 1], c = v & M32, v >> 32
    if carry_to is None:
        assert c == 0, "carry out of a chain that drops it"
    else:
        e[carry_to] += c
        assert e[carry_to] <= M32, "carry word overflows"


def merge(E, O):
    t = val(E[:16]) + (val(O[:15]) << 32)
    assert t < 1 << 512 and O[15] == 0
    return limbs(t, 16)


def mul_wide(a, b):
    E, O = [0] * 17, [0] * 17
    mac(E, 0, a[0::2], b[0])
    mac(O, 0, a[1::2], b[0])
    for j in (1, 3, 5, 7):
        mac(O, j - 1, a[0::2], b[j], carry_to=j + 7)
        mac(E, j + 1, a[1::2], b[j])
        if j < 7:
            mac(E, j + 1, a[0::2], b[j + 1], carry_to=j + 9)
            mac(O, j + 1, a[1::2], b[j + 1])
    return merge(E, O)


def sqr_wide(a):
    E, O = [0] * 16, [0] * 16
    mac(O, 0, a[1::2], a[0])
    mac(E, 2, a[2::2], a[0])
    mac(O, 2, a[2::2], a[1], carry_to=8)
    mac(E, 4, a[3::2], a[1])
    mac(O, 4, a[3::2], a[2])
    mac(E, 6, a[4::2], a[2], carry_to=10)
    mac(O, 6, a[4::2], a[3], carry_to=10)
    mac(E, 8, a[5::2], a[3])
    mac(O, 8, a[5::2], a[4])
    mac(E, 10, a[6::2], a[4], carry_to=12)
    mac(O, 10, a[6::2], a[5], carry_to=12)
    mac(E, 12, a[7::2], a[5])
    mac(O, 12, a[7::2], a[6])
    T = limbs(2 * val(merge(E, O)), 16)
    c = 0
    for i in range(8):
        for k, part in ((2 * i, a[i] * a[i] & M32), (2 * i + 1, a[i] * a[i] >> 32)):
            v = part + T[k] + c
            T[k], c = v & M32, v >> 32
    assert c == 0
    return T


def redc_lazy(T, m):
    inv, p = -pow(m, -1, 1 << 32) % (1 << 32), limbs(m)
    A, B = T[:8] + [0] * 9, [0] * 17
    for i in range(8):
        s, o = (A, B) if i % 2 == 0 else (B, A)
        v = s[i] + o[i]
        s[i], c = v & M32, v >> 32
        q = s[i] * inv & M32
        mac(o, i + 1, p[1::2], q, cin=c)
        mac(s, i, p[0::2], q, carry_to=i + 8)
        assert s[i] == 0
    assert A[16] == 0 and B[16] == 0
    r = val(A[8:16]) + val(B[8:16])
    assert r < 1 << 256
    r += val(T[8:])
    assert r < 1 << 256
    return r


def operands(m, k, seed):
    rng = random.Random(seed)
    edge = [0, 1, 2, m - 1, m - 2, (1 << 128) - 1, 1 << 128, (1 << 253) % m, m // 2,
            val([M32, 0] * 4) % m, val([0, M32] * 4) % m]
    return edge + [rng.randrange(m) for _ in range(k)]


@pytest.mark.parametrize("m", [P, R], ids=["fp", "fr"])
def test_product_square_and_reduction(m):
    rinv = pow(1 << 256, -1, m)
    xs = operands(m, 250, 3)
    for i, a in enumerate(xs):
        for b in (xs[(7 * i + 3) % len(xs)], m - 1):
            T = mul_wide(limbs(a), limbs(b))
            assert val(T) == a * b
            r = redc_lazy(T, m)
            assert r < 2 * m and r % m == a * b * rinv % m
        S = sqr_wide(limbs(a))
        assert val(S) == a * a
        assert redc_lazy(S, m) % m == a * a * rinv % m


def test_wide_products_of_any_256_bit_values():
    rng = random.Random(5)
    top = (1 << 256) - 1
    xs = [0, 1, top, top - 1, 1 << 255, val([M32, 0] * 4), val([0, M32] * 4)]
    xs += [rng.getrandbits(256) for _ in range(60)]
    for a in xs:
        assert val(sqr_wide(limbs(a))) == a * a
        for b in xs[:12]:
            assert val(mul_wide(limbs(a), limbs(b))) == a * b


@pytest.mark.parametrize("m", [P, R], ids=["fp", "fr"])
def test_reduction_at_its_bounds(m):
    """T up to 2^256 m (below 2m afterwards) and low halves that carry everywhere"""
    rng = random.Random(9)
    rinv = pow(1 << 256, -1, m)
    lows = [0, 1, (1 << 256) - 1, (1 << 256) - (1 << 32), val([M32, 0] * 4), val([0, M32] * 4)]
    for hi in (0, 1, m - 1, rng.randrange(m)):
        for lo in lows + [rng.getrandbits(256) for _ in range(60)]:
            T = (hi << 256) + lo
            r = redc_lazy(limbs(T, 16), m)
            assert r < 2 * m and r % m == T * rinv % m
