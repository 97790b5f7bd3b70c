"""Sums of unreduced products in zyklop_b200/csrc/field.cuh and curve_quad.cuh,
restated word by word and checked against Python integers on edge and random
operands (CPU only): the Fp2 product with two reductions (fp2_mul_call), the
difference of products with one (fp_mul_sub_call), the component of an Fp2
product that one lane of a pair forms (fp2_lane_mul_call) and the norm
(fp2_norm_call).  The wide products, squares and reductions they are made of
are those of test_field_pair_chains.py.

The CUDA code drops carries and borrows where its comments prove they cannot
occur (the top word of a sum, the final borrow of a subtraction whose result is
known nonnegative).  Here each of those places asserts that the dropped carry
is zero, so a bound that does not hold fails the test.  This pins the bounds of
the derivation; test_gpu_field_edges.py and the parity tests run the compiled
code."""
import random

import pytest

from test_field_pair_chains import limbs, mul_wide, redc_lazy, sqr_wide, val

P = 21888242871839275222246405745257275088696311157297823662689037894645226208583
R = 21888242871839275222246405745257275088548364400416034343698204186575808495617
M32 = (1 << 32) - 1


class Cc:
    """The carry flag of a chain of .cc instructions."""

    def __init__(self):
        self.f = 0

    def add(self, a, b, cin=False, cout=True):
        return self._out(a + b + (self.f if cin else 0), cout)

    def sub(self, a, b, cin=False, cout=True):
        v = a - b - (self.f if cin else 0)
        if cout:
            self.f = 1 if v < 0 else 0
        else:
            assert v >= 0, "borrow out of a chain that drops it"
        return v & M32

    def _out(self, v, cout):
        if cout:
            self.f = v >> 32
        else:
            assert v >> 32 == 0, "carry out of a chain that drops it"
        return v & M32


def chain_add(a, b):
    c = Cc()
    return [c.add(x, y, cin=i > 0, cout=i < len(a) - 1) for i, (x, y) in enumerate(zip(a, b))]


def chain_sub(a, b):
    c = Cc()
    return [c.sub(x, y, cin=i > 0, cout=i < len(a) - 1) for i, (x, y) in enumerate(zip(a, b))]


def redc(T, m):
    """fe_redc: one conditional subtraction after the lazy reduction"""
    assert val(T) < m << 256
    r = redc_lazy(T, m)
    assert r < 2 * m, "one conditional subtraction is not enough"
    return r - m if r >= m else r


def fp2_mul(a0, a1, b0, b1):
    s, t = chain_add(limbs(a0), limbs(a1)), chain_add(limbs(b0), limbs(b1))
    x, w = mul_wide(s, t), mul_wide(limbs(a0), limbs(b0))
    x = chain_sub(x, w)
    y = chain_add(w, limbs(P * P, 16))
    w = mul_wide(limbs(a1), limbs(b1))
    return redc(chain_sub(y, w), P), redc(chain_sub(x, w), P)


def fp_mul_sub(a, b, c, d):
    x = chain_add(mul_wide(limbs(a), limbs(b)), limbs(P * P, 16))
    return redc(chain_sub(x, mul_wide(limbs(c), limbs(d))), P)


def fp2_lane_mul(a, ao, b0, b1, c1):
    """one component: a b0 plus ao b1, which component 0 takes from p^2"""
    w = mul_wide(limbs(ao), limbs(b1))
    x = w if c1 else chain_sub(limbs(P * P, 16), w)
    return redc(chain_add(x, mul_wide(limbs(a), limbs(b0))), P)


def fp2_norm(a0, a1):
    return redc(chain_add(sqr_wide(limbs(a0)), sqr_wide(limbs(a1))), P)


def operands(m, k, seed):
    rng = random.Random(seed)
    edge = [0, 1, 2, m - 1, m - 2, (1 << 128) - 1, 1 << 128, (1 << 253) % m, m // 2]
    return edge + [rng.randrange(m) for _ in range(k)]


@pytest.mark.parametrize("m", [P, R], ids=["fp", "fr"])
def test_product_square_and_reduction(m):
    rinv = pow(1 << 256, -1, m)
    xs = operands(m, 300, 11)
    for i, a in enumerate(xs):
        b = xs[(7 * i + 3) % len(xs)]
        T = mul_wide(limbs(a), limbs(b))
        assert val(T) == a * b
        assert redc(T, m) == a * b * rinv % m
        S = sqr_wide(limbs(a))
        assert val(S) == a * a
        assert redc(S, m) == a * a * rinv % m


def test_wide_products_up_to_2_255():
    """Unreduced sums of two field elements (< 2p < 2^255) enter the products."""
    rng = random.Random(5)
    xs = [(1 << 255) - 1, (1 << 254) + 12345, 2 * P - 2] + [rng.getrandbits(255) for _ in range(100)]
    for a in xs:
        for b in xs[:6]:
            assert val(mul_wide(limbs(a), limbs(b))) == a * b
        assert val(sqr_wide(limbs(a))) == a * a


def test_fp2_product_two_reductions():
    rinv = pow(1 << 256, -1, P)
    xs = operands(P, 200, 13)
    cases = [(xs[i], xs[i + 1], xs[i + 2], xs[(5 * i + 1) % len(xs)]) for i in range(len(xs) - 3)]
    cases += [(a, b, c, d) for a in (0, P - 1) for b in (0, P - 1) for c in (0, P - 1) for d in (0, P - 1)]
    for a0, a1, b0, b1 in cases:
        c0, c1 = fp2_mul(a0, a1, b0, b1)
        assert c0 == (a0 * b0 - a1 * b1) * rinv % P
        assert c1 == (a0 * b1 + a1 * b0) * rinv % P
        # the same product by two lanes, each with its own and its partner's part
        assert fp2_lane_mul(a0, a1, b0, b1, False) == c0
        assert fp2_lane_mul(a1, a0, b0, b1, True) == c1
        assert fp2_norm(a0, a1) == (a0 * a0 + a1 * a1) * rinv % P


def test_difference_of_products_one_reduction():
    rinv = pow(1 << 256, -1, P)
    xs = operands(P, 200, 17)
    for i in range(len(xs) - 3):
        a, b, c, d = xs[i], xs[i + 1], xs[i + 2], xs[(3 * i + 5) % len(xs)]
        assert fp_mul_sub(a, b, c, d) == (a * b - c * d) * rinv % P
    for a, c in ((0, P - 1), (P - 1, 0), (P - 1, P - 1)):
        assert fp_mul_sub(a, P - 1, c, P - 1) == (a * (P - 1) - c * (P - 1)) * rinv % P
