"""The compiled field products, squares, reductions and inverses at the edges of
their ranges, against Python integers.  The CPU tests of the carry chains check
the derivation; these run the code itself: limbs of all ones and zeros, values
next to the modulus, and operands of any 256 bits where the code takes them (the
partly reduced values of the transforms)."""
import numpy as np
import pytest

from _oracle import R

pytestmark = pytest.mark.gpu

P = 21888242871839275222246405745257275088696311157297823662689037894645226208583
M32 = (1 << 32) - 1
FIELDS = [(0, P), (1, R)]


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zyklop_b200 import api as A
    return A


def pack(xs):
    return np.array([[(x >> (64 * j)) & (2**64 - 1) for j in range(4)] for x in xs], np.uint64)


def unpack(a):
    return [int.from_bytes(row.tobytes(), "little") for row in a]


def pattern(mask):
    """a 256-bit value whose limb i is all ones where bit i of mask is set"""
    return sum(M32 << (32 * i) for i in range(8) if mask >> i & 1)


def canonical(m, seed):
    rng = np.random.default_rng(seed)
    xs = [0, 1, 2, m - 1, m - 2, m // 2, m // 2 + 1, (1 << 128) - 1, 1 << 128, (1 << 253) % m]
    xs += [pattern(mask) % m for mask in range(256)]
    return xs + [int.from_bytes(rng.bytes(32), "little") % m for _ in range(250)]


def any256(m):
    top = (1 << 256) - 1
    return [top, top - 1, 1 << 255, m, 2 * m - 1, 2 * m, 4 * m - 1] + [pattern(k) for k in range(256)]


@pytest.mark.parametrize("field,m", FIELDS, ids=["fp", "fr"])
def test_products_squares_and_inverses(api, field, m):
    rinv = pow(1 << 256, -1, m)
    xs = canonical(m, field)
    pairs = [(a, b) for a in xs[:60] for b in xs[:60]] + list(zip(xs, xs[::-1]))
    got = unpack(api.field_op(field, "mul", pack([a for a, _ in pairs]), pack([b for _, b in pairs])))
    assert got == [a * b * rinv % m for a, b in pairs]
    assert unpack(api.field_op(field, "sqr", pack(xs))) == [a * a * rinv % m for a in xs]
    rr = pow(1 << 256, 2, m)
    assert unpack(api.field_op(field, "inv", pack(xs))) == [
        pow(a, -1, m) * rr % m if a else 0 for a in xs]


@pytest.mark.parametrize("field,m", FIELDS, ids=["fp", "fr"])
def test_any_256_bit_operand_beside_a_reduced_one(api, field, m):
    """a product below 2^256 m reduces fully whatever its factors, and so does a
    square of a value below 2m; decoding takes any 256 bits"""
    rinv = pow(1 << 256, -1, m)
    wide, edge = any256(m), [0, 1, m - 1, m - 2, pattern(0x55) % m, pattern(0xAA) % m]
    pairs = [(a, b) for a in wide for b in edge]
    got = unpack(api.field_op(field, "mul", pack([a for a, _ in pairs]), pack([b for _, b in pairs])))
    assert got == [a * b * rinv % m for a, b in pairs]
    assert unpack(api.field_op(field, "decode", pack(wide))) == [a * rinv % m for a in wide]
    rr = pow(1 << 256, 2, m)
    assert unpack(api.field_op(field, "inv", pack(wide))) == [
        pow(a, -1, m) * rr % m if a % m else 0 for a in wide]
    lazy = [m, 2 * m - 1] + [m + x for x in canonical(m, 7) if x]
    assert unpack(api.field_op(field, "sqr", pack(lazy))) == [a * a * rinv % m for a in lazy]
