"""Transforms whose last pass reorders and scales (natural order, 1/N), and the
partly reduced values between passes, bit-exact against the CPU oracle: every
small size, pass radixes that make one to four passes, both directions, and
operands at the edges of the range."""
import numpy as np
import pytest

from _oracle import R, arr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zyklop_b200 import api as A
    return A


def operands(log_n, kind):
    n = 1 << log_n
    if kind == "random":
        rng = np.random.default_rng(log_n)
        return arr([int.from_bytes(rng.bytes(32), "little") % R for _ in range(n)])
    if kind == "largest":
        return arr([R - 1] * n)
    if kind == "alternating":
        return arr([R - 1 if i & 1 else 0 for i in range(n)])
    return arr([R - 1 if i == n - 1 else 0 for i in range(n)])  # one value


@pytest.fixture
def radix(api):
    def use(log_n, bits):
        api.tune_import(f"ntt {log_n} {bits}")
    used = []
    yield lambda log_n, bits: (used.append(log_n), use(log_n, bits))
    for log_n in used:
        use(log_n, 8)


@pytest.mark.parametrize("log_n", range(1, 15))
def test_both_directions_and_radixes(api, oracle, radix, log_n):
    for kind in ("random", "largest", "alternating", "last"):
        a = operands(log_n, kind)
        want = [oracle.ntt(a, log_n, inv) for inv in (False, True)]
        for bits in (8, 5, 4):
            radix(log_n, bits)
            for inv in (False, True):
                assert np.array_equal(api.ntt(a, log_n, inv), want[inv]), (kind, bits, inv)


@pytest.mark.parametrize("log_n", range(1, 13))
def test_hpoly_radixes(api, oracle, radix, log_n):
    for kind in ("random", "largest", "alternating"):
        a, b = operands(log_n, kind), operands(log_n, kind)[::-1].copy()
        want = oracle.hpoly(a, b, log_n)
        for bits in (8, 4):
            radix(log_n, bits)
            assert np.array_equal(api.hpoly(a, b, log_n), want), (kind, bits)


@pytest.mark.parametrize("log_n", [13, 14, 15])
def test_hpoly_around_one_wave_of_coset_threads(api, oracle, log_n):
    """up to 2^13 a thread scales one vector's coefficient, from 2^14 on those of all three"""
    for kind in ("random", "largest"):
        a, b = operands(log_n, kind), operands(log_n, kind)[::-1].copy()
        assert np.array_equal(api.hpoly(a, b, log_n), oracle.hpoly(a, b, log_n)), kind
