"""The batched affine accumulation of large G2 MSMs: bases k_i G with known k_i,
so the sum is (sum k_i s_i) G by one oracle multiplication.  Long, short and
uneven runs, doublings, cancelling pairs, infinities among the bases, skewed
scalars whose list is much shorter than its bound, second waves of tiles, and
the multi-instance chains of a fused batch."""
import os

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


def values(rng, n):
    a = rng.integers(0, 1 << 64, size=(n, 4), dtype=np.uint64)
    a[:, 3] &= np.uint64((1 << 60) - 1)  # below r
    return a


def dot(a, b):
    total = 0
    for at in range(0, len(a), 1 << 20):  # 16-bit limbs, sums exact in float64
        x = a[at:at + (1 << 20)].view(np.uint16).astype(np.float64)
        y = b[at:at + (1 << 20)].view(np.uint16).astype(np.float64)
        m = x.T @ y
        total += sum(int(m[i, j]) << (16 * (i + j)) for i in range(16) for j in range(16))
    return total % R


def expect(oracle, ks, sc):
    k = dot(ks, sc)
    return oracle.g2_mul(oracle.g2_gen(), k), k == 0


def make(rng, n, kind):
    ks, sc = values(rng, n), values(rng, n)
    if kind == "one_point":  # every addition of a bucket's first pairs is a doubling
        ks[:] = ks[0]
    elif kind == "few_points":
        ks[:] = ks[np.arange(n) % 7]
    elif kind == "infinities":
        ks[::3] = 0
    elif kind == "cancel":  # P and -P with equal scalars: sums at infinity
        for i in range(0, n - 1, 2):
            k = int.from_bytes(ks[i].tobytes(), "little")
            ks[i + 1] = arr([(R - k) % R])[0]
        sc[1::2] = sc[0::2][: len(sc[1::2])]
    elif kind == "same_scalar":
        sc[:] = sc[0]
    elif kind == "circom":
        u = rng.random(n)
        sc[u < 0.7, 1:] = 0
        sc[u < 0.55, 0] &= np.uint64(1)
    elif kind == "crowded":  # most records in few buckets, the rest in runs of one or two
        sc[: n // 2] &= np.uint64(0x0003000300030003)
    return ks, sc


@pytest.mark.parametrize("kind", ["uniform", "one_point", "few_points", "infinities", "cancel",
                                  "same_scalar", "circom", "crowded"])
@pytest.mark.parametrize("n,c", [(40001, 8), (60000, 12), (65535, 14)])
def test_windowed(api, oracle, kind, n, c):
    rng = np.random.default_rng(n + len(kind))
    ks, sc = make(rng, n, kind)
    px, py = api.mul_generator(2, ks)
    want, winf = expect(oracle, ks, sc)
    try:
        api.msm_set_config(2, c=c)
        got, inf = api.msm_g2(px, py, sc)
    finally:
        api.msm_set_config(2)
    assert inf == winf and np.array_equal(got, want)


@pytest.mark.parametrize("kind", ["uniform", "circom"])
def test_windowed_second_wave(api, oracle, kind):
    """18 windows of 2^20 + 1 points: 18.9 M records, where a wave of tiles on 148 SMs
    holds 14.5 M; the second wave reuses the scratch of the first, and runs of
    one bucket cross from one to the other"""
    n = (1 << 20) + 1
    rng = np.random.default_rng(20 + len(kind))
    ks, sc = make(rng, n, kind)
    px, py = api.mul_generator(2, ks)
    got, inf = api.msm_g2(px, py, sc)
    want, winf = expect(oracle, ks, sc)
    assert inf == winf and np.array_equal(got, want)


@pytest.mark.parametrize("n,c,kind", [(100003, 0, "uniform"), (100003, 14, "circom"),
                                      (90001, 13, "few_points"), (900001, 18, "uniform"),
                                      (1000003, 18, "uniform"), (1000003, 18, "circom")])
def test_fixed_base(api, oracle, n, c, kind):
    """900001 points (13.5 M records) are more than the 10.9 M of a wave of three
    blocks per SM, so four run; 1000003 (15.0 M) take two waves of those"""
    rng = np.random.default_rng(n + c)
    ks, sc = make(rng, n, kind)
    px, py = api.mul_generator(2, ks)
    t = api.MsmTable(2, px, py, c=c)
    got, inf = t.run(sc)
    want, winf = expect(oracle, ks, sc)
    assert inf == winf and np.array_equal(got, want)
    part = sc[: n // 3]
    got, inf = t.run(part)
    t.close()
    want, winf = expect(oracle, ks[: n // 3], part)
    assert inf == winf and np.array_equal(got, want)


def test_fused_batch_shares_the_chain(api, tmp_path):
    """the B2 MSMs of a group are one list of several instances; each proof is
    the one the circuit gives alone"""
    circuits, wits = [], []
    for i, log_n in enumerate((16, 14, 16)):
        z, w = os.path.join(tmp_path, f"c{i}.zkey"), os.path.join(tmp_path, f"c{i}.wtns")
        api.synth_circuit(z, w, log_n, nnz=(1, 3), witness="uniform", seed=40 + i)
        c = api.Circuit(z)
        c.precompute(14, 14)
        circuits.append(c)
        wits.append(api.read_wtns(w))
    alone = [c.prove(w) for c, w in zip(circuits, wits)]
    api.set_batch_mode(api.BATCH_FUSED)
    try:
        got = api.prove_batch(circuits, wits)
    finally:
        api.set_batch_mode(api.BATCH_AUTO)
    for a, b in zip(alone, got):
        assert np.array_equal(a, b)
