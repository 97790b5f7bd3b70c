"""Scratch that is there for speed makes no call fail and holds none back: the
affine accumulation of G2, whose scratch is many times the rest of the arena, is
left out where the device has no room for it, and gives its memory back to a
call that needs it.  Results are the same either way."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 19  # windowed G2: 2.0 GB of scratch with the affine accumulation, 0.24 GB without


@pytest.fixture(scope="module")
def api():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zyklop_b200 import api as A
    return A


def context():
    from zyklop_b200._lib import check, lib
    h = ctypes.c_void_p()
    check(lib().zk_ctx_create(0, ctypes.byref(h)))
    return h


def destroy(h):
    from zyklop_b200._lib import check, lib
    check(lib().zk_ctx_destroy(h))
    check(lib().zk_release_cached_memory(None))


def free_bytes():
    """the device's free memory with the unused blocks of the library's pool"""
    import torch
    from zyklop_b200._lib import memory_stats
    s = memory_stats(0)
    return torch.cuda.mem_get_info()[0] + s["pool_reserved_bytes"] - s["pool_used_bytes"]


class Filled:
    """all but `left` bytes of the device's memory taken"""

    def __init__(self, left):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.held = []
        while (n := torch.cuda.mem_get_info()[0] - left) > 4 << 20:
            self.held.append(torch.empty(min(n, 16 << 30) >> 21 << 21, dtype=torch.uint8,
                                         device="cuda"))

    def close(self):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


def values(rng, n):
    a = rng.integers(0, 1 << 64, size=(n, 4), dtype=np.uint64)
    a[:, 3] &= np.uint64((1 << 60) - 1)
    return a


@pytest.fixture(scope="module")
def msm(api):
    """a large G2 MSM and its result with room for everything"""
    rng = np.random.default_rng(8)
    ks, sc = values(rng, N), values(rng, N)
    px, py = api.mul_generator(2, ks)
    h = context()
    want = api.msm_g2(px, py, sc, ctx=h)[0]
    destroy(h)
    return px, py, sc, want


def test_msm_runs_where_its_affine_scratch_does_not_fit(api, msm):
    px, py, sc, want = msm
    h = context()
    filled = Filled(1200 << 20)
    try:
        got = [api.msm_g2(px, py, sc, ctx=h)[0] for _ in range(2)]
        assert free_bytes() > 500 << 20
    finally:
        filled.close()
        destroy(h)
    assert all(np.array_equal(g, want) for g in got)


def test_an_msm_gives_its_scratch_back_to_a_call_that_needs_it(api, msm):
    px, py, sc, want = msm
    x1, y1 = api.mul_generator(1, values(np.random.default_rng(9), N))
    h = context()
    filled = Filled(3000 << 20)
    try:
        assert np.array_equal(api.msm_g2(px, py, sc, ctx=h)[0], want)
        before = free_bytes()
        assert before < 1300 << 20  # the affine scratch is held
        t = api.MsmTable(1, x1, y1, c=5, ctx=h)  # 51 multiples a point: 1.7 GB
        t.close()
        assert np.array_equal(api.msm_g2(px, py, sc, ctx=h)[0], want)
    finally:
        filled.close()
        destroy(h)


def test_server_admits_without_affine_scratch(api, tmp_path):
    """2^16 constraints: a slot takes about 0.1 GB, 0.4 GB with the affine scratch;
    in 0.5 GB beside the reserve two slots run, none waits"""
    z, w = os.path.join(tmp_path, "c.zkey"), os.path.join(tmp_path, "c.wtns")
    api.synth_circuit(z, w, 16, nnz=(1, 3), witness="uniform", seed=4)
    h = context()
    c = api.Circuit(z, ctx=h)
    wit = api.read_wtns(w)
    want = c.prove(wit)
    with api.Server(max_inflight=2, reserve_bytes=free_bytes() - (500 << 20), ctx=h) as srv:
        ts = [srv.submit(c, wit) for _ in range(6)]
        proofs = [srv.wait(t)[0] for t in ts]
        st = srv.stats()
    c.close()
    destroy(h)
    assert all(np.array_equal(p, want) for p in proofs)
    assert st["admission_waits"] == 0 and st["peak_inflight"] == 2, st


@pytest.mark.parametrize("tables,left", [(False, 2200), (True, 1600)])
def test_batches_run_where_not_every_slot_has_affine_scratch(api, tmp_path, tables, left):
    """six proofs of 2^17 constraints at once, in slots of their own (0.2 GB, 0.8 GB with
    the affine scratch) or in groups of two that share one list"""
    z, w = os.path.join(tmp_path, "c.zkey"), os.path.join(tmp_path, "c.wtns")
    api.synth_circuit(z, w, 17, nnz=(1, 3), witness="uniform", seed=5)
    h = context()
    c = api.Circuit(z, ctx=h)
    if tables:
        c.precompute()
    wit = api.read_wtns(w)
    want = c.prove(wit)
    mode = api.BATCH_FUSED if tables else api.BATCH_INFLIGHT
    api.set_batch_mode(mode, 2, ctx=h)
    filled = Filled(left << 20)
    try:
        proofs = api.prove_batch([c] * 6, [wit] * 6, inflight=6, ctx=h)
    finally:
        filled.close()
        c.close()
        destroy(h)
    assert all(np.array_equal(p, want) for p in proofs)
