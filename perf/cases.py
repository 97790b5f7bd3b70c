"""The work a user of this prover has it do, as measurable cases.

Primitives go through the C ABI on device buffers, as a C or C++ caller uses
them; proofs go through the Python binding of the same calls with a host
witness.  Every result is an exact integer computation, so outputs are compared
exactly.
"""
import ctypes
import os
import tempfile

import numpy as np
import torch

from zyklop_b200 import api
from zyklop_b200._lib import check, lib

P = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
R = 0x30644E72E131A029B85045B68181585D2833E84879B97091_43E1F593F0000001
R_TOP = 0x30644E72E131A029
MONT = 1 << 256
M64 = (1 << 64) - 1

# generators as canonical integers: G1 = (1, 2), and the standard G2 generator
G1_GEN = (1, 2)
G2_GEN = ((10857046999023057135944570762232829481370756359578518086990519993285655852781,
           11559732032986387107991004021392285783925812861821192530917403151452391805634),
          (8495653923123431417604973247489272438418190587263600148770280649306958101930,
           4082367875863433681332203403145435568316851327593401208105741076214120093531))


def listed():
    return [
        # the smallest call: one short transform, bound by launches and latency
        {"name": "ntt_2e10", "kind": "ntt", "log_n": 10, "inverse": False},
        # a large transform on its own, inverse direction
        {"name": "intt_2e22", "kind": "ntt", "log_n": 22, "inverse": True},
        # the H polynomial of a 2^20-constraint proof: three coset INTT / NTT pairs
        {"name": "hpoly_2e20", "kind": "hpoly", "log_n": 20},
        # a small ragged MSM (verification-key sized sets, small circuits)
        {"name": "msm_g1_777", "kind": "msm", "group": 1, "n": 777, "dist": "uniform"},
        # an ordinary MSM over witness values as circom circuits make them
        {"name": "msm_g1_50021_circom", "kind": "msm", "group": 1, "n": 50021, "dist": "circom"},
        # a large G1 MSM, uniform scalars
        {"name": "msm_g1_2e22", "kind": "msm", "group": 1, "n": 1 << 22, "dist": "uniform"},
        # a mid-sized ragged G2 MSM
        {"name": "msm_g2_200003", "kind": "msm", "group": 2, "n": 200003, "dist": "uniform"},
        # fixed bases (a resident commitment key), more points than scalars
        {"name": "table_g1_300007", "kind": "table", "group": 1, "n": 300007, "used": 250000,
         "dist": "circom"},
        # a small proof against a resident circuit, blinded, without tables
        {"name": "prove_2e13_blind", "kind": "prove", "log_n": 13, "nnz_max": 4,
         "dist": "circom", "tables": False, "blind": True},
        # the headline: a 2^20-constraint proof, resident circuit with tables
        {"name": "prove_2e20", "kind": "prove", "log_n": 20, "nnz_max": 2, "dist": "uniform",
         "tables": True, "blind": False},
        # the drop-in one-shot call from zkey and wtns images in host memory
        {"name": "oneshot_2e17", "kind": "oneshot", "log_n": 17, "nnz_max": 4, "dist": "circom"},
        # a batch of uneven proofs over two resident circuits with tables
        {"name": "batch_12_2e12_2e15", "kind": "batch", "count": 12, "log_a": 12, "log_b": 15,
         "nnz_max": 3, "dist": "circom"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(2 ** rng.uniform(lo, hi)))


def draw(rng):
    """One more case of the same kinds: sizes over the same ranges, odd ones among them."""
    kind = rng.choice(["ntt", "hpoly", "msm", "msm", "table", "prove", "oneshot", "batch"])
    dist = rng.choice(["uniform", "circom"])
    if kind == "ntt":
        return {"kind": "ntt", "log_n": rng.randint(8, 23), "inverse": rng.random() < 0.5}
    if kind == "hpoly":
        return {"kind": "hpoly", "log_n": rng.randint(10, 20)}
    if kind == "msm":
        group = rng.choice([1, 2])
        n = _log_uniform(rng, 6, 21.5 if group == 1 else 19) | rng.randint(0, 1)
        return {"kind": "msm", "group": group, "n": n, "dist": dist}
    if kind == "table":
        group = rng.choice([1, 2])
        n = _log_uniform(rng, 8, 19 if group == 1 else 17) | rng.randint(0, 1)
        used = n if rng.random() < 0.5 else max(1, int(n * rng.uniform(0.3, 1.0)))
        return {"kind": "table", "group": group, "n": n, "used": used, "dist": dist}
    if kind == "prove":
        return {"kind": "prove", "log_n": rng.randint(10, 18), "nnz_max": rng.randint(2, 4),
                "dist": dist, "tables": rng.random() < 0.5, "blind": rng.random() < 0.5}
    if kind == "oneshot":
        return {"kind": "oneshot", "log_n": rng.randint(10, 18), "nnz_max": rng.randint(2, 4),
                "dist": dist}
    return {"kind": "batch", "count": rng.randint(3, 20), "log_a": rng.randint(10, 13),
            "log_b": rng.randint(13, 16), "nnz_max": rng.randint(2, 4), "dist": dist}


# ---------------------------------------------------------------- inputs
def _uniform(g, n):
    """n canonical values below r (the top limb stays below r's), 4 u64 limbs each"""
    a = g.integers(0, 1 << 64, size=(n, 4), dtype=np.uint64)
    a[:, 3] = g.integers(0, R_TOP, size=n, dtype=np.uint64)
    return a


def _scalars(g, n, dist):
    """uniform, or the circom-like mix: 55% bits, 15% below 2^64, 30% uniform"""
    a = _uniform(g, n)
    if dist == "circom":
        u = g.random(n)
        a[u < 0.70, 1:] = 0
        bits = u < 0.55
        a[bits, 0] &= np.uint64(1)
    return a


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


def _host_inputs(case, seed):
    g = np.random.default_rng([seed, len(case["kind"])])
    if case["kind"] == "ntt":
        return (_uniform(g, 1 << case["log_n"]),)
    if case["kind"] == "hpoly":
        return _uniform(g, 1 << case["log_n"]), _uniform(g, 1 << case["log_n"])
    n = case["n"]
    return _uniform(g, n), _scalars(g, case.get("used", n), case["dist"])


def _points(group, ks):
    """ks[i] * G on the device, x and y in arrays of their own"""
    n, w = len(ks), 4 if group == 1 else 8
    d = _device(ks)
    px = torch.empty((n, w), dtype=torch.int64, device="cuda")
    py = torch.empty((n, w), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    check(lib().zk_mul_generator(None, group, api.ptr(d), n, api.ptr(px), api.ptr(py)))
    return px, py


class _Table:
    """a resident fixed-base table, released with the state"""

    def __init__(self, group, px, py):
        h = ctypes.c_void_p()
        check(lib().zk_msm_table_create(None, group, api.ptr(px), api.ptr(py), px.shape[0], 0,
                                        ctypes.byref(h)))
        self.handle = h

    def __del__(self):
        if self.handle:
            lib().zk_msm_table_free(self.handle)
            self.handle = None


def _synth(folder, log_n, nnz_max, dist, seed):
    z, w = os.path.join(folder, "c%d.zkey" % log_n), os.path.join(folder, "c%d.wtns" % log_n)
    api.synth_circuit(z, w, log_n, n_public=8, n_private_inputs=8,
                      nnz=(2 if nnz_max == 2 else 1, nnz_max), witness=dist, seed=seed)
    return z, w


def _folder():
    shm = "/dev/shm"
    return tempfile.TemporaryDirectory(dir=shm if os.access(shm, os.W_OK) else None)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ntt", "hpoly"):
        src = [_device(a) for a in _host_inputs(case, seed)]
        s = {"case": case, "src": src, "work": [torch.empty_like(a) for a in src]}
        if kind == "hpoly":
            s["h"] = torch.empty_like(src[0])
        return s
    if kind in ("msm", "table"):
        ks, sc = _host_inputs(case, seed)
        px, py = _points(case["group"], ks)
        s = {"case": case, "sc": _device(sc)}
        if kind == "msm":
            s["px"], s["py"] = px, py
        else:
            s["table"] = _Table(case["group"], px, py)
        torch.cuda.synchronize()
        return s
    with _folder() as d:
        seed = seed & 0x7FFFFFFF
        if kind == "batch":
            circuits, witnesses = [], []
            for log_n in (case["log_a"], case["log_b"]):
                z, w = _synth(d, log_n, case["nnz_max"], case["dist"], seed + log_n)
                c = api.Circuit(z)
                c.precompute()
                circuits.append(c)
                witnesses.append(api.read_wtns(w))
            pick = [(i * 7 % 3) % 2 for i in range(case["count"])]
            return {"case": case, "circuits": [circuits[k] for k in pick],
                    "witnesses": [witnesses[k] for k in pick]}
        z, w = _synth(d, case["log_n"], case["nnz_max"], case["dist"], seed)
        if kind == "oneshot":
            with open(z, "rb") as f, open(w, "rb") as g:
                return {"case": case, "zkey": f.read(), "wtns": g.read()}
        c = api.Circuit(z)
        if case["tables"]:
            c.precompute()
        s = {"case": case, "circuit": c, "witness": api.read_wtns(w), "r": None, "s": None}
        if case["blind"]:
            g = np.random.default_rng(seed)
            s["r"], s["s"] = (int.from_bytes(g.bytes(32), "little") % R for _ in range(2))
        return s


# ---------------------------------------------------------------- the calls
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ntt":
        # the call works in place: this pass's input goes into its buffer first
        s["work"][0].copy_(s["src"][0])
        check(lib().zk_ntt(None, api.ptr(s["work"][0]), case["log_n"], int(case["inverse"])))
        return s["work"][0]
    if kind == "hpoly":
        for w, a in zip(s["work"], s["src"]):
            w.copy_(a)
        check(lib().zk_hpoly(None, api.ptr(s["work"][0]), api.ptr(s["work"][1]), case["log_n"],
                             api.ptr(s["h"])))
        return s["h"]
    if kind in ("msm", "table"):
        group = case["group"]
        out = np.zeros(8 if group == 1 else 16, dtype=np.uint64)
        inf = ctypes.c_int(0)
        po = out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))
        if kind == "table":
            check(lib().zk_msm_table_run(s["table"].handle, api.ptr(s["sc"]), case["used"], po,
                                         ctypes.byref(inf)))
        else:
            f = lib().zk_msm_g1 if group == 1 else lib().zk_msm_g2
            check(f(None, api.ptr(s["px"]), api.ptr(s["py"]), api.ptr(s["sc"]), case["n"], po,
                    ctypes.byref(inf)))
        return out.view(np.int64), inf.value
    if kind == "oneshot":
        return api.prove_mem(s["zkey"], s["wtns"]).view(np.int64)
    if kind == "batch":
        return api.prove_batch(s["circuits"], s["witnesses"]).view(np.int64)
    return s["circuit"].prove(s["witness"], s["r"], s["s"]).view(np.int64)


# ---------------------------------------------------------------- work
# Operations are 32-bit integer multiply-adds, two operations each.  A field
# product with its reduction is about 120 of them (64-bit results).
_PRODUCT = 240.0


def _ntt_work(log_n, transforms=1):
    n = 1 << log_n
    return {"bytes": 64.0 * n * transforms, "flops": _PRODUCT * transforms * n / 2 * log_n}


def _msm_work(group, n, dist, table=False):
    """one addition of 6 products (G1; about 2.2 times that on G2) per point and nonzero digit
    of windows of log2(n) bits"""
    bits = max(8, min(20, n.bit_length() - 1))
    digits = -(-254 // bits)
    if dist == "circom":
        digits = 0.30 * digits + 0.15 * -(-64 // bits) + 0.55 * 0.5
    point = 64 if group == 1 else 128
    reads = digits * point if table else point  # a table holds one record for each digit
    return {"bytes": n * (32.0 + reads), "flops": n * digits * 6 * _PRODUCT * (1 if group == 1 else 2.2)}


def _proof_work(log_n, nnz_max, dist, tables, blind, oneshot=False):
    n = 1 << log_n
    nnz = n * (2.0 if nnz_max == 2 else (1 + nnz_max) / 2) * 2
    parts = [_msm_work(1, n, dist, tables), _msm_work(1, n, dist, tables),
             _msm_work(2, n, dist, tables), _msm_work(1, n, "uniform", tables),
             {"bytes": 36 * nnz + 100.0 * n, "flops": _PRODUCT * nnz},
             {"bytes": 0.0, "flops": 6 * _PRODUCT * n / 2 * log_n}]
    if blind:
        parts.append(_msm_work(1, n, dist, tables))
    if oneshot:
        parts.append({"bytes": 320.0 * n + 44 * nnz, "flops": 0.0})
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    if kind == "ntt":
        return _ntt_work(case["log_n"])
    if kind == "hpoly":
        w = _ntt_work(case["log_n"], 6)
        w["bytes"] = 96.0 * (1 << case["log_n"])
        return w
    if kind in ("msm", "table"):
        return _msm_work(case["group"], case.get("used", case["n"]), case["dist"], kind == "table")
    if kind == "batch":
        parts = [_proof_work(case["log_b" if (i * 7 % 3) % 2 else "log_a"], case["nnz_max"],
                             case["dist"], True, False) for i in range(case["count"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    return _proof_work(case["log_n"], case["nnz_max"], case["dist"], case.get("tables", False),
                       case.get("blind", False), kind == "oneshot")


def tolerance(case):
    return "exact"


# ---------------------------------------------------------------- plain check
def _ints(a):
    b = np.ascontiguousarray(a).tobytes()
    return np.array([int.from_bytes(b[i:i + 32], "little") for i in range(0, len(b), 32)],
                    dtype=object)


def _limbs(v):
    return np.frombuffer(b"".join(int(x).to_bytes(32, "little") for x in v),
                         dtype=np.int64).reshape(-1, 4)


def _dft(x, log_n, root):
    """natural-order transform of an object array, radix 2"""
    n = 1 << log_n
    rev = np.zeros(1, dtype=np.int64)
    for _ in range(log_n):
        rev = np.concatenate([2 * rev, 2 * rev + 1])
    x = x[rev]
    for st in range(log_n):
        half = 1 << st
        w = np.empty(half, dtype=object)
        step, v = pow(root, n >> (st + 1), R), 1
        for i in range(half):
            w[i], v = v, v * step % R
        x = x.reshape(-1, 2, half)
        t = x[:, 1] * w % R
        x = np.stack([(x[:, 0] + t) % R, (x[:, 0] - t) % R], axis=1)
    return x.reshape(n)


def _root(log_n):
    return pow(5, (R - 1) >> log_n, R)


def _exact_hpoly(aw, bw, log_n):
    n, unmont = 1 << log_n, pow(MONT, -1, R)
    a, b = _ints(aw) * unmont % R, _ints(bw) * unmont % R
    shift, out = _root(log_n + 1), []
    for v in (a, b, a * b % R):
        c = _dft(v, log_n, pow(_root(log_n), -1, R)) * pow(n, -1, R) % R
        f, t = np.empty(n, dtype=object), 1
        for i in range(n):
            f[i], t = t, t * shift % R
        out.append(_dft(c * f % R, log_n, _root(log_n)))
    return _limbs((out[0] * out[1] - out[2]) % R)


class _Fp2:
    """a0 + a1 u with u^2 = -1 (a1 = 0 throughout for G1)"""

    def __init__(self, a, b=0):
        self.a, self.b = a % P, b % P

    def __add__(self, o):
        return _Fp2(self.a + o.a, self.b + o.b)

    def __sub__(self, o):
        return _Fp2(self.a - o.a, self.b - o.b)

    def __mul__(self, o):
        return _Fp2(self.a * o.a - self.b * o.b, self.a * o.b + self.b * o.a)

    def inv(self):
        n = pow(self.a * self.a + self.b * self.b, -1, P)
        return _Fp2(self.a * n, -self.b * n)


def _add(p, q):
    if p is None or q is None:
        return q if p is None else p
    (x1, y1), (x2, y2) = p, q
    d = x2 - x1
    if d.a or d.b:
        m = (y2 - y1) * d.inv()
    elif (y1.a, y1.b) == (y2.a, y2.b):
        m = x1 * x1 * _Fp2(3) * (y1 + y1).inv()
    else:
        return None
    x = m * m - x1 - x2
    return x, m * (x1 - x) - y1


def _mul_gen(group, k):
    g = tuple(_Fp2(c) for c in G1_GEN) if group == 1 else tuple(_Fp2(*c) for c in G2_GEN)
    acc = None
    for bit in bin(k % R)[2:]:
        acc = _add(acc, acc)
        if bit == "1":
            acc = _add(acc, g)
    return acc


def _dot(a, b):
    """sum a_i b_i of 256-bit values: 16-bit limbs, products summed exactly in float64"""
    total = 0
    for at in range(0, len(b), 1 << 20):
        x = np.ascontiguousarray(a[at:at + (1 << 20)][:len(b) - at]).view(np.uint16).astype(np.float64)
        y = np.ascontiguousarray(b[at:at + (1 << 20)]).view(np.uint16).astype(np.float64)
        m = x.T @ y
        total += sum(int(m[i, j]) << (16 * (i + j)) for i in range(16) for j in range(16))
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "ntt" and case["log_n"] <= 17:
        x, L = _ints(_host_inputs(case, seed)[0]), case["log_n"]
        if case["inverse"]:
            return _limbs(_dft(x, L, pow(_root(L), -1, R)) * pow(1 << L, -1, R) % R)
        return _limbs(_dft(x, L, _root(L)))
    if kind == "hpoly" and case["log_n"] <= 15:
        return _exact_hpoly(*_host_inputs(case, seed), case["log_n"])
    if kind in ("msm", "table"):
        ks, sc = _host_inputs(case, seed)
        p = _mul_gen(case["group"], _dot(ks[:len(sc)], sc))
        if p is None:
            return np.zeros(8 if case["group"] == 1 else 16, dtype=np.int64), 1
        c = [v for e in p for v in ((e.a,) if case["group"] == 1 else (e.a, e.b))]
        return _limbs([v * MONT % P for v in c]).reshape(-1), 0
    return None
