"""The division-step inversion (zyklop_b200/csrc/field_inv.cuh, plain C++)
compiled for the host and checked against Python's modular inverse (CPU only)."""
import ctypes
import os
import random
import subprocess

import pytest

from conftest import ROOT

P = 21888242871839275222246405745257275088696311157297823662689037894645226208583
R = 21888242871839275222246405745257275088548364400416034343698204186575808495617

SRC = """
#include "field_inv.cuh"
extern "C" void inv(const uint32_t* x, const uint32_t* m, uint32_t neg_inv30, uint32_t* out) {
  zk::inv_divsteps(x, m, neg_inv30, out);
}
"""


@pytest.fixture(scope="module")
def inv(tmp_path_factory):
    d = tmp_path_factory.mktemp("inv")
    src, so = d / "inv.cpp", d / "inv.so"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "zyklop_b200", "csrc"), "-o", str(so), str(src)])
    lib = ctypes.CDLL(str(so))
    words = ctypes.c_uint32 * 8

    def run(x, m):
        out = words()
        lib.inv(words(*[(x >> (32 * i)) & 0xFFFFFFFF for i in range(8)]),
                words(*[(m >> (32 * i)) & 0xFFFFFFFF for i in range(8)]),
                -pow(m, -1, 1 << 30) % (1 << 30), out)
        return sum(out[i] << (32 * i) for i in range(8))
    return run


@pytest.mark.parametrize("m", [P, R], ids=["fp", "fr"])
def test_inverse(inv, m):
    rng = random.Random(m & 0xFFFF)
    edge = [1, 2, 3, m - 1, m - 2, m // 2, m // 2 + 1, (1 << 30) - 1, 1 << 30, (1 << 253) % m]
    edge += [1 << i for i in range(253)] + [m - (1 << i) for i in range(253)]
    for x in edge + [rng.randrange(1, m) for _ in range(3000)]:
        assert inv(x, m) == pow(x, -1, m), hex(x)
    assert inv(0, m) == 0


@pytest.mark.parametrize("m", [P, R], ids=["fp", "fr"])
def test_unreduced_operands(inv, m):
    """any 256 bits: the field operations take values that are not reduced"""
    rng = random.Random(m & 0xFFF)
    top = (1 << 256) - 1
    for x in [m, 2 * m, 3 * m, 4 * m, 5 * m]:
        assert inv(x, m) == 0, hex(x)
    for x in [m + 1, 2 * m - 1, top, top - 1, 1 << 255] + [rng.getrandbits(256) for _ in range(3000)]:
        assert inv(x, m) == pow(x, -1, m), hex(x)
