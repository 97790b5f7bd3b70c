"""The tiles and the scratch of the batched affine accumulation
(zyklop_b200/csrc/affine_layout.hpp, plain C++), compiled for the host: for every
number of records per thread that the host can size for, and every smaller one
that a shorter list takes in the same layout (CPU only)."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SRC = """
#include "affine_layout.hpp"
extern "C" void shape(int S, int* out) {
  const zk::AffShape a = zk::aff_shape(S);
  const int v[] = {a.nsub, a.rows, (int)a.pre, (int)a.mask, (int)a.state, (int)a.bytes,
                   a.slots[0], a.slots[1]};
  for (int i = 0; i < 8; i++) out[i] = v[i];
}
extern "C" int limit(int S, int h, int buf) { return zk::aff_shape(S).limit(h, buf); }
extern "C" int span(size_t total, unsigned ntiles) { return zk::aff_span(total, ntiles); }
"""
T, POINT, PAIR = 128, 128, 64
SPANS = range(32, 193, 2)


@pytest.fixture(scope="module")
def lay(tmp_path_factory):
    d = tmp_path_factory.mktemp("affine")
    (d / "t.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-Wall", "-I",
                           os.path.join(ROOT, "zyklop_b200", "csrc"), "-o", str(d / "t.so"),
                           str(d / "t.cpp")])
    lib = ctypes.CDLL(str(d / "t.so"))
    lib.span.argtypes = [ctypes.c_size_t, ctypes.c_uint]
    return lib


def shape(lay, S):
    out = (ctypes.c_int * 8)()
    lay.shape(S, out)
    d = dict(zip(("nsub", "rows", "pre", "mask", "state", "bytes"), out))
    return dict(d, slots=(out[6], out[7]))


def test_every_region_holds_what_the_kernels_write(lay):
    for most in SPANS:
        a = shape(lay, most)
        lens = [min(most - 64 * h, 64) for h in range(a["nsub"])]
        assert a["nsub"] <= 3 and sum(lens) == most and min(lens) > 0
        # slot row of point j of sub-segment h: the buffers and sub-segments do
        # not overlap while no sub-segment holds more than its limit
        end = 0
        for buf, first in ((0, 0), (1, a["rows"])):
            for h, n in enumerate(lens):
                limit = lay.limit(most, h, buf)
                assert first + h * a["slots"][buf] >= end
                end = first + h * a["slots"][buf] + limit
                # a round of all pairs leaves half of the points, the next one a
                # quarter; a handful of points fits whatever their runs
                assert limit >= (n + 1) // 2 if buf else limit >= (n + 3) // 4
                assert n > 8 or limit == n
        assert end * T * POINT == a["pre"]
        # all pairs of a list of `most` records, or of a shorter one
        assert a["mask"] == a["pre"] + sum(n // 2 for n in lens) * T * PAIR
        assert a["state"] == a["mask"] + 3 * a["nsub"] * T * 8
        assert a["bytes"] == a["state"] + 4 * T
        # 16-byte vectors, 8-byte masks; the next block's scratch begins at bytes
        assert all(a[k] % 16 == 0 for k in ("pre", "mask", "state", "bytes"))
        for S in SPANS:
            if S <= most:
                short = [min(S - 64 * h, 64) for h in range((S + 63) // 64)]
                assert len(short) <= a["nsub"]
                assert all(x <= y for x, y in zip(short, lens))


def test_scratch_follows_the_records(lay):
    """slots of 1 1/4 points and half a pair a record, at most 7 % above that for the
    rounding and the masks, and never less for more records"""
    last = 0
    for S in SPANS:
        a = shape(lay, S)
        per_record = a["bytes"] / (S * T)
        assert per_record < 1.07 * (1.25 * POINT + 0.5 * PAIR) + 4, (S, per_record)
        assert a["bytes"] >= last
        last = a["bytes"]


def test_spans_cover_the_list(lay):
    for ntiles in (1, 7, 444, 592, 1184):
        for total in (0, 1, ntiles * T * 32 - 1, ntiles * T * 32, ntiles * T * 32 + 1,
                      ntiles * T * 100 + 17, ntiles * T * 192):
            S = lay.span(total, ntiles)
            assert 32 <= S <= 192 and S % 2 == 0 and S * ntiles * T >= total
