"""The measured multiply-add rates that the rooflines are read against."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_probe_runs_the_rows_as_wide_multiply_adds():
    """the carry-chain rate is that of aligned lo / hi pairs: above independent
    unpaired ones, and no more than 64 multiply-adds per clock and SM"""
    import torch
    from zyklop_b200._lib import check, lib
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rate = []
    for kind in (0, 1):
        v = ctypes.c_double(0)
        check(lib().zk_int_probe(None, kind, ctypes.byref(v)))
        rate.append(v.value)
    p = torch.cuda.get_device_properties(0)
    print("rows %.2f, independent %.2f T/s" % tuple(rate))
    assert rate[1] < rate[0] < 1.02 * 64 * p.multi_processor_count * 1.965e-3
