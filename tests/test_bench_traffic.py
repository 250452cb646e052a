"""The benchmark's traffic figure is of the kernel that its roofline names: at
least that kernel's own bytes, and none where no capture of the kernel exists."""
import importlib.util
import os

from conftest import ROOT


def _bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_traffic_is_of_the_named_kernel():
    b = _bench()
    cells = 512 * 512 * 640
    assert 50 * cells <= b.ncu_traffic("scaling-box-512x512x640", "k_fused") < 100 * cells
    assert 39 * cells <= b.ncu_traffic("scaling-box-512x512x640", "k_step_e") < 50 * cells
    assert b.ncu_traffic("scaling-box-512x512x640", "k_other") is None
    assert b.ncu_traffic("no-such-box", "k_fused") is None
