"""The one-pass expansion level (k_ks_expand) in the ring of the PIR workloads, n = 2^12:
by default that ring takes the four-step kernels, with the threshold raised above it
the one-pass kernel, up to and past the last level that fits its tile."""
import ctypes

import pytest

import test_gpu_expand as base
from conftest import Q59, Q60

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,q,levels,log_b,items,count", [
    (12, Q59, 5, 20, 7, 2), (12, Q60, 3, 59, 1, 5), (12, Q60, 11, 30, 40, 1)])
def test_one_pass_level(sg, oracle, monkeypatch, log_n, q, levels, log_b, items, count):
    class Raised(sg.Context):
        def __init__(self, *args, **kw):
            super().__init__(*args, **kw)
            sg.check(sg.lib().shg_context_set_four_step_min(self.h, 14))

    monkeypatch.setattr(sg, "Context", Raised)
    lib = sg.lib()
    sg.check(lib.shg_profile_start())
    base.test_expand_and_absorb(sg, oracle, log_n, q, levels, log_b, items, count)
    sg.check(lib.shg_profile_stop())
    ms, launches = ctypes.c_double(), ctypes.c_uint64()
    sg.check(lib.shg_profile_query(b"ks_expand", ctypes.byref(ms), ctypes.byref(launches)))
    assert launches.value >= min(levels, 10)
