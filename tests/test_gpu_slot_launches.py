"""Calls on one slot of a large batch launch for that slot, and instances past the active ones cost their
launch only."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forward_us(pkg, lib, b, slot, field, calls=50):
    """Device time of the forward plane pass of set_physical."""
    nc = lib.mhd_kernel_class_count()
    launches, ms = (C.c_longlong * nc)(), (C.c_double * nc)()
    b.set_physical(slot, 0, field)
    best = 1e300
    for _ in range(3):
        pkg._lib.check(lib.mhd_profile_enable(b.handle, 1))
        for _ in range(calls):
            b.set_physical(slot, 0, field)
        pkg._lib.check(lib.mhd_profile_read(b.handle, launches, ms, nc))
        pkg._lib.check(lib.mhd_profile_enable(b.handle, 0))
        z = next(c for c in range(nc) if lib.mhd_kernel_class_name(c) == b"z_forward")
        assert launches[z] == calls
        best = min(best, ms[z] / calls * 1e3)
    return best


def test_one_slot_of_4096(pkg, lib):
    """At 16^3 a launch over the capacity has 20480 blocks in place of 5: many times the time.  One
    slot's launch is the same whatever the capacity; 1.5 leaves room for the timing of a few us."""
    n = 16
    field = np.random.default_rng(1).standard_normal((n, n, n)).astype(np.float32)
    us = []
    for cap in (1, 4096):
        with pkg.Batch(n, cap) as b:
            s = b.add(1e-3, 1e-3, 1e-3)
            us.append(_forward_us(pkg, lib, b, s, field))
            assert np.array_equal(b.get_physical(s, 1), np.zeros_like(field))
    assert us[1] < 1.5 * us[0], us


def _us_per_step(b, steps=60):
    b.step(4)
    b.synchronize()
    best = 1e300
    for _ in range(5):
        t = time.perf_counter()
        b.step(steps)
        b.synchronize()
        best = min(best, time.perf_counter() - t)
    return best / steps * 1e6


@pytest.mark.parametrize("n", [96, 128])
def test_a_nearly_empty_batch(pkg, n):
    """One box in a class of 16 steps in 1.25 times a single problem's time (192 us against 154 at 96^3):
    the blocks of the other instances start and return.  With their first loads it was 1.6 times; the
    limit lies between."""
    us = []
    for cap in (1, 16):
        with pkg.Batch(n, cap) as b:
            b.add(1e-3, 1e-3, 1e-4)
            us.append(_us_per_step(b))
    assert us[1] < 1.4 * us[0], us
