"""Recorded coarse steps beside calls of another thread that wait for the whole device, on a GB300.

A solver records its step after a few launches (or at once, with FLAG_GRAPH).  Meanwhile another thread's
cudaDeviceSynchronize has to succeed, as it does beside plain launches, and the steps are the same bits.
"""
import collections
import ctypes
import threading

import numpy as np
import pytest

import jpsolver as J

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, J.FLAG_GRAPH])
def test_recording_beside_a_thread_that_waits_for_the_device(flags):
    kw = dict(n=16, re=400.0, l1_mode="slab", l2_mode="all", max_gb=4.0)
    with J.Solver("amr", **kw) as s:
        for _ in range(4):
            s.step(1)
        s.sync()
        want = [s.get_populations(lv, layout="blocked") for lv in range(3)]
    rt = ctypes.CDLL("libcudart.so.13")
    codes, stop = collections.Counter(), threading.Event()

    def wait_for_device():
        rt.cudaSetDevice(0)
        while not stop.is_set():
            codes[rt.cudaDeviceSynchronize()] += 1

    t = threading.Thread(target=wait_for_device)
    t.start()
    try:
        for _ in range(40):
            with J.Solver("amr", flags=flags, **kw) as s:
                s.step(4)
                got = [s.get_populations(lv, layout="blocked") for lv in range(3)]
                s.step(8)
                s.sync()
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
    finally:
        stop.set()
        t.join()
    assert set(codes) == {0}, codes
