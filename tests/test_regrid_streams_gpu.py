"""Regrids of an AMR solve beside other work on the device, on a GB300.

A regrid builds its tables and lists on two streams; what it leaves must not depend on how these are scheduled.
The same run of steps and regrids, alone and while an ensemble of other solves keeps the device busy from
another thread, gives the same bits in every table and level.
"""
import threading

import numpy as np
import pytest

import jpsolver as J

pytestmark = pytest.mark.gpu

TABLES = ("ref0", "fof0", "rl0", "l1pcb", "l1oct", "f1pos", "l1grid", "ref1", "fof1", "rl1", "l2pl1", "l2oct", "skin0", "skin1")


def run(storage, regrids):
    with J.Solver("amr", n=32, re=800.0, l1_mode="sensor", l2_mode="sensor", storage=storage, develop_steps=20,
                  max_gb=16.0) as s:
        out = []
        for _ in range(regrids):
            s.step(3)
            s.regrid()
            out.append(s.counts())
        s.step(2)
        out += [s.table(t) for t in TABLES]
        out += [s.get_populations(lv, layout="blocked") for lv in range(3)]
        return out


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_regrids_beside_busy_streams_bit_exact(storage):
    alone = run(storage, 12)
    assert alone[-4 - len(TABLES)]["nf2"] > 0
    others = [J.Solver("uniform", n=n, re=400.0) for n in (64, 96, 128)]
    others += [J.Solver("amr", n=16, re=400.0, l1_mode="slab", l2_mode="all", max_gb=4.0) for _ in range(3)]
    e = J.Ensemble()
    for s in others:
        e.add(s)
    stop = threading.Event()
    failed = []

    def work():
        try:
            while not stop.is_set():
                e.step(8)
                e.sync()
        except Exception as x:  # noqa: BLE001 - reported by the test's thread
            failed.append(x)

    t = threading.Thread(target=work)
    t.start()
    try:
        busy = run(storage, 12)
    finally:
        stop.set()
        t.join()
    assert not failed
    e.close()
    for s in others:
        s.close()
    for a, b in zip(alone, busy):
        if isinstance(a, dict):
            assert a == b
        else:
            np.testing.assert_array_equal(a, b)


def test_diagnostics_after_a_pool_grew(tmp_path):
    # the buffer of the first diagnostic belongs to the smaller pools; a solver that loads the state, which has
    # not taken a diagnostic before, gives the same numbers
    n = 32
    kw = dict(n=n, re=800.0, l1_mode="sensor", l2_mode="sensor", frac1=0.1, frac2=0.1, develop_steps=2, max_gb=16.0)
    with J.Solver("amr", **kw) as s, J.Solver("amr", **kw) as t:
        s.diag()
        cap = s.counts()
        s.set_sensor_override(np.ones(cap["cnb0"], dtype=np.float32), np.ones((2 * n // 8) ** 3, dtype=np.float32))
        s.regrid()                                           # every block ties at the threshold
        grown = s.counts()
        assert grown["cap1"] > cap["cap1"] and grown["cap2"] > cap["cap2"]
        s.step(1)
        p = str(tmp_path / "grown.jps")
        s.save_state(p)
        t.load_state(p)
        assert s.diag() == t.diag()
