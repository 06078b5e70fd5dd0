"""Regrids of an AMR solve, on a GB300: beside other work on the device, with pools that grow, and refused.

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


def test_refused_level2_growth_needs_a_new_state(tmp_path):
    # ties on level 1 ask for more level-2 blocks than the budget holds: the regrid reports it, the calls that need
    # a grid refuse, and a state file or a new initial state brings the solve back to the same bits
    n, cnb0, ng1 = 32, 64, 512
    rng = np.random.default_rng(3)
    sen0 = (2.0 * (np.arange(cnb0) < cnb0 // 2) + 0.5 * rng.random(cnb0)).astype(np.float32)
    with J.Solver("amr", n=n, re=800.0, l1_mode="sensor", l2_mode="sensor", frac1=0.5, frac2=0.1, develop_steps=2,
                  max_gb=0.11, flags=J.FLAG_DEFER_INIT) as s:
        distinct = rng.random(ng1).astype(np.float32)

        def start():
            s.set_sensor_override(sen0, distinct)
            s.init_tgv()
            s.step(2)
            return s.diag()

        first = start()
        assert 0 < s.counts()["nf2"] <= s.counts()["cap2"] < 1024
        p = str(tmp_path / "ok.jps")
        s.save_state(p)
        for back in ("load", "init"):
            s.set_sensor_override(sen0, np.ones(ng1, dtype=np.float32))
            with pytest.raises(J.JPError) as x:
                s.regrid()
            assert x.value.status == 3                           # JP_ERR_CAPACITY
            for call in (s.diag, s.regrid, lambda: s.step(1)):
                with pytest.raises(J.JPError) as x:
                    call()
                assert x.value.status == 5                       # JP_ERR_STATE
            c = s.counts()
            assert c["nf1"] == c["nf2"] == 0
            assert [s.population_count(lv) for lv in range(3)] == [19 * n ** 3, 0, 0]
            assert s.output_fields()[0].size == (4 * n) ** 3     # of the coarse level
            if back == "load":
                s.load_state(p)
                assert s.diag() == first
            else:
                assert start() == first
