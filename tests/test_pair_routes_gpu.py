"""Where the two-step pass is taken, and its bits there, on a GB300: lone cubes, ensembles and served solves.

The launches are counted, so that a case that is meant to take the pass cannot be one that compares single steps
with themselves.  Every FP32 result is compared with steps taken one at a time (`step(1)` never takes the pass).
"""
import math

import numpy as np
import pytest

import jpsolver as J

pytestmark = pytest.mark.gpu


def mb_of(n):
    return 8 if n % 8 == 0 else 4


def cube(n, re=400.0, **kw):
    return J.Solver("uniform", n=n, re=re, mb=mb_of(n), **kw)


def launches(call):
    c0 = J.launch_count()
    call()
    return J.launch_count() - c0


def one_at_a_time(n, steps, re=400.0, **kw):
    with cube(n, re, **kw) as s:
        assert launches(lambda: [s.step(1) for _ in range(steps)]) == steps
        return s.get_populations()


# one tile and less than one (4, 8), ragged along x (12, 92, 132, 180, 260) and y (40, 92, 256), chunks with a remainder
# (92, 132, 256, 260), and more items than SMs, so that a CTA walks several (132: 297, 180: 300, 256: 580, 260: 910)
@pytest.mark.parametrize("n", [4, 8, 12, 40, 92, 132, 180, 256, 260])
def test_lone_cubes_that_take_the_pass(n):
    with cube(n) as s:
        assert launches(lambda: s.step(5)) == 3
        a = s.get_populations()
    np.testing.assert_array_equal(a, one_at_a_time(n, 5))


@pytest.mark.parametrize("n,kw", [(44, {}), (64, {}), (68, {}), (100, {}), (48, dict(storage="fp16")), (32, dict(storage="fp64")),
                                  (128, dict(vec=4)), (128, dict(threads_per_block=128)), (32, dict(flags=J.FLAG_INPLACE))])
def test_lone_cubes_that_step_one_at_a_time(n, kw):
    with cube(n, **kw) as s:
        assert launches(lambda: s.step(4)) == 4


# the mapping tests of the single step, a step at a time whatever the plan
@pytest.mark.parametrize("vec,tpb", [(1, 256), (2, 128), (4, 64), (4, 128), (4, 256), (4, 512)])
def test_chosen_mappings_are_used_by_every_step(vec, tpb):
    with cube(32, vec=vec, threads_per_block=tpb) as s:
        assert launches(lambda: s.step(3)) == 3
        np.testing.assert_array_equal(s.get_populations(), one_at_a_time(32, 3))


def amr_members():
    return [J.Solver("amr", n=n, re=400.0, l1_mode="slab", l2_mode="all", max_gb=4.0) for n in (16, 24)]


def step_launches(members, steps):
    e = J.Ensemble()
    for s in members:
        e.add(s)
    n = launches(lambda: e.step(steps))
    e.sync()
    e.close()
    return n


@pytest.mark.parametrize("with_amr", [False, True])
@pytest.mark.parametrize("steps", [2, 5])
@pytest.mark.parametrize("sizes", [(32, 48, 64, 96, 128) * 2, (132, 124, 108, 100, 100, 92, 76, 60)])
def test_ensembles_that_take_the_pass(sizes, steps, with_amr):
    cubes = [cube(n, 200.0 + 50.0 * i) for i, n in enumerate(sizes)]
    amr = amr_members() if with_amr else []
    alone = amr_members() if with_amr else []
    of_amr = step_launches(alone, steps) if with_amr else 0
    # one launch per two steps of all cubes, one for the odd step
    assert step_launches(cubes + amr, steps) - of_amr == steps // 2 + steps % 2
    for i, (n, s) in enumerate(zip(sizes, cubes)):
        assert s.info["step_count"] == steps
        np.testing.assert_array_equal(s.get_populations(), one_at_a_time(n, steps, 200.0 + 50.0 * i), err_msg=str(n))
    for a, b in zip(amr, alone):
        for lv in range(3):
            np.testing.assert_array_equal(a.get_populations(lv, layout="blocked"), b.get_populations(lv, layout="blocked"))
    for s in cubes + amr + alone:
        s.close()


def test_ensemble_of_more_cubes_than_one_pass_holds():
    # 48 cubes in the first launch, the 49th (the smallest) alone in the second
    sizes = [48] * 48 + [32]
    cubes = [cube(n, 300.0 + 100.0 * (i % 3)) for i, n in enumerate(sizes)]
    assert step_launches(cubes, 2) == 2
    want = {(n, re): one_at_a_time(n, 2, re) for n, re in {(n, 300.0 + 100.0 * (i % 3)) for i, n in enumerate(sizes)}}
    for i, (n, s) in enumerate(zip(sizes, cubes)):
        np.testing.assert_array_equal(s.get_populations(), want[n, 300.0 + 100.0 * (i % 3)], err_msg=str(i))
        s.close()


# ---- served solves ----------------------------------------------------------------------------------------

U0 = 0.05


def tstar(n, steps):
    return steps * U0 * 2 * math.pi / n


def serve(requests, **kw):
    sv = J.Server(**kw)
    for r in requests:
        assert sv.submit(**r) == 0
    out = {}
    while len(out) < len(requests):
        sv.tick()
        for r in sv.poll():
            out[r["id"]] = r
    sv.close()
    return out


def program_loop(r):
    """The `uniform` program's loop over one request, a step at a time."""
    kw = {k: v for k, v in r.items() if k not in ("rid", "kind", "diag_every")}
    with J.Solver("uniform", **kw) as s:
        steps, kf = s.info["steps"], s.info["kf"]
        e0, mass0, last, peak, peak_ts, drift, samples = None, None, None, -1.0, -1.0, 0.0, 0
        for step in range(steps + 1):
            if step % r["diag_every"] == 0:
                e, ens, mass = s.diag()
                e0 = e if e0 is None else e0
                mass0 = mass if mass0 is None else mass0
                drift = max(drift, abs(mass - mass0) / mass0)
                last = e
                samples += 1
                if ens > peak:
                    peak, peak_ts = ens, step * U0 * kf
            if step < steps:
                s.step(1)
    return dict(steps=steps, samples=samples, peak_enstrophy=peak, peak_tstar=peak_ts, energy_ratio=last / e0, mass_drift=drift)


def requests(cadences, steps, **kw):
    sizes = (32, 48, 64, 96, 128) * 2
    return [dict(rid=i, kind="uniform", n=n, re=200.0 + 50.0 * i, tstar=tstar(n, steps[i % len(steps)]),
                 diag_every=cadences[i % len(cadences)], **kw) for i, n in enumerate(sizes)]


# cadences that leave solves at odd and even distances from their next diagnostic, so that some take the pass while
# others step twice beside it, with diagnostics between the two; a tick that ends on an odd step
@pytest.mark.parametrize("tick_steps", [64, 17])
def test_served_solves_between_diagnostics_match_the_program_loop(tick_steps):
    reqs = requests((5, 8, 7, 1, 20), (41, 40, 33))
    reqs += [dict(rid=20, kind="uniform", n=48, re=500.0, storage="fp16", tstar=tstar(48, 37), diag_every=3),
             dict(rid=21, kind="uniform", n=16, re=300.0, storage="fp64", tstar=tstar(16, 30), diag_every=4),
             dict(rid=22, kind="uniform", n=32, re=300.0, flags=J.FLAG_INPLACE, tstar=tstar(32, 35), diag_every=6),
             dict(rid=23, kind="uniform", n=64, re=300.0, vec=2, tstar=tstar(64, 35), diag_every=9)]
    got = serve(reqs, tick_steps=tick_steps)
    for r in reqs:
        assert got[r["rid"]]["status"] == 0
        for k, v in program_loop(r).items():
            assert got[r["rid"]][k] == v, (r["rid"], k)


def test_served_solves_take_the_pass():
    # the same requests with a mapping chosen, whose every step is a launch of its own: 40 launches for all cubes
    # against 20 passes
    plain = requests((20,), (40,))
    mapped = requests((20,), (40,), threads_per_block=128)
    out = []
    n = [launches(lambda: out.append(serve(r))) for r in (plain, mapped)]
    assert n[1] - n[0] == 20
    for rid in out[0]:
        for k in ("samples", "peak_enstrophy", "energy_ratio", "mass_drift"):
            assert out[0][rid][k] == out[1][rid][k]
