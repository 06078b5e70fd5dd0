"""Rules that pick a kernel or a launch form, against the general path, on a GB300.

AMR diagnostics by leaf blocks (amr_diag.cu) against the oracle; coarse steps replayed after a few launches
and coarse steps of a grid without level-2 blocks against a solver that replays from the start; single steps of
small cubes, whose rule takes vectors of two cells, against vectors of four; the mass that the relaxation's
coefficients leave.
"""
import numpy as np
import pytest

import jpsolver as J
import oracle as O

pytestmark = pytest.mark.gpu


# The edges of the leaf walk: a slab (neighbours on other levels and across the period), level 1 without level 2,
# every block edge; grids that both sides build alike without comparing sensors (l2 "slab" marks by the sensor,
# which ties on the initial flow, so it stands where no block is deep enough to be marked).
@pytest.mark.parametrize("n,mb,l1,l2", [(16, 8, "slab", "slab"), (16, 4, "slab", "all"), (32, 16, "slab", "slab"),
                                        (48, 16, "slab", "all"), (24, 8, "slab", "sensor"), (20, 4, "slab", "all"),
                                        (32, 8, "slab", "all"), (16, 8, "all", "all")])
def test_leaf_diagnostics_match_oracle(n, mb, l1, l2):
    # both sum the same FP64 terms in another order: a relative 1e-10 leaves 5 digits over the sums' 1e-15 * log2(cells)
    with J.Solver("amr", n=n, re=800.0, l1_mode=l1, l2_mode=l2, frac1=0.35, frac2=0.35, develop_steps=3, max_gb=64.0,
                  mb=mb) as e:
        o = O.AmrBackend("oracle", n, 800.0, l1, l2, 0.35, 0.35, develop=3, budget=64.0 * 2 ** 30, mb=mb)
        assert (e.counts()["nf1"], e.counts()["nf2"]) == (o.counts()["nf1"], o.counts()["nf2"])
        for t in ("fof0", "fof1", "f1pos", "l2pl1", "l2oct"):
            np.testing.assert_array_equal(e.table(t), o.table(t), err_msg=t)
        rng = np.random.default_rng(n + mb)
        for lv in range(3):
            if e.counts()[("cnb0", "nf1", "nf2")[lv]] == 0:
                continue
            p = e.get_populations(lv, layout="blocked")
            p = (p * (1 + 0.01 * rng.random(p.shape, dtype=np.float32))).astype(np.float32)
            e.set_populations(p, level=lv, layout="blocked")
            o.set_pops(lv, p)
        for x, y in zip(e.diag(), o.diag()):
            assert abs(x - y) <= 1e-10 * abs(y)
        o.close()


@pytest.mark.parametrize("n,storage,l2", [(16, "fp32", "sensor"), (24, "fp32", "sensor"), (24, "fp16", "sensor"),
                                          (16, "fp32", "slab")])
def test_replayed_steps_bit_exact_with_graph_solver(n, storage, l2):
    kw = dict(n=n, re=800.0, l1_mode="slab" if l2 == "slab" else "sensor", l2_mode=l2, storage=storage, develop_steps=20,
              max_gb=64.0)
    with J.Solver("amr", **kw) as a, J.Solver("amr", flags=J.FLAG_GRAPH, **kw) as b:
        for k in (1, 2, 1, 5, 20):  # across the count that captures, and a regrid after each
            for s in (a, b):
                s.step(k)
            assert a.counts() == b.counts()
            for lv in range(3):
                if a.counts()[("cnb0", "nf1", "nf2")[lv]] == 0:
                    continue
                np.testing.assert_array_equal(a.get_populations(lv, layout="blocked"),
                                              b.get_populations(lv, layout="blocked"), err_msg="%d steps, level %d" % (k, lv))
            for s in (a, b):
                s.regrid()


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("n", [8, 16, 24, 40, 48, 64, 80])
def test_small_cubes_bit_exact_with_vectors_of_four(n, storage):
    kw = dict(n=n, storage=storage, re=300.0, mb=8 if n % 8 == 0 else 4)
    with J.Solver("uniform", **kw) as a, J.Solver("uniform", vec=4, **kw) as b:
        for _ in range(3):
            a.step(1)
            b.step(1)
        np.testing.assert_array_equal(a.get_populations(), b.get_populations())


@pytest.mark.parametrize("n,re,steps", [(64, 400.0, 2000), (96, 300.0, 1000), (32, 100.0, 2000)])
def test_relaxation_coefficients_keep_mass(n, re, steps):
    # what rounding leaves of the coefficients' balance is within 1.5e-8, times the mean u.u (6e-4 at most), in every
    # step: 1e-11; the stored populations' rounding adds some 1e-10 of either sign per step, sqrt(steps) of it in all
    with J.Solver("uniform", n=n, re=re) as s:
        m0 = s.diag()[2]
        s.step(steps)
        assert abs(s.diag()[2] / m0 - 1) < 1e-11 * steps + 5e-10 * steps ** 0.5
