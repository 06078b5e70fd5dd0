"""Where the two-step pass is taken, and its bits there, on a GB300.

The launches are counted, so that a case that is meant to take the pass cannot be one that compares single steps
with themselves.  Every FP32 result is compared with steps taken one at a time (`step(1)` never takes the pass).
"""
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


# the mapping tests of the single step, a step at a time whatever the plan
@pytest.mark.parametrize("vec,tpb", [(1, 256), (2, 128), (4, 64), (4, 128), (4, 256), (4, 512)])
def test_chosen_mappings_are_used_by_every_step(vec, tpb):
    with cube(32, vec=vec, threads_per_block=tpb) as s:
        assert launches(lambda: s.step(3)) == 3
        np.testing.assert_array_equal(s.get_populations(), one_at_a_time(32, 3))
