"""Two-step passes of the uniform cube (uniform_pair.cu) against single steps, on a GB300.

step(k) takes two steps in one pass where that is planned to be faster, step(1) never does; both relax with
the same arithmetic and round every step to the storage format, so k steps either way are the same bits.
The edges cover cubes of one tile, ragged tiles along x and y, chunks with a remainder and several rounds
of items per CTA.
"""
import numpy as np
import pytest

import jpsolver as J

pytestmark = pytest.mark.gpu


def solver(n, storage="fp32", re=400.0):
    return J.Solver("uniform", n=n, storage=storage, re=re, mb=8 if n % 8 == 0 else 4)


def single_steps(n, storage, steps, re=400.0):
    with solver(n, storage, re) as s:
        for _ in range(steps):
            s.step(1)
        return s.get_populations()


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("n,steps", [(16, 4), (20, 5), (24, 2), (32, 7), (36, 4), (48, 2), (64, 3), (68, 4), (100, 4), (128, 2)])
def test_two_step_pass_bit_exact_with_single_steps(n, steps, storage):
    with solver(n, storage) as s:
        s.step(steps)
        assert s.info["step_count"] == steps
        a = s.get_populations()
    np.testing.assert_array_equal(a, single_steps(n, storage, steps))


def test_two_step_pass_of_a_large_cube_bit_exact():
    with solver(200) as s:
        s.step(2)
        a = s.get_populations()
    np.testing.assert_array_equal(a, single_steps(200, "fp32", 2))


@pytest.mark.parametrize("steps", [2, 5])
def test_ensemble_two_step_passes_bit_exact(steps):
    shapes = [(32, "fp32"), (96, "fp32"), (128, "fp32"), (20, "fp32"), (64, "fp16"), (48, "fp16"), (100, "fp32"), (68, "bf16")]
    solvers = [solver(n, st, 200.0 + 100.0 * i) for i, (n, st) in enumerate(shapes)]
    e = J.Ensemble()
    for s in solvers:
        e.add(s)
    e.step(steps)
    for i, ((n, st), s) in enumerate(zip(shapes, solvers)):
        np.testing.assert_array_equal(s.get_populations(), single_steps(n, st, steps, 200.0 + 100.0 * i), err_msg="%d %s" % (n, st))
    e.close()
    for s in solvers:
        s.close()
