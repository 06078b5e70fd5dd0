"""Populations across the C ABI in other types and orders than the state's (convert.cu), on a GB300.

Expected values are numpy's: shifted storages round f - w_q through float to the stored format and give back
w_q + stored; orders are index permutations.  Everything is exact, so there is no tolerance.
"""
import numpy as np
import pytest
import torch

import jpsolver as J

pytestmark = pytest.mark.gpu
Q = 19
W = np.array([np.float32(1.0) / np.float32(3.0)] + [np.float32(1.0) / np.float32(18.0)] * 6
             + [np.float32(1.0) / np.float32(36.0)] * 12, dtype=np.float32).astype(np.float64)


def stored(v, storage):
    """What the solver holds of v[q, ...], as 64-bit populations."""
    w = W.reshape(Q, 1, 1, 1)
    if storage == "fp64":
        return v.astype(np.float64)
    if storage == "fp32":
        return v.astype(np.float32).astype(np.float64)
    g = torch.from_numpy((v.astype(np.float64) - w).astype(np.float32))
    h = g.to(torch.float16 if storage == "fp16" else torch.bfloat16).to(torch.float64).numpy()
    return w + h


def blocked(f, mb):
    n = f.shape[1]
    g = n // mb
    return f.reshape(Q, g, mb, g, mb, g, mb).transpose(1, 3, 5, 0, 2, 4, 6).reshape(-1)


@pytest.mark.parametrize("inplace", [False, True])
@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16", "fp64"])
@pytest.mark.parametrize("n,mb", [(8, 8), (20, 4), (32, 16), (36, 4)])
def test_round_trips_in_every_type_and_order(n, mb, storage, inplace):
    rng = np.random.default_rng(n)
    v = (W.reshape(Q, 1, 1, 1) * (1.0 + 0.2 * rng.standard_normal((Q, n, n, n))))
    with J.Solver("uniform", n=n, mb=mb, storage=storage, flags=J.FLAG_INPLACE if inplace else 0) as s:
        for dt in (np.float32, np.float64):
            x = v.astype(dt)
            want = stored(x, storage).astype(np.float32).astype(np.float64) if storage == "fp32" else stored(x, storage)
            for layout in ("flat", "blocked"):
                s.set_populations(x if layout == "flat" else blocked(x, mb), layout=layout)
                for out in (np.float32, np.float64):
                    np.testing.assert_array_equal(s.get_populations(layout="flat", dtype=out), want.astype(out).reshape(-1))
                    np.testing.assert_array_equal(s.get_populations(layout="blocked", dtype=out), blocked(want.astype(out), mb))


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("steps", [1, 2])
def test_in_place_layouts_after_steps(storage, steps):
    n = 20
    out = []
    for flags in (0, J.FLAG_INPLACE):
        with J.Solver("uniform", n=n, mb=4, storage=storage, flags=flags) as s:
            s.step(steps)
            out.append((s.get_populations(layout="flat", dtype=np.float64), s.get_populations(layout="blocked")))
            s.set_populations(out[-1][0])                       # back into the layout of this step count
            np.testing.assert_array_equal(s.get_populations(dtype=np.float64), out[-1][0])
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][1], blocked(out[0][0].reshape(Q, n, n, n), 4).astype(np.float32))


@pytest.mark.parametrize("storage", ["fp16", "bf16"])
def test_amr_levels_round_trip(storage):
    with J.Solver("amr", n=16, l1_mode="all", l2_mode="all", storage=storage, max_gb=4.0) as s:
        s.step(1)
        for level in range(3):
            a = s.get_populations(level, "blocked", np.float64)
            b = s.get_populations(level, "blocked")
            np.testing.assert_array_equal(b, a.astype(np.float32))
            s.set_populations(a, level, "blocked")
            np.testing.assert_array_equal(s.get_populations(level, "blocked", np.float64), a)
