"""ggx_b (kpt_shade.cuh): the GGX denominator ndh * (a2 - 1) + 1 from float
operations with their exact errors, against the double-precision expression
rounded to float and against the exact value."""

import numpy as np
import pytest

F = np.float32


def _float_form(x, a2):
    h = F(1) - x
    hl = (F(1) - h) - x
    p = x * a2
    pl = F(x.astype(np.float64) * a2.astype(np.float64) - p.astype(np.float64))   # the fused operation's result
    s = h + p
    q = s - h
    sl = (h - (s - q)) + (p - q)
    return s + (sl + (pl + hl))


def _draws(which, n=1_000_000):
    rng = np.random.default_rng(3)
    one = np.ones(n)
    cos = {"uniform": rng.random(n), "peak": 1.0 - 10.0 ** rng.uniform(-7.0, -0.1, n), "one": one, "zero": 0.0 * one,
           "smooth": 1.0 - 10.0 ** rng.uniform(-8.0, -3.0, n), "rough": rng.random(n)}[which].astype(F)
    alpha = {"smooth": np.full(n, 1e-3), "rough": rng.uniform(1.0, 4.0, n)}.get(which, rng.uniform(0.0, 1.0, n) ** 2)
    alpha = np.maximum(alpha, 1e-3).astype(F)
    return cos * cos, alpha * alpha


@pytest.mark.parametrize("which", ["uniform", "peak", "one", "zero", "smooth", "rough"])
def test_ggx_b(which):
    x, a2 = _draws(which)
    got = _float_form(x, a2)
    t = a2.astype(np.float64) - 1.0
    ref = (x.astype(np.longdouble) * t + 1).astype(np.float64).astype(F)   # rounded to double, then to float
    assert np.mean(got != ref) <= 1e-5
    exact = x.astype(np.longdouble) * (a2.astype(np.longdouble) - 1) + 1
    assert (np.abs(got - exact) <= np.spacing(got) * np.longdouble(0.5000001)).all()
