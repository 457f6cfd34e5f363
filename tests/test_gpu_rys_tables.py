"""The Rys roots and weights on the device: polynomials on unit intervals of T
(FP64 tables of one and two roots: quarter intervals) below 30.5 + 5 N, the
Gauss-Laguerre limit above.  A quartet (aa|bb) of two single-primitive shells
of exponent 1/2 has zeta 1 on both sides and T equal to half the squared
distance, so the distance sets T: at interval edges, inside the first and last
intervals, on both sides of the crossover and beyond.

s shells (N = 1) are held to the closed form within the fits' 2e-14 of a
weight (the reference's bound for its tables) and rounding; p, d and f
(N = 3, 5, 7) to the oracle at its engines' agreement on such blocks (1e-11 + 1e-10 |x|,
tests/cross_engine.rs:40-56)."""
import math

import numpy as np
import pytest

import integral_b200 as ib
import oracle_py as O

pytestmark = pytest.mark.gpu


def distances(n):
    hi = 30.5 + 5 * n
    ts = [0.0, 1e-9, 0.5, 1.0 - 1e-12, 1.0, 17.0, 17.25, math.floor(hi), hi - 1e-9, hi, hi + 1e-9, 3.0 * hi]
    return [math.sqrt(2.0 * t) for t in ts]


def shells(l, r):
    return [dict(l=l, spherical=False, center=[0.0, 0.0, 0.0], exps=[0.5], coefs=[1.0]),
            dict(l=l, spherical=False, center=[0.0, 0.0, r], exps=[0.5], coefs=[1.0])]


def test_ss_closed_form():
    for r in distances(1):
        t = 0.5 * r * r
        f0 = 1.0 - t / 3 if t < 1e-8 else 0.5 * math.sqrt(math.pi / t) * math.erf(math.sqrt(t))
        norm = (1.0 / math.pi) ** 0.75  # (2 alpha / pi)^(3/4)
        pref = norm ** 4 * 2 * math.pi ** 2.5 / math.sqrt(2.0)
        got = float(ib.Basis(shells(0, r)).eri_block(0, 0, 1, 1)[0])
        assert abs(got - pref * f0) < pref * (2e-14 + 2e-15 * f0), (t, got, pref * f0)


@pytest.mark.parametrize("l", [1, 2, 3])
def test_blocks_across_the_intervals(l):
    for r in distances(2 * l + 1):
        s = shells(l, r)
        got = ib.Basis(s).eri_block(0, 0, 1, 1)
        want = np.asarray(O.OracleBasis(s).eri_block(0, 0, 1, 1)).reshape(-1)
        assert np.all(np.abs(got - want) <= 1e-11 + 1e-10 * np.abs(want)), (r, float(np.max(np.abs(got - want))))
