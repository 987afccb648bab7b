"""The fused loops' sums over the grid where they leave the range of the sum
before: a diverging solve, a residual that falls by many orders of magnitude in
one step, infinities and NaN.

What a loop reports as its error is r.r of the r it leaves.  A lane adds up the
squares of at most 64 rows of two cells in FP64, 128 * 2^-53 = 1.4e-14, and the
lanes' sums are added exactly and rounded once: 2e-14 is allowed against
math.fsum of the squares.
"""
import math
import re

import numpy as np
import pytest

from parity_util import random_deck

pytestmark = pytest.mark.gpu


def _scaled(text, factor):
    return re.sub(r"energy=(\S+)", lambda m: f"energy={float(m.group(1)) * factor!r}", text)


def _solve(tl, text, change=None, **kw):
    s = tl.Settings.from_text(text, mode=1, **kw)
    c = tl.initialiseapp(s)
    if change:
        change(c)
    tl.haloupdate(c, s, 1, ["energy", "density"])
    res = tl.SOLVERS[s.solver].solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2)
    f = {k: c.field(k)[2:-2, 2:-2] for k in ("u", "r")}
    c.close()
    return res, f


def _rr(f):
    with np.errstate(under="ignore"):
        return math.fsum((f["r"] ** 2).ravel())


@pytest.mark.parametrize("seed", [6, 11, 17])
def test_diverging_chebyshev(tl, built_lib, seed):
    """Five presteps leave the largest eigenvalue underestimated, and r.r grows by
    4e3 to 3e5 in ten steps: the fused loop runs to its budget as the exact one does.
    Both amplify the rounding of the same coefficients, by less than 1e-9."""
    text = _scaled(random_deck(256, seed, solver="cheby", presteps=5, eps=1e-15), 1e-3)
    text = text.replace("max_iters=5000", "max_iters=200")
    (a, f), (b, _) = _solve(tl, text), _solve(tl, text, exact=True)
    assert not b.converged and b.iters == 200 and b.error > 1e60
    assert not a.converged and a.iters == 200
    assert abs(a.error - b.error) <= 1e-9 * b.error
    assert not np.isnan(f["u"]).any()


@pytest.mark.parametrize("n,inner,factor", [(512, 200, 1.0), (256, 100, 1e-3), (61, 100, 1.0), (2700, 300, 1.0)])
def test_ppcg_long_outer_steps(tl, built_lib, n, inner, factor):
    """Hundreds of inner sweeps take r.r down by up to 1e-20 in an outer step; the
    iterations as test_gpu_persist.py's, within two of the exact loop's."""
    text = _scaled(random_deck(n, 6, solver="ppcg", presteps=30, ppcg_inner_steps=inner, eps=1e-15), factor)
    text = text.replace("max_iters=5000", "max_iters=1500")
    a, f = _solve(tl, text, criterion=1)
    assert a.error > 0 and abs(a.error - _rr(f)) <= 2e-14 * a.error
    if n < 1000:
        b, _ = _solve(tl, text, criterion=1, exact=True)
        assert a.converged == b.converged and abs(a.iters - b.iters) <= 2


@pytest.mark.parametrize("nx,ny", [(1, 5), (3, 1), (10, 10), (61, 33), (400, 300), (3100, 2500)])
@pytest.mark.parametrize("iters", [1, 2, 4, 8])
def test_cg_error_is_the_residual(tl, built_lib, nx, ny, iters):
    """On the smallest decks CG is through after a few steps and r.r falls by 1e-30
    in one; without a bound to meet it goes on from there as the exact loop does."""
    text = random_deck(nx, 6, ny=ny, eps=0.0).replace("max_iters=5000", f"max_iters={iters}")
    a, f = _solve(tl, text)
    assert a.iters == iters and a.error > 0 and abs(a.error - _rr(f)) <= 2e-14 * a.error
    if nx < 1000:
        b, g = _solve(tl, text, exact=True)
        assert np.max(np.abs(f["u"] - g["u"])) <= 1e-13 * np.max(np.abs(g["u"]))


@pytest.mark.parametrize("nx,ny", [(250, 250), (900, 700), (2700, 2600)])
@pytest.mark.parametrize("solver", ["jacobi", "cheby"])
def test_infinities_and_nan(tl, built_lib, nx, ny, solver):
    """Two cells of NaN and three of infinity, whose terms of the first sweep's sum
    are as many NaN as infinities: no such deck converges."""
    def change(c):
        e = c.field("energy0")
        for i, j in ((20, 20), (100, 120)):
            e[i, j] = np.nan
        for i, j in ((40, 60), (150, 30), (200, 200)):
            e[i, j] = np.inf
        c.set_field("energy", e)

    text = random_deck(nx, 6, ny=ny, solver=solver, presteps=5, eps=1e-15).replace("max_iters=5000", "max_iters=40")
    (a, _), (b, _) = _solve(tl, text, change), _solve(tl, text, change, exact=True)
    assert (a.iters, a.converged, b.converged) == (b.iters, False, False)
    assert math.isnan(a.error) == math.isnan(b.error)


@pytest.mark.parametrize("solver,nx,ny,k", [("cg", 256, 256, 51), ("cheby", 256, 256, 51), ("ppcg", 256, 256, 51),
                                            ("cg", 1021, 769, 45), ("ppcg", 1021, 769, 45), ("cg", 2700, 2600, 40)])
def test_fp32_sums_beyond_fp32(tl, built_lib, solver, nx, ny, k):
    """Energies times 2^k, where r.r of the grid is above 3.4e38 and 16 products still
    are not: every number of the solve is the unscaled one times a power of two, so the
    steps are the same and u the same bits times 2^k."""
    text = random_deck(nx, 6, ny=ny, solver=solver, presteps=40, eps=1e-10, errorswitch=1, epslim=1e250)
    a, f = _solve(tl, text, precision=1, criterion=1)
    b, g = _solve(tl, _scaled(text, 2.0 ** k), precision=1, criterion=1)
    assert a.converged and b.converged and (a.iters, a.refinements) == (b.iters, b.refinements)
    np.testing.assert_array_equal(g["u"], f["u"] * 2.0 ** k)


@pytest.mark.parametrize("eps", [math.nan, -1.0, -0.0])
@pytest.mark.parametrize("solver,criterion", [("cg", 0), ("cg", 1), ("cheby", 0), ("ppcg", 0), ("jacobi", 0)])
def test_bounds_that_nothing_meets(tl, built_lib, solver, criterion, eps):
    """No error is below NaN, a negative number or zero: the fused loops run to their
    budget as the exact ones do."""
    text = random_deck(61, 6, ny=47, solver=solver, presteps=10, errorswitch=1, epslim=1e9)
    text = text.replace("max_iters=5000", "max_iters=40")
    got = []
    for exact in (False, True):
        s = tl.Settings.from_text(text, mode=1, criterion=criterion, exact=exact)
        s.eps = eps
        c = tl.initialiseapp(s)
        tl.haloupdate(c, s, 1, ["energy", "density"])
        r = tl.SOLVERS[s.solver].solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2)
        got.append((r.converged, r.iters))
        c.close()
    assert got[0] == got[1] == (False, 40)
