"""PPCG with more inner steps than the context has iterations: the coefficients are
those of a context with room for them from the start, so the solves are the same
bits.  Fewer inner steps afterwards use the same tables."""
import numpy as np
import pytest

from parity_util import random_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(exact=True), dict(criterion=1, precision=1)], ids=["fp64", "exact", "fp32"])
@pytest.mark.parametrize("inner", [41, 42, 100])
def test_more_inner_steps_than_iterations(tl, built_lib, kw, inner):
    text = random_deck(100, 6, ny=81, solver="ppcg", presteps=10, errorswitch=1, epslim=1e9, eps=1e-12,
                       ppcg_inner_steps=inner)
    got = []
    for room in (40, 400):
        s = tl.Settings.from_text(text.replace("max_iters=5000", f"max_iters={room}"), mode=1, **kw)
        c = tl.initialiseapp(s)
        s.maxiters = 40
        for steps in (inner, 10):
            s.ppcginnersteps = steps
            tl.haloupdate(c, s, 1, ["energy", "density"])
            r = tl.SOLVERS[s.solver].solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2)
            assert r.inner_iters > 0
            got.append((r.iters, r.error, c.field("u")[2:-2, 2:-2]))
            tl.solvefinished(c, s)
        c.close()
    for a, b in zip(got[:2], got[2:]):
        assert a[:2] == b[:2]
        assert np.isfinite(a[2]).all()
        np.testing.assert_array_equal(a[2], b[2])
