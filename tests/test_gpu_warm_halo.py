"""The warm start changes the iterate it starts from, u's interior and the layer
about it; u's corners and further halo layers stay the plain start's, energy times
density, whatever the candidate's buffer held there."""
import numpy as np
import pytest

from parity_util import random_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [1, 2, 3])
@pytest.mark.parametrize("mode", ["NETWORK", "HISTORY", "EXTRAPOLATE"])
def test_outer_halo_of_u(tl, built_lib, hd, mode):
    nx, ny = 67, 45
    s = tl.Settings.from_text(random_deck(nx, 91, ny=ny, eps=1e-10, halo_depth=hd), mode=1, criterion=1,
                              warmstart=getattr(tl._abi, "WARM_" + mode))
    c = tl.initialiseapp(s)
    if mode == "NETWORK":
        c.warm_load(tl.warmstart.load_params())
    rx, ry = s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2
    for _ in range(3):
        tl.haloupdate(c, s, 1, ["energy", "density"])
        tl.CG.solve(c, s, rx, ry)
        tl.solvefinished(c, s)
    s.eps = 1e10  # the start already meets it
    tl.haloupdate(c, s, 1, ["energy", "density"])
    res = tl.CG.solve(c, s, rx, ry)
    u, start = c.field("u"), c.field("energy") * c.field("density")
    c.close()
    assert res.iters == 0 and res.warm in (1, 3), res  # a prediction was taken
    inner = np.zeros(u.shape, bool)
    inner[hd - 1:nx + hd + 1, hd:-hd] = inner[hd:-hd, hd - 1:ny + hd + 1] = True
    np.testing.assert_array_equal(u[~inner], start[~inner])
    assert not np.array_equal(u[inner], start[inner])
