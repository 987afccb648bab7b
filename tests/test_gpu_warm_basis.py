"""The warm start's candidates for every size of the basis, with and without the
network's term: a solve whose bound the start already meets leaves the start it
chose in u, r and p.  r must be u0 - A u (a few roundings of sums of four
products of kx u, so 1e-14 of the largest term; 1e-13 allowed), p equal to it,
u's halo its reflection, and the reported residual its norm.
"""
import numpy as np
import pytest

from parity_util import random_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(97, 61), (33, 130)])
@pytest.mark.parametrize("earlier", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("mode", ["NETWORK", "HISTORY"])
def test_candidate_is_the_start(tl, built_lib, nx, ny, earlier, mode):
    s = tl.Settings.from_text(random_deck(nx, 91, ny=ny, eps=1e-10), mode=1, criterion=1,
                              warmstart=getattr(tl._abi, "WARM_" + mode))
    c = tl.initialiseapp(s)
    c.warm_load(tl.warmstart.load_params())
    rx, ry, hd = s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2, s.halodepth
    for _ in range(earlier):
        tl.haloupdate(c, s, 1, ["energy", "density"])
        tl.CG.solve(c, s, rx, ry)
        tl.solvefinished(c, s)
    s.eps = 1e10
    tl.haloupdate(c, s, 1, ["energy", "density"])
    res = tl.CG.solve(c, s, rx, ry)
    full = {f: c.field(f) for f in ("u", "u0", "r", "p", "kx", "ky")}
    c.close()
    u, u0, r, p = (full[f][hd:-hd, hd:-hd] for f in ("u", "u0", "r", "p"))
    assert res.iters == 0 and res.warm in ((1, 2, 3) if mode == "NETWORK" else (1, 2))
    kx, ky = full["kx"], full["ky"]
    e, w = kx[hd + 1:kx.shape[0] - hd + 1, hd:-hd], kx[hd:-hd, hd:-hd]
    n, so = ky[hd:-hd, hd + 1:ky.shape[1] - hd + 1], ky[hd:-hd, hd:-hd]
    q = np.pad(u, 1, mode="edge")
    Au = u + e * (u - q[2:, 1:-1]) + w * (u - q[:-2, 1:-1]) + n * (u - q[1:-1, 2:]) + so * (u - q[1:-1, :-2])
    size = np.max(np.abs(u) * (1 + e + w + n + so))
    assert np.max(np.abs(r - (u0 - Au))) <= 1e-13 * size
    np.testing.assert_array_equal(p, r)
    np.testing.assert_array_equal(full["u"][hd - 1:-hd + 1, hd:-hd], q[:, 1:-1])
    np.testing.assert_array_equal(full["u"][hd:-hd, hd - 1:-hd + 1], q[1:-1])
    rel = np.linalg.norm(r) / np.linalg.norm(u0)
    if res.warm == 2:
        assert np.array_equal(u, u0) and res.r0_pred >= res.r0_plain
    else:
        assert abs(res.r0_pred - rel) <= 1e-9 * rel + 1e-14 and res.r0_pred < res.r0_plain
