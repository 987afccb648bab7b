"""The persistent iteration kernels at the sizes where their tiling can go
wrong: the edges of a warp's strip, one block against many, one tile a warp
against tiles handed out as warps come free.

FP32-refined CG is compared with exact FP64 CG, which is bit-identical to the
CPU oracle: both meet the 1e-10 relative true residual, and A >= I, so each
solution is within 1e-10 ||u0|| of the true one in the 2-norm and the two
within 2e-10 ||u0|| of each other (4e-10 allows for the second step's right-hand
sides, which differ by as much).
"""
import numpy as np
import pytest

from parity_util import gpu_run, random_deck

pytestmark = pytest.mark.gpu
TEA = 1


def _interior(a, hd=2):
    return a[hd:-hd, hd:-hd]


@pytest.mark.parametrize("nx,ny", [
    (119, 3), (120, 32), (121, 33), (124, 1), (1, 300), (240, 16), (361, 47),  # strip edges; one block up to 32 strip rows
    (512, 512), (1021, 769),            # one tile a warp
    (2203, 1301), (4099, 1801),         # tiles handed out
])
def test_fp32_cg_tilings(tl, built_lib, nx, ny):
    text = random_deck(nx, 81, ny=ny, nrect=4, steps=2, eps=1e-10)
    runs = {}
    for name, kw in (("ir", dict(precision=1)), ("again", dict(precision=1)), ("exact", dict(exact=True))):
        c, res, _, _ = gpu_run(tl, text, TEA, criterion=1, **kw)
        runs[name] = (_interior(c.field("u")), res)
        u0 = _interior(c.field("u0"))
        c.close()
    u, res = runs["ir"]
    v, ref = runs["exact"]
    for a, b in zip(res, ref):
        assert a.converged and 0 <= a.rel_residual < 1e-10 and b.converged
        assert a.iters <= 1.5 * b.iters + 20, (a.iters, b.iters)  # the bound of test_gpu_ir.py: refinement restarts cost some
    assert np.linalg.norm(u - v) <= 4e-10 * np.linalg.norm(u0)
    # whatever warp took which tile, the sums and the solution are the same bits
    np.testing.assert_array_equal(u, runs["again"][0])
    assert [r.iters for r in res] == [r.iters for r in runs["again"][1]]
