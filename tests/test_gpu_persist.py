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


@pytest.mark.parametrize("nx,ny,hd", [
    (1, 7, 2), (59, 5, 1), (60, 4, 3), (61, 9, 2), (62, 3, 1), (119, 40, 2), (121, 33, 2), (3, 400, 2),  # strip edges, one block
    (513, 511, 2), (1023, 401, 1),      # one tile a warp
    (1801, 1403, 2),                    # tiles handed out
])
def test_fp64_cg_tilings(tl, built_lib, nx, ny, hd):
    """Fused FP64 CG against exact FP64 CG: the same bound on u, iteration
    counts within one (the arithmetic differs in rounding alone), and p, w of
    the last step where both took the same steps: p within 1e-6 of its norm
    (CG's vectors drift apart by rounding, by some 1e-9 here)."""
    text = random_deck(nx, 82, ny=ny, nrect=4, steps=2, eps=1e-10, halo_depth=hd)
    runs = {}
    for name, kw in (("fused", {}), ("again", {}), ("exact", dict(exact=True))):
        c, res, _, _ = gpu_run(tl, text, TEA, criterion=1, **kw)
        runs[name] = ({f: _interior(c.field(f), hd) for f in ("u", "u0", "p")}, res)
        c.close()
    (f, res), (g, ref) = runs["fused"], runs["exact"]
    for a, b in zip(res, ref):
        assert a.converged and 0 <= a.rel_residual < 1e-10 and b.converged
        assert abs(a.iters - b.iters) <= 1, (a.iters, b.iters)
    assert np.linalg.norm(f["u"] - g["u"]) <= 4e-10 * np.linalg.norm(g["u0"])
    if [r.iters for r in res] == [r.iters for r in ref] and min(nx, ny) > 30:
        assert np.linalg.norm(f["p"] - g["p"]) <= 1e-6 * np.linalg.norm(g["p"])
    for k in f:
        np.testing.assert_array_equal(f[k], runs["again"][0][k], err_msg=k)
