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


@pytest.mark.parametrize("nx,ny,hd", [(1, 9, 2), (59, 7, 1), (61, 33, 3), (120, 40, 2), (243, 131, 2), (3100, 2500, 2)])
def test_jacobi_tilings(tl, built_lib, nx, ny, hd):
    """Fused Jacobi against exact Jacobi over 53 sweeps (one residual check
    among them): each sweep is a weighted mean of neighbours and the
    right-hand side, so the two drift by a few roundings a sweep: u within
    1e-13 of its maximum, r (the last sweep's input) alike, and its faces."""
    text = random_deck(nx, 83, ny=ny, nrect=4, steps=1, eps=0.0, solver="jacobi", halo_depth=hd)
    text = text.replace("max_iters=5000", "max_iters=53")
    f = {}
    for name, exact in (("fused", False), ("exact", True)):
        st = tl.Settings.from_text(text, mode=TEA, exact=exact)
        c = tl.initialiseapp(st)
        tl.haloupdate(c, st, 1, ["energy", "density"])
        res = tl.Jacobi.solve(c, st, st.dtinit / st.dx ** 2, st.dtinit / st.dy ** 2)  # solvefinished! overwrites r
        f[name] = (c.field("u"), c.field("r"), res)
        c.close()
    (u, r, a), (v, s, b) = f["fused"], f["exact"]
    assert a.iters == b.iters == 53
    assert abs(a.error - b.error) <= 1e-9 * abs(b.error) + 1e-13 * np.max(np.abs(v)) * nx * ny
    scale = np.max(np.abs(v))
    assert np.max(np.abs(u - v)) <= 1e-13 * scale
    # the halo layers past the first hold what the solve before it left: faces and interior are compared
    k = hd - 1
    cut = lambda x: x[k:x.shape[0] - k, k:x.shape[1] - k]
    rf, sf = cut(r)[:, 1:-1], cut(s)[:, 1:-1]
    assert np.max(np.abs(rf - sf)) <= 1e-13 * scale
    assert np.max(np.abs(cut(r)[1:-1] - cut(s)[1:-1])) <= 1e-13 * scale


@pytest.mark.parametrize("solver", ["cheby", "ppcg"])
@pytest.mark.parametrize("nx,ny,hd", [(61, 120, 1), (119, 64, 3), (181, 240, 2), (513, 300, 2)])
def test_cheby_ppcg_tilings(tl, built_lib, solver, nx, ny, hd):
    """Fused Chebyshev and PPCG against their exact form, 40 presteps: the
    tolerances of test_gpu_solvers.py (iterations within 2, u within 1e-9 of
    its maximum)."""
    text = random_deck(nx, 84, ny=ny, nrect=5, steps=2, eps=1e-12, solver=solver, halo_depth=hd, presteps=40,
                       ppcg_inner_steps=5)
    f = {}
    for name, exact in (("fused", False), ("again", False), ("exact", True)):
        c, res, _, _ = gpu_run(tl, text, TEA, exact=exact)
        f[name] = (_interior(c.field("u"), hd), res)
        c.close()
    (u, res), (v, ref) = f["fused"], f["exact"]
    for a, b in zip(res, ref):
        assert abs(a.iters - b.iters) <= 2, (a.iters, b.iters)
    assert np.max(np.abs(u - v)) <= 1e-9 * np.max(np.abs(v))
    np.testing.assert_array_equal(u, f["again"][0])


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_groups(tl, built_lib, precision):
    """More decks than a batch has groups of blocks, from three cells to some
    hundred thousand (one block of a group against all of it): each deck
    converged and, as two solutions of a system A >= I that both meet 1e-10,
    within 2e-10 ||u0|| of its own single-deck solve."""
    sizes = [(700, 611), (3, 1), (121, 33), (512, 256), (64, 64), (31, 200), (901, 40), (240, 240), (5, 5), (333, 222),
             (120, 120), (60, 61), (450, 300), (17, 19), (256, 129), (128, 500), (77, 78), (19, 350), (404, 404), (90, 30)]
    texts = [random_deck(nx, 500 + k, ny=ny, nrect=3, steps=1, eps=1e-10) for k, (nx, ny) in enumerate(sizes)]
    kw = dict(mode=TEA, criterion=1, precision=precision)
    sets = [tl.Settings.from_text(t, **kw) for t in texts]
    chunks = [tl.initialiseapp(s) for s in sets]
    hist = tl.diffuse_batch(chunks, sets, steps=1)
    for k, t in enumerate(texts):
        s = tl.Settings.from_text(t, **kw)
        c = tl.initialiseapp(s)
        tl.haloupdate(c, s, 1, ["energy", "density"])
        one = tl.CG.solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2)
        b = hist[0][k]
        assert b.converged and 0 <= b.rel_residual < 1e-10, (sizes[k], b)
        assert abs(b.iters - one.iters) <= max(1, 0.05 * one.iters), (sizes[k], b.iters, one.iters)
        d = _interior(chunks[k].field("u")) - _interior(c.field("u"))
        assert np.linalg.norm(d) <= 2e-10 * np.linalg.norm(_interior(c.field("u0"))), sizes[k]
        c.close()
        chunks[k].close()


@pytest.mark.parametrize("solver,inner", [("cheby", 10), ("ppcg", 1), ("ppcg", 4), ("ppcg", 5)])
@pytest.mark.parametrize("nx,ny,hd", [(61, 120, 1), (119, 64, 3), (121, 200, 2), (513, 300, 2), (1201, 1000, 2)])
def test_fp32_sweep_tilings(tl, built_lib, solver, inner, nx, ny, hd):
    """FP32 Chebyshev and PPCG (an odd and an even number of sweeps after the
    first, or none) at the edges of strips and bands: every step meets 1e-10 on
    the true residual, so u is within 2e-10 ||u0|| of exact FP64 CG's (4e-10 at
    the second step, see above), and two runs are the same bits."""
    text = random_deck(nx, 84, ny=ny, nrect=5, steps=2, eps=1e-10, solver=solver, halo_depth=hd, presteps=40,
                       ppcg_inner_steps=inner)
    c, _, _, _ = gpu_run(tl, text.replace(f"use_{solver}", "use_cg"), TEA, exact=True, criterion=1)
    v, u0 = _interior(c.field("u"), hd), _interior(c.field("u0"), hd)
    c.close()
    u = []
    for _ in range(2):
        c, res, _, _ = gpu_run(tl, text, TEA, criterion=1, precision=1)
        assert all(r.converged and 0 <= r.rel_residual < 1e-10 for r in res), res
        u.append(_interior(c.field("u"), hd))
        c.close()
    assert np.linalg.norm(u[0] - v) <= 4e-10 * np.linalg.norm(u0)
    np.testing.assert_array_equal(u[0], u[1])


@pytest.mark.parametrize("hd", [1, 2, 3])
@pytest.mark.parametrize("coefficient", [1, 2])
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 3), (26, 5), (28, 1), (29, 31), (61, 64), (90, 7), (700, 611)])
def test_start_and_end_of_a_solve(tl, built_lib, nx, ny, hd, coefficient):
    """The one-kernel start and end of a step against the separate kernels of the
    exact path, halo included: the same operations per cell, so equal bit for
    bit.  A bound on the residual that the start already meets ends the solve
    there."""
    text = random_deck(nx, 7, ny=ny, nrect=3, eps=1e10).replace("halo_depth=2", f"halo_depth={hd}")
    text = text.replace("coefficient=1", f"coefficient={coefficient}")
    chunks, results = [], []
    for exact in (False, True):
        s = tl.Settings.from_text(text, mode=TEA, exact=exact, criterion=1)
        c = tl.initialiseapp(s)
        tl.haloupdate(c, s, 1, ["energy", "density"])
        results.append(tl.CG.solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2))
        chunks.append((c, s))
    (a, sa), (b, sb) = chunks
    assert results[0].iters == results[1].iters == 0 and results[0].converged
    assert abs(results[0].error - results[1].error) <= 1e-12 * results[1].error
    for f in ("u", "u0", "p", "r", "w", "kx", "ky"):
        np.testing.assert_array_equal(a.field(f), b.field(f), err_msg=f)
    tl.solvefinished(a, sa)
    tl.residual(b)
    tl.finalise(b)
    tl.haloupdate(b, sb, 1, ["energy"])
    for f in ("r", "energy"):
        np.testing.assert_array_equal(a.field(f), b.field(f), err_msg=f)
    a.close()
    b.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 2), (61, 33), (62, 1), (243, 131), (600, 449),  # the blocks hold the deck
                                   (600, 481), (901, 700)])
@pytest.mark.parametrize("iters,eps", [(1, 0.0), (2, 0.0), (3, 0.0), (50, 0.0), (51, 0.0), (52, 0.0),
                                       (400, 3.0), (400, 2.0), (400, 1.4)])
def test_jacobi_pairs(tl, built_lib, nx, ny, iters, eps):
    """Fused Jacobi, two sweeps a pass, against the exact sweeps where it can end:
    after the first or the second of a pair, at a check, by its bound or its
    budget.  The bounds are in units of the 7th sweep's change.  Tolerances as
    in test_jacobi_tilings."""
    text = random_deck(nx, 84, ny=ny, nrect=4, steps=1, eps=0.0, solver="jacobi")
    if eps:
        changes = []
        for k in (1, 7):
            s = tl.Settings.from_text(text.replace("max_iters=5000", f"max_iters={k}"), mode=TEA, exact=True)
            c = tl.initialiseapp(s)
            tl.haloupdate(c, s, 1, ["energy", "density"])
            changes.append(tl.Jacobi.solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2).error)
            c.close()
        eps *= max(changes[1], 1e-8 * changes[0])  # not a bound within rounding, on decks that are done by then
    text = text.replace("max_iters=5000", f"max_iters={iters}").replace("eps=0.0", f"eps={eps!r}")
    f = []
    for exact in (False, True):
        s = tl.Settings.from_text(text, mode=TEA, exact=exact)
        c = tl.initialiseapp(s)
        tl.haloupdate(c, s, 1, ["energy", "density"])
        res = tl.Jacobi.solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2)
        f.append((_interior(c.field("u"), 1), _interior(c.field("r"), 1), res))
        k = 1 + 2 * (np.max(np.abs(_interior(c.field("kx")))) + np.max(np.abs(_interior(c.field("ky")))))
        c.close()
    (u, r, a), (v, s, b) = f
    assert (a.iters, a.converged) == (b.iters, b.converged)
    scale = np.max(np.abs(v))
    assert np.max(np.abs(u - v)) <= 1e-13 * scale
    # after a check r is u0 - A u, which multiplies what u is off by up to 1 + sum k
    at_check = b.iters % 50 == 0
    assert np.max(np.abs(r - s)) <= 1e-13 * scale * (k if at_check else 1)
    assert abs(a.error - b.error) <= 1e-9 * abs(b.error) + 1e-13 * scale * nx * ny


@pytest.mark.parametrize("nx,ny", [(1, 1), (60, 16), (60, 17), (61, 8), (61, 9), (300, 480), (300, 487), (540, 271)])
@pytest.mark.parametrize("iters", [1, 2, 7])
def test_fp64_cg_one_row_a_warp(tl, built_lib, nx, ny, iters):
    """FP64 CG where a warp has one row (r and w stay with it between the passes)
    and on either side of that line, stopped early: u, p, r and w of the last
    step against the exact loop's.  Their roundings, some 1e-16 of a vector a step
    before the residual's own fall (by less than 1e3 in seven steps of these
    decks) scales them up, stay below 1e-9 of its norm."""
    text = random_deck(nx, 85, ny=ny, nrect=4, steps=1, eps=1e-300).replace("max_iters=5000", f"max_iters={iters}")
    f = []
    for exact in (False, True):
        s = tl.Settings.from_text(text, mode=TEA, exact=exact)
        c = tl.initialiseapp(s)
        tl.haloupdate(c, s, 1, ["energy", "density"])
        res = tl.CG.solve(c, s, s.dtinit / s.dx ** 2, s.dtinit / s.dy ** 2)
        f.append(({k: c.field(k) for k in ("u", "p", "r", "w")}, res))
        c.close()
    (a, ra), (b, rb) = f
    if min(nx, ny) > 1:
        assert ra.iters == rb.iters == iters
        for k in "uprw":
            x, y = _interior(a[k], 1 if k in "up" else 2), _interior(b[k], 1 if k in "up" else 2)
            assert np.linalg.norm(x - y) <= 1e-9 * np.linalg.norm(y), k
    else:
        assert np.max(np.abs(_interior(a["u"]) - _interior(b["u"]))) <= 1e-14 * np.max(np.abs(b["u"]))
