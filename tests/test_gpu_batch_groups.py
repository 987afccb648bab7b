"""Batches' groups of blocks.  Blocks of a group have nothing to do for as long
as a deck of one block takes: here some seconds, with a large iteration budget and
no bound to meet, longer than any wait's own limit.
"""
import numpy as np
import pytest

from parity_util import random_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_long_solves_on_one_block(tl, built_lib, precision):
    budget = 300_000
    texts = [random_deck(n, 6, eps=0.0).replace("max_iters=5000", f"max_iters={budget}") for n in (300, 10, 10, 11)]
    sets = [tl.Settings.from_text(t, mode=1, criterion=1, precision=precision) for t in texts]
    chunks = [tl.initialiseapp(s) for s in sets]
    for c, s in zip(chunks, sets):
        tl.haloupdate(c, s, 1, ["energy", "density"])
    b = tl.Batch(chunks)
    res = b.solve(sets)
    b.close()
    for c in chunks:
        c.close()
    # FP32's refinements may end where the residual is NaN (0/0 after it has become 0)
    assert all(not r.converged and (r.iters == budget if precision == 0 else r.iters > 0) for r in res)


@pytest.mark.parametrize("after", [False, True])
def test_batches_choose_their_own_layout(tl, built_lib, after):
    """tl_set_layout on a context, before or after a batch's first solve, changes
    nothing for the batch: the sums' order, and so u's bits, are those of a context
    without it."""
    text = random_deck(300, 8, ny=211, eps=1e-10, steps=2)
    u = []
    for change in (False, True):
        s = tl.Settings.from_text(text, mode=1, criterion=1, precision=1)
        c = tl.initialiseapp(s)
        b = tl.Batch([c])
        for step in range(2):
            if change and step == after:
                c.check(c.lib.tl_set_layout(c.ctx, 9, 8, 7, 2))
            tl.haloupdate(c, s, 1, ["energy", "density"])
            assert b.solve([s])[0].converged
            tl.solvefinished(c, s)
        u.append(c.field("u"))
        b.close()
        c.close()
    np.testing.assert_array_equal(u[0], u[1])
