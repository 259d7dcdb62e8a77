"""GPU: several handles of different sizes alive at once. A kernel's limit of
dynamic shared memory belongs to the kernel, so a small handle built (or used)
after a large one must leave the large one's calls as they are: they go
through, and the fields have the same bits before and after (the adjoint adds
with atomics, whose order is free, so of its call only that it goes through)."""
import numpy as np
import pytest

import giftbte_b200 as g
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def calls(s, nc):
    s.set_initial(300.0 + 0.1 * np.cos(np.arange(nc)))
    s.solve(max_iter=2, err_temp=0.0, err_flux=0.0)
    out = [s.fields()["T"]]
    s.vjp(T_bar=np.full(nc, 1.0 / nc), max_iter=2, tol=1e-300)
    s.set_initial(np.full(nc, 300.0))
    s.fourier_initial()
    return out + [s.fields()["T"]]


def test_a_small_handle_leaves_a_large_one():
    large, small = decks.config1_deck(70, n_phi=2), decks.config1_deck(8, n_phi=2)
    a = g.StaticBTESynthetic.from_deck(large, macro_exact=1)
    want = calls(a, large.mesh.n_cells)
    b = g.StaticBTESynthetic.from_deck(small, macro_exact=1)
    got = [calls(a, large.mesh.n_cells)]
    calls(b, small.mesh.n_cells)
    got.append(calls(a, large.mesh.n_cells))
    for r in got:
        for x, y in zip(want, r):
            assert np.array_equal(x, y)
    a.close()
    b.close()
