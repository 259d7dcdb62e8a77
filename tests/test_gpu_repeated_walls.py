"""GPU: boundary elements that name a cell face more than once, given twice in
the mesh or through two rows of the boundary table. The face itself refers to
the last of them; the others stay boundary sides whose values periodic
partners (transport, so in the Sequential scheme too) and node interpolations
(the synthetic source) read. Naming the pore's elements again doubles their
weights at its nodes, which are normalised, and a repeated periodic wall has
the values of the first, so the fields are those of the plain deck to
rounding: six outer iterations from the same start, with the tolerances of the step-by-step
comparisons in FP64 (1e-10 of the temperature, 1e-9 of the flux, whose sums
cancel) and 1e-5 in FP32."""
import dataclasses

import numpy as np
import pytest

import giftbte_b200 as g
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def twice(d, tags):
    m = d.mesh
    again = np.isin(m.edge_tags, tags)
    return dataclasses.replace(d, mesh=dataclasses.replace(
        m, edges=np.concatenate([m.edges, np.asarray(m.edges)[again]]),
        edge_tags=np.concatenate([m.edge_tags, np.asarray(m.edge_tags)[again]])))


def fields(d, prec):
    s = g.StaticBTESynthetic.from_deck(d, precision=prec, macro_exact=1)
    s.set_initial(0.1 * np.cos(np.arange(d.mesh.n_cells)))
    s.solve(max_iter=6, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    return f


@pytest.mark.parametrize("prec", [g.GBTE_FP64, g.GBTE_FP32_MIXED])
@pytest.mark.parametrize("nb", [4, 5])
@pytest.mark.parametrize("scheme,again", [
    ("Sequential", lambda d: twice(d, [1, 2, 3, 4, 5])),
    ("Synthetic", lambda d: twice(d, [5])),
    ("Sequential", lambda d: dataclasses.replace(d, bcs=list(d.bcs) + list(d.bcs))),
], ids=["all_twice", "pore_twice", "two_rows"])
def test_repeated_walls_change_nothing(scheme, again, nb, prec):
    d = decks.config4_deck(h_nm=20.0, n_bands=nb, n_phi=3, scheme=scheme)
    f, o = fields(again(d), prec), fields(d, prec)
    for k, tol in (("T", 1e-10), ("q", 1e-9)):
        tol = tol if prec == g.GBTE_FP64 else 1e-5
        assert np.linalg.norm(f[k] - o[k]) <= tol * np.linalg.norm(o[k]), k
