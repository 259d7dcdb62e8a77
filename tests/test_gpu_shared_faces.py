"""GPU: cells that share two faces (a concave quadrilateral and the cell in its
notch). The global face list then has no one-to-one pairing of cell faces, so
these meshes take the gradient-array kernels, and every cell face keeps its
own centre. Against the CPU restatement in the Sequential scheme, that is the
transport alone, with directions in which no two cells feed each other (the
sweep would lag one of them), six outer iterations from the same start, with the tolerances of the other step-by-step comparisons in FP64
(1e-10 of the temperature, 1e-9 of the flux, whose sums cancel) and 1e-5 in
FP32."""
import dataclasses

import numpy as np
import pytest

import giftbte_b200 as g
import oracle
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def notched_square(n, nb):
    """n x n squares, each cut into a concave and a convex quadrilateral that
    share the two edges at an inner point."""
    m = decks.square_quad_mesh(n, n)
    nodes, cells = [tuple(p) for p in m.nodes], []
    for a, b, d, c in m.cells:
        A, B, D = (np.asarray(nodes[i]) for i in (a, b, d))
        p = len(nodes)
        nodes.append(tuple(A + 0.47 * (B - A) + 0.48 * (D - A)))
        cells += [(b, p, a, d), (b, c, p, d)]
    mesh = dataclasses.replace(m, nodes=np.asarray(nodes), cells=np.asarray(cells),
                               cell_region=np.zeros(len(cells), dtype=np.int64))
    return dataclasses.replace(decks.config1_deck(n, n_phi=2, scheme="Sequential"), mesh=mesh, bands=decks.sine_dispersion_bands(nb))


@pytest.mark.parametrize("prec", [g.GBTE_FP64, g.GBTE_FP32_MIXED])
@pytest.mark.parametrize("nb", [4, 5])
def test_cells_sharing_two_faces_match_oracle(nb, prec):
    d = notched_square(8, nb)
    T0 = 300.0 + 0.1 * np.cos(np.arange(d.mesh.n_cells))
    s = g.StaticBTESynthetic.from_deck(d, precision=prec, macro_exact=1)
    s.set_initial(T0)
    s.solve(max_iter=6, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    o = oracle.solve(d, T0=T0, max_iter=6, err_T=0.0, err_q=0.0)
    for k, tol in (("T", 1e-10), ("q", 1e-9)):
        tol = tol if prec == g.GBTE_FP64 else 1e-5
        assert np.linalg.norm(f[k] - o[k]) <= tol * np.linalg.norm(o[k]), k
