"""GPU: the explicit step from face values, in place, against the step from
gradient arrays (options.gradient_dirs = residual_form = 1). Both evaluate the
same expression with the same gradients; the sums are associated differently,
so a step differs by a few FP64 roundings of the field: 1e-12 of the
temperature and of the probe's history after 20 steps, 1e-10 of the flux,
whose sums cancel. Sizes: rows of one and several 16-byte pieces, a last block
short of cells, direction batches, triangles, quadrilaterals and tetrahedra;
an odd band count takes the gradient arrays on both sides."""
import dataclasses

import numpy as np
import pytest

import giftbte_b200 as g
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def build(name, nb):
    if name == "grating":
        return decks.grating_deck(nx=13, ny=5, n_bands=nb)
    if name == "quads":
        return dataclasses.replace(decks.grating_deck(n_bands=nb), mesh=decks.square_quad_mesh(9, 7))
    if name == "triangles":
        return decks.config2_deck(h_nm=12.0, n_bands=nb, n_phi=2, seed=3)
    return decks.config3_deck(h_nm=20.0, size_nm=(60.0, 60.0, 40.0), n_bands=nb, n_theta=2, n_phi=1)


@pytest.mark.parametrize("name,nb,batch", [("grating", 2, 0), ("grating", 20, 0), ("grating", 6, 3), ("quads", 6, 0),
                                           ("triangles", 20, 0), ("triangles", 4, 5), ("tets", 2, 0), ("tets", 8, 3),
                                           ("grating", 3, 0)])
def test_face_step_matches_gradient_arrays(name, nb, batch):
    d = build(name, nb)
    out = []
    for shape in (1, 0):
        s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP64, gradient_dirs=shape, residual_form=shape,
                                           direction_batch=batch)
        r = s.transient_solve(1e-14, 20e-14)
        f = s.fields()
        s.close()
        out.append((r, f))
    (ra, fa), (rb, fb) = out
    assert ra["steps"] == rb["steps"]
    assert np.isfinite(fa["T"]).all()
    for k in fa:
        tol = 1e-10 if k == "q" else 1e-12
        assert np.linalg.norm(fa[k] - fb[k]) <= tol * np.linalg.norm(fa[k]), k
    assert np.linalg.norm(ra["history"] - rb["history"]) <= 1e-12 * np.linalg.norm(ra["history"])
