"""GPU: the face-value transport on quadrilaterals (four faces per 2D cell) in
both precisions, against the gradient arrays as in test_gpu_face_values.py and
with its tolerances: one and several 16-byte pieces per row, heat and specular
walls, direction batches."""
import dataclasses

import pytest

from giftbte_b200 import decks
from test_gpu_face_values import F32, F64, compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("nb,batch", [(4, 0), (8, 5), (20, 0)])
def test_quadrilaterals_match_gradient_arrays(prec, nb, batch):
    d = decks.config1_deck(9, n_phi=3)
    mesh = decks.jitter_interior(decks.square_quad_mesh(9, 7), 0.02, seed=4)
    bcs = [decks.BC(1, 1, 301.0), decks.BC(2, 1, 299.0), decks.BC(3, 3, 0.0), decks.BC(4, 6, 0.4)]
    d = dataclasses.replace(d, mesh=mesh, bands=decks.sine_dispersion_bands(nb), bcs=bcs, heat_source=1e16)
    compare(d, prec, direction_batch=batch)
