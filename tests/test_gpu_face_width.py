"""GPU: the face-value gradient where the mesh's tiles are too large for two
blocks of the widest kind on an SM: cells in the caller's order, shuffled
within windows of growing length, so that the block width goes down from its
widest through the fine steps to a block alone on its SM. Against the
gradient arrays, as in test_gpu_face_values.py and with its tolerances."""
import dataclasses

import numpy as np
import pytest

from giftbte_b200 import decks
from test_gpu_face_values import F32, F64, compare

pytestmark = pytest.mark.gpu


def shuffled(window):
    d = decks.config3_deck(h_nm=10.0, size_nm=(100.0, 100.0, 70.0), n_bands=4, n_theta=2, n_phi=1)
    m = d.mesh
    n = m.n_cells
    rng = np.random.default_rng(window)
    key = np.arange(n) // window + rng.random(n)
    idx = np.argsort(key, kind="stable")
    return dataclasses.replace(d, mesh=dataclasses.replace(m, cells=np.asarray(m.cells)[idx],
                                                           cell_region=np.asarray(m.cell_region)[idx]))


@pytest.mark.parametrize("prec", [F32, F64])
@pytest.mark.parametrize("window", [1, 60, 120, 4200])
def test_block_widths(prec, window):
    compare(shuffled(window), prec, cell_order=1)
