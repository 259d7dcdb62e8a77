"""GPU: band tables of many materials. The face-value residual stages the whole
table and its coefficients in shared memory, 48 KB at most; larger tables run
on the gradient arrays. At both sides of that line (in FP64 a row of 2 or 4
bands has 32 KB of coefficients beside 24 bytes per band and material) the
solve goes through, and agrees with the gradient arrays as in
test_gpu_face_values.py and with its tolerances."""
import dataclasses

import numpy as np
import pytest

from giftbte_b200 import decks
from test_gpu_face_values import F32, F64, fields

pytestmark = pytest.mark.gpu


def table(n_bands, n_mat):
    d = decks.interface_deck(6, n_bands=n_bands)
    left, right = d.bands, d.extra_materials[0]
    t = np.concatenate([b.trans for b in d.bcs if b.trans is not None])
    t = np.concatenate([t, np.full((n_mat - 2, n_bands), 0.5)])
    return dataclasses.replace(d, extra_materials=[right] + [left] * (n_mat - 2),
                               bcs=[dataclasses.replace(b, trans=t) if b.type == 5 else b for b in d.bcs])


@pytest.mark.parametrize("prec,nb,n_mat,faces", [(F64, 4, 170, True), (F64, 4, 171, False), (F64, 2, 341, True),
                                                 (F64, 2, 342, False), (F64, 8, 171, False), (F32, 4, 409, True),
                                                 (F32, 4, 410, False)])
def test_band_table_at_the_shared_memory_line(prec, nb, n_mat, faces):
    d = table(nb, n_mat)
    a, _ = fields(d, prec, 1)
    b, st = fields(d, prec, 0)
    assert (st["residual_form"] == 9) == faces
    for k in a:
        tol = (1e-10 if k == "q" else 1e-12) if prec == F64 else 1e-6
        assert np.linalg.norm(a[k] - b[k]) <= tol * np.linalg.norm(a[k]), k
