"""GPU: the face-value transport (the automatic launch shapes) against the
gradient-array kernels (options.gradient_dirs = residual_form = 1). Both
form the same face values from the same gradients, so FP64 fields differ by
rounding of the operations that follow (1e-12 of the field, 1e-10 of the
flux, whose sums cancel), and FP32 fields by at most a few ulps of the
deviations per iteration (1e-6). Sizes: band counts whose rows are one or
several 16-byte pieces, slabs that cross directions and end ragged, blocks
with a short last block, direction batches, quads, two materials, several
geometries."""
import numpy as np
import pytest

import giftbte_b200 as g
import make_golden as mg
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu

F32, F64 = g.GBTE_FP32_MIXED, g.GBTE_FP64


def fields(deck, prec, shape, iters=6, **kw):
    make = g.StaticBTESynthetic.from_decks if isinstance(deck, list) else g.StaticBTESynthetic.from_deck
    s = make(deck, precision=prec, gradient_dirs=shape, residual_form=shape, macro_exact=1, **kw)
    st = s.solve(max_iter=iters, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    return f, st


def compare(deck, prec, **kw):
    a, _ = fields(deck, prec, 1, **kw)
    b, st = fields(deck, prec, 0, **kw)
    assert st["residual_form"] == 9 and st["gradient_dirs"] == 11
    for k in a:
        tol = (1e-10 if k == "q" else 1e-12) if prec == F64 else 1e-6
        assert np.linalg.norm(a[k] - b[k]) <= tol * np.linalg.norm(a[k]), k


@pytest.mark.parametrize("prec,nb,n_phi", [(F32, 4, 1), (F32, 12, 3), (F32, 40, 2), (F32, 100, 1), (F64, 2, 1), (F64, 6, 3),
                                           (F64, 40, 2), (F64, 74, 1)])
def test_plane_matches_gradient_arrays(prec, nb, n_phi):
    compare(decks.config2_deck(h_nm=11.0, n_bands=nb, n_phi=n_phi, seed=3), prec)


@pytest.mark.parametrize("prec,nb,batch", [(F32, 4, 0), (F32, 12, 5), (F32, 40, 0), (F64, 2, 3), (F64, 10, 0),
                                           (F64, 40, 7)])
def test_tetrahedra_match_gradient_arrays(prec, nb, batch):
    d = decks.config3_deck(h_nm=10.0, size_nm=(30.0, 40.0, 50.0), n_bands=nb, n_theta=2, n_phi=1)
    compare(d, prec, direction_batch=batch)


@pytest.mark.parametrize("prec", [F32, F64])
def test_quads_materials_and_batches(prec):
    quad, _ = mg.load("quad_heat_specular")
    if quad.bands.n_bands * (4 if prec == F32 else 8) % 16 == 0:
        compare(quad, prec)
    compare(decks.interface_deck(10, n_bands=8), prec)
    compare(decks.porous_population(2, seed=1, h_nm=(15.0, 22.0), r_nm=(40.0, 80.0), n_bands=8, n_phi=2), prec)


def test_other_band_counts_keep_the_one_band_kernels():
    d = decks.config2_deck(h_nm=14.0, n_bands=6, n_phi=2, seed=3)
    assert fields(d, F32, 0)[1]["residual_form"] == 0
    assert fields(decks.config2_deck(h_nm=14.0, n_bands=5, n_phi=2, seed=3), F64, 0)[1]["residual_form"] == 0
