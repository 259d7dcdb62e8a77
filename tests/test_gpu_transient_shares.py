"""GPU: the explicit step from face values where its blocks take eight, four,
two or one direction of their cells (fewer as the grid gets too small for the
SMs), a last share short of directions; against the gradient arrays as in
test_gpu_transient_faces.py, with its tolerances."""
import numpy as np
import pytest

import giftbte_b200 as g
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nb,n_phi", [(48, 40, 8), (16, 40, 13), (16, 20, 19), (12, 6, 17), (9, 2, 5)])
def test_shares_match_gradient_arrays(nx, nb, n_phi):
    d = decks.grating_deck(nx=nx, ny=nx // 3, n_bands=nb, n_phi=n_phi)
    out = []
    for shape in (1, 0):
        s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP64, gradient_dirs=shape, residual_form=shape)
        r = s.transient_solve(1e-14, 10e-14)
        out.append((r["history"], s.fields()))
        s.close()
    (ha, fa), (hb, fb) = out
    for k in fa:
        tol = 1e-10 if k == "q" else 1e-12
        assert np.linalg.norm(fa[k] - fb[k]) <= tol * np.linalg.norm(fa[k]), k
    assert np.linalg.norm(ha - hb) <= 1e-12 * np.linalg.norm(ha)
