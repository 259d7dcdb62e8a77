"""GPU: the moment kernel with two bands per thread, which FP64 solves of an even
band count take where the launch then needs fewer waves: 190 and 570 blocks (one
band per thread) and 1,140 (two), rows that do not fill a warp. Against the CPU restatement as in
test_gpu_moments.py, with its tolerances."""
import numpy as np
import pytest

import giftbte_b200 as g
import oracle
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [40, 128, 130, 256])
def test_pairs_of_bands(nb):
    d = decks.config2_deck(h_nm=12.0, n_bands=nb, n_phi=2, seed=3)
    T0 = 0.1 * np.cos(np.arange(d.mesh.n_cells))
    s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP64, macro_exact=1)
    s.set_initial(T0)
    s.solve(max_iter=3, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    o = oracle.solve(d, T0=T0, max_iter=3, err_T=0.0, err_q=0.0)
    for k, tol in (("T", 1e-10), ("q", 1e-9)):
        assert np.linalg.norm(f[k] - o[k]) <= tol * np.linalg.norm(o[k]), k
