"""GPU: the moment kernel's two lane layouts. An FP64 solve with an even band
count gives a thread two bands, an odd count one; both form a band's sums in
the same order. Against the CPU restatement for counts of each kind (one band,
one pair, odd, several pairs; the last block short of cells), six outer
iterations from the same start, with the tolerances of the other step-by-step
comparisons (1e-10 of the temperature, 1e-9 of the flux, whose sums cancel)."""
import numpy as np
import pytest

import giftbte_b200 as g
import oracle
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 2, 3, 6, 20])
def test_moments_per_band_count(nb):
    d = decks.config2_deck(h_nm=12.0, n_bands=nb, n_phi=2, seed=3)
    T0 = 0.1 * np.cos(np.arange(d.mesh.n_cells))
    s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP64, macro_exact=1)
    s.set_initial(T0)
    s.solve(max_iter=6, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    o = oracle.solve(d, T0=T0, max_iter=6, err_T=0.0, err_q=0.0)
    for k, tol in (("T", 1e-10), ("q", 1e-9)):
        assert np.linalg.norm(f[k] - o[k]) <= tol * np.linalg.norm(o[k]), k
