"""GPU: the macro CG on systems at the edges of its kernels. The cluster
kernel serves 16 cells (one aggregate too small for the coarse level) up to
what 16 CTAs hold; smaller and larger systems take the grid-wide kernel,
with up to 4 rows per thread in registers or none. Every solve reaches 1e-13 of the
right-hand side (macro_exact), so two iterations of the synthetic scheme
agree with the CPU oracle to 1e-9."""
import dataclasses

import numpy as np
import pytest

import giftbte_b200 as g
import oracle
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def check(d, iters=2):
    s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP64, macro_exact=1)
    st = s.solve(max_iter=iters, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    o = oracle.solve(dataclasses.replace(d, residual_temp=0.0, residual_flux=0.0), max_iter=iters)
    assert st["macro_cg_iterations"] > 0
    for k in ("T", "E"):
        assert np.linalg.norm(f[k] - o[k]) <= 1e-9 * np.linalg.norm(o[k]), k


@pytest.mark.parametrize("n", [1, 2, 3, 11, 46])
def test_squares_match_oracle(n):
    # 2, 8 (grid-wide), 18 (cluster, no coarse level), 242 and 4232 cells
    check(decks.config1_deck(n, n_phi=1))


@pytest.mark.parametrize("copies,rows", [(5, 1), (9, 2), (16, 3), (22, 4), (26, 0)])
def test_grid_wide_kernel_matches_the_cluster(copies, rows):
    # 12,000 tetrahedra alone fit the cluster; `copies` of them as one system
    # take the grid-wide kernel with `rows` rows per thread of 148 x 512 (0:
    # more than registers hold). Each copy's temperatures are the single
    # block's to the solves' 1e-13, through a few Picard steps
    d = decks.config3_deck(h_nm=1.0, size_nm=(10.0, 10.0, 20.0), n_bands=1, n_theta=1, n_phi=1)
    n = d.mesh.n_cells * copies
    assert (75776 * (rows - 1) < n <= 75776 * rows) if rows else n > 4 * 75776
    fields = []
    for make, arg in ((g.StaticBTESynthetic.from_deck, d), (g.StaticBTESynthetic.from_decks, [d] * copies)):
        s = make(arg, precision=g.GBTE_FP64, macro_exact=1)
        s.solve(max_iter=2, err_temp=0.0, err_flux=0.0)
        fields.append(s.fields()["T"])
        s.close()
    one, all_ = fields[0], fields[1].reshape(copies, -1)
    assert np.max(np.abs(all_ - one)) <= 1e-9 * np.max(np.abs(one))
