"""GPU: the wall passes where several threads share the directions of a wall's
band: few bands, 64 directions or more, shares that come out even or not (the
last one short). Against the CPU restatement with diffuse, partially specular
and periodic walls; across an interface, where that has no counterpart,
against the same materials with every band cut into 128 equal ones (all
directions of a band then with one thread). Three outer iterations in FP64
from the same start, with the tolerances of the other step-by-step comparisons
(1e-10 of the temperature, 1e-9 of the flux, whose sums cancel)."""
import dataclasses

import numpy as np
import pytest

import giftbte_b200 as g
import oracle
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def solve(d, T0):
    s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP64, macro_exact=1)
    s.set_initial(T0)
    s.solve(max_iter=3, err_temp=0.0, err_flux=0.0)
    f = s.fields()
    s.close()
    return f


def agree(f, o):
    for k, tol in (("T", 1e-10), ("q", 1e-9)):
        assert np.linalg.norm(f[k] - o[k]) <= tol * np.linalg.norm(o[k]), k


@pytest.mark.parametrize("scheme", ["Synthetic", "Sequential"])
@pytest.mark.parametrize("make", [
    lambda **k: decks.config1_deck(6, n_phi=65, **k),
    lambda **k: decks.config4_deck(h_nm=25.0, n_bands=1, n_phi=16, **k),
    lambda **k: decks.config4_deck(h_nm=25.0, n_bands=2, n_phi=25, **k),
    lambda **k: decks.config4_deck(h_nm=25.0, n_bands=7, n_phi=51, **k),
], ids=["gray260", "one64", "two100", "seven204"])
def test_many_directions_match_oracle(make, scheme):
    d = make(scheme=scheme)
    T0 = d.tref + 0.1 * np.cos(np.arange(d.mesh.n_cells))
    agree(solve(d, T0), oracle.solve(d, T0=T0, max_iter=3, err_T=0.0, err_q=0.0))


@pytest.mark.parametrize("n_phi", [17, 40])
def test_interface_matches_a_finer_band_table(n_phi):
    d = decks.interface_deck(4, n_bands=2, n_phi=n_phi)

    def cut(b):
        r = {k: np.repeat(getattr(b, k), 128) for k in ("v", "tau", "C", "lattice_ratio", "heat_ratio")}
        for k in ("C", "lattice_ratio", "heat_ratio"):
            r[k] = r[k] / 128
        return dataclasses.replace(b, **r)

    fine = dataclasses.replace(
        d, bands=cut(d.bands), extra_materials=[cut(m) for m in d.extra_materials],
        bcs=[b if b.type != 5 else dataclasses.replace(b, trans=np.repeat(b.trans, 128, axis=1)) for b in d.bcs])
    T0 = 300.0 + 0.1 * np.cos(np.arange(d.mesh.n_cells))
    agree(solve(d, T0), solve(fine, T0))
