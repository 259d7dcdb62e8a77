"""GPU: the adjoint's gradient assembly where several threads share the
directions of a (cell, band) or (side, band): few bands, 64 directions or more,
shares that come out even or not, against central finite differences of the
forward solve as in test_gpu_adjoint.py, with its step and tolerance."""
import dataclasses

import numpy as np
import pytest

import test_gpu_adjoint as ta
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,n_phi", [(1, 16), (2, 19)])
def test_shared_directions(nb, n_phi):
    def deck(p=0.3):
        return decks.config4_deck(h_nm=25.0, n_bands=nb, n_phi=n_phi, seed=3, specularity=p, residual_temp=1e-12,
                                  residual_flux=1e-12, max_iter=8000)

    d0 = deck()
    sc = decks.lognormal_scatter(d0.mesh.n_cells, sigma=0.2, seed=4)

    def objective(s):
        qb = s.keff_cotangent(axis=0, length=ta.L, delta_T=1.0)
        return float(np.sum(qb * s.fields()["q"])), None, qb

    def tau_mult(b, h):
        m = np.ones(nb)
        m[b] += h
        return dataclasses.replace(d0, bands=dataclasses.replace(d0.bands, tau=d0.bands.tau * m))

    row = [i for i, b in enumerate(d0.bcs) if b.tag == 5][0]
    last = d0.mesh.n_cells - 1
    rows = ta.fd_check(lambda h, _: d0, sc, objective, [
        ("tau", lambda a: a["tau"][nb - 1], lambda h: (tau_mult(nb - 1, h), sc)),
        ("p", lambda a: a["specularity"][row], lambda h: (deck(0.3 + h), sc)),
        ("s", lambda a: a["scatter"][last] * sc[last],
         lambda h: (d0, sc * np.where(np.arange(len(sc)) == last, 1 + h, 1.0)))])
    for name, ga, fd in rows:
        assert abs(ga - fd) <= ta.TOL * max(abs(fd), 1e-3 * max(abs(r[2]) for r in rows)), (name, ga, fd)
