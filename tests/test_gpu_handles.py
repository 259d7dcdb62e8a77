"""GPU: what a handle holds, and several handles of different sizes alive at
once. A kernel's limit of
dynamic shared memory belongs to the kernel, so a small handle built (or used)
after a large one must leave the large one's calls as they are: they go
through, and the fields have the same bits before and after (the adjoint adds
with atomics, whose order is free, so of its call only that it goes through)."""
import dataclasses

import numpy as np
import pytest
import torch

import giftbte_b200 as g
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


def calls(s, nc):
    s.set_initial(300.0 + 0.1 * np.cos(np.arange(nc)))
    s.solve(max_iter=2, err_temp=0.0, err_flux=0.0)
    out = [s.fields()["T"]]
    s.vjp(T_bar=np.full(nc, 1.0 / nc), max_iter=2, tol=1e-300)
    s.set_initial(np.full(nc, 300.0))
    s.fourier_initial()
    return out + [s.fields()["T"]]


def test_a_small_handle_leaves_a_large_one():
    large, small = decks.config1_deck(70, n_phi=2), decks.config1_deck(8, n_phi=2)
    a = g.StaticBTESynthetic.from_deck(large, macro_exact=1)
    want = calls(a, large.mesh.n_cells)
    b = g.StaticBTESynthetic.from_deck(small, macro_exact=1)
    got = [calls(a, large.mesh.n_cells)]
    calls(b, small.mesh.n_cells)
    got.append(calls(a, large.mesh.n_cells))
    for r in got:
        for x, y in zip(want, r):
            assert np.array_equal(x, y)
    a.close()
    b.close()


def test_face_value_buffers_only_where_they_can_be_used():
    # the mask (a byte per direction and cell) and the wall gradients belong to
    # handles that can take the face-value transport; a fixed launch shape cannot
    d = decks.config1_deck(70, n_phi=256)
    nc, nd = d.mesh.n_cells, 1024

    def held(**kw):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s = g.StaticBTESynthetic.from_deck(d, precision=g.GBTE_FP32_MIXED, **kw)
        used = before - torch.cuda.mem_get_info()[0]
        assert s.num_directions == nd
        s.close()
        return used

    d = dataclasses.replace(d, bands=decks.sine_dispersion_bands(4))
    held()  # the context's own first allocations
    both = held(gradient_dirs=1, residual_form=1), held()
    assert both[1] - both[0] >= nc * nd
