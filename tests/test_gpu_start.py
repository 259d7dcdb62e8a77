"""GPU: the start of the face-value transport. An FP32 start has no deviation
from its base and gets zeros instead of a field and its gradient; the first
iteration of a new start does without its gradient where the start's face
values are all there. Neither may leak into a later iteration or a later call:
two calls of one iteration give the bits of one call of two, and a handle that
is given a new start gives the bits of a new handle. With direction batches
the FP64 form has to form the gradients again; an FP32 start need not."""
import numpy as np
import pytest

import giftbte_b200 as g
from giftbte_b200 import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [0, 5])
@pytest.mark.parametrize("prec", [g.GBTE_FP32_MIXED, g.GBTE_FP64])
def test_start_is_the_first_iterations_gradient_only(prec, batch):
    d = decks.config2_deck(h_nm=12.0, n_bands=8, n_phi=2, seed=3)
    T0 = 0.1 * np.cos(np.arange(d.mesh.n_cells))

    def handle():
        s = g.StaticBTESynthetic.from_deck(d, precision=prec, macro_exact=1, direction_batch=batch)
        s.set_initial(T0)
        return s

    def run(s, *iters):
        for n in iters:
            s.solve(max_iter=n, err_temp=0.0, err_flux=0.0)
        return s.fields()

    a = handle()
    b = handle()
    want = run(a, 2)
    assert a.stats["gradient_dirs"] == 11
    got = [run(b, 1, 1)]
    run(b, 1)
    b.set_initial(T0)
    got.append(run(b, 2))
    for f in got:
        for k in want:
            assert np.array_equal(f[k], want[k]), k
    a.close()
    b.close()
