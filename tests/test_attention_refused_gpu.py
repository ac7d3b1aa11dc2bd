"""How often the split attention's tile phase runs: once where its guards hold, once
where they fire whatever the exact maxima are (a refused call), and again, with
exact maxima, where a row lies between the bounds that the fast form keeps."""
import numpy as np
import pytest

from tests.launched import kernels_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset,spread,zeros,runs,taken", [
    (0.0, 10.0, True, 1, True), (0.0, 800.0, False, 1, True), (0.0, 800.0, True, 1, False),
    (2.0 ** 20, 800.0, True, 1, False),
    # The lightest score lies between two high words (half a unit apart there), the
    # limit of 707.69 between the spreads to them.
    (2.0 ** 20, 707.6, True, 2, True), (2.0 ** 20, 707.9, True, 2, False), (2.0 ** 20, 600.0, True, 1, True)])
def test_runs_of_the_tile_phase(offset, spread, zeros, runs, taken):
    import torch

    from einfold_b200 import autograd as A
    from einfold_b200.kernels import Precision

    q = torch.ones((2, 160, 1), dtype=torch.float64, device="cuda")
    k = (offset + torch.linspace(0.0, -spread, 130, dtype=torch.float64, device="cuda"))[None, :, None].repeat(2, 1, 1)
    v = torch.ones((2, 130, 5), dtype=torch.float64, device="cuda")
    if zeros:
        v[:, :, 3] = 0.0  # an output of 0: no lost term vanishes in its rounding

    def call():
        try:
            A.attention_forward(q, k, v, (), 1.0, Precision.SPLIT)
            return True
        except A.Declined:
            return False

    assert call() == taken  # (the shape's schedules are timed here)
    seen = kernels_of(call)
    assert seen is None or sum("attn_fwd_split" in name for name in seen) == runs
    assert call() == taken
