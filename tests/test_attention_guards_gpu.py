"""The split attention's guards at their threshold: the fast form keeps bounds of
a row's largest and lightest scores from their high words and leaves what they
don't settle to exact ones, so a spread of scores is taken or refused as by the
FP64 form on both sides of the limit, and the values agree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [1.0, 2.0 ** -40, 2.0 ** 900])
@pytest.mark.parametrize("keys", [2, 65, 130])
def test_spreads_are_taken_and_refused_as_in_fp64(keys, value):
    import torch

    from einfold_b200 import autograd as A
    from einfold_b200.kernels import Precision

    # The least normal weight times the value: exp(-spread)·value = 2^-1022.
    edge = (1022.0 + min(np.log2(value), 0.0)) * np.log(2.0)
    taken = 0
    for spread in (1.0, edge - 40.0, edge - 1.0, edge - 1e-3, edge - 1e-4, edge + 1e-4, edge + 1e-3, edge + 1.0, 800.0):
        q = torch.full((1, 5, 1), 3.0, dtype=torch.float64, device="cuda")
        k = torch.linspace(0.0, -spread / 3.0, keys, dtype=torch.float64, device="cuda")[None, :, None].contiguous()
        v = torch.full((1, keys, 3), value, dtype=torch.float64, device="cuda")
        v[:, ::2, 1] *= -1.0

        def outcome(precision):
            try:
                return A.attention_forward(q, k, v, (), 1.0, precision)
            except Exception as e:
                return type(e).__name__

        # Ragged, so that a few queries take the tile kernels too.
        def ragged(precision):
            try:
                return A.attention_forward(q, k, v, (), 1.0, precision, q_lengths=torch.tensor([5]))
            except Exception as e:
                return type(e).__name__

        for run in (outcome, ragged):
            a, b = run(Precision.SPLIT), run(Precision.FP64)
            assert isinstance(a, str) == isinstance(b, str), (spread, a, b)
            if isinstance(a, str):
                assert a == b
                continue
            taken += 1
            # Scores to 2·2^-45 of the spread, doubled by the sum; values to 2^-45.
            bound = (4 * spread + 4) * 2.0 ** -45
            assert float((a[0] - b[0]).abs().max()) <= bound * value
            assert float((a[1] - b[1]).abs().max()) <= bound
    assert taken >= 4
