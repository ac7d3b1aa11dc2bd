"""The Gaussian smoother's rows with scores past its clamp (weights below e^-700
counted as lost): the same outcome as the exact kernel's (EINFOLD_TILES_GENERAL=1),
and where both take the call, the same values."""
import numpy as np
import pytest

from einfold_b200 import ir
from tests import pipelines as P
from tests.test_gauss_rows_gpu import _run

pytestmark = pytest.mark.gpu

# The near key's value and the far keys', and the far keys' score (the near one's
# is 0): outputs the clamped weights would show in, and ones they wouldn't.
CASES = [(0.0, 1.0, -900.0), (0.0, 1e300, -900.0), (0.0, 1e300, -701.0), (1e-200, 1e200, -1000.0),
         (1e-300, 1.0, -900.0), (1e-300, 1.0, -720.0), (1e-280, 1.0, -800.0), (1.0, 1.0, -900.0),
         (1.0, 1e280, -900.0), (1.0, 1e300, -900.0), (1.0, -1.0, -701.0), (3.0, 2.0, -699.0), (0.0, 0.0, -900.0)]


@pytest.mark.parametrize("normalizer", [ir.Normalizer.KEPT_GROUPS, ir.Normalizer.NONE])
@pytest.mark.parametrize("rows,keys", [(3, 2), (200, 130)])
@pytest.mark.parametrize("near,far,score", CASES)
def test_clamped_weights_count_as_lost(near, far, score, rows, keys, normalizer, monkeypatch):
    _compare(near, far, score, rows, keys, normalizer, monkeypatch)


@pytest.mark.parametrize("near,far,score", [(1e-300, 1.0, -900.0), (1.0, 1.0, -900.0)])
def test_clamped_weights_of_two_rows_a_thread(near, far, score, monkeypatch):
    _compare(near, far, score, 152_000, 3, ir.Normalizer.KEPT_GROUPS, monkeypatch)


def _compare(near, far, score, rows, keys, normalizer, monkeypatch):
    def keyed(first, rest):
        def values(n):
            x = np.full(n, rest)
            x[:1] = first
            return x

        return values

    for h, scale in ((1.0, ir.Scale.one()), (0.25, ir.Scale.over(0.25))):
        case = P.attention(rows, d=1, lk=keys, scores=P.gaussian_scores(), weight=ir.Weight.exp(scale, ir.Shift.NONE),
                           normalizer=normalizer, q_value=lambda n: np.zeros(n),
                           k_value=keyed(0.0, np.sqrt(-score * h)), v_value=keyed(near, far))
        got, want = _run(case, monkeypatch), _run(case, monkeypatch, general=True)
        assert (got is None) == (want is None), (near, far, score)
        if want is not None:
            assert got[0] == want[0]
            # Weights round to a unit or two, with half a unit of a score of 900
            # in the exponent where one counts at all.
            assert np.max(np.abs(got[2] - want[2])) <= 1e-12 * np.max(np.abs(want[2]))
