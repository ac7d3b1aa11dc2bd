"""When keys are ranked by a prefix of their bytes: where the prefix leaves few runs
to settle, and short ones. Grouped keys (high halves from n / share values, low
halves random) whose runs would be long, or more than are listed, take more bytes
or all, and none is sorted twice."""
import numpy as np
import pytest

from tests.launched import kernels_of
from tests.test_rank_gpu import _rank
from tests.test_rank_prefix_gpu import _check

pytestmark = pytest.mark.gpu


def _passes(words):
    seen = kernels_of(lambda: _rank(words))
    return None if seen is None else sum("onesweep_pass" in name for name in seen)


# Keys a group (0: random keys); the most passes. Sampled in part, a longer prefix
# may do where a short one doesn't.
@pytest.mark.parametrize("n,share,most", [
    (20_000, 0, 7), (65_536, 0, 7), (65_537, 0, 7), (1 << 20, 0, 7), (3_000_000, 0, 7),
    (20_000, 32, 7), (65_536, 48, 7), (20_000, 4, 8), (20_000, 8, 8), (50_000, 200, 8),
    (65_536, 600, 8), (100_000, 2, 8), (1 << 20, 2, 8), (1 << 22, 1, 8), (1 << 24, 2, 8)])
def test_prefixes_only_where_they_pay(n, share, most):
    rng = np.random.default_rng(n + share)
    words = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if share:
        groups = rng.integers(0, 1 << 32, n // share, dtype=np.uint64) << np.uint64(32)
        words = groups[rng.integers(0, len(groups), n)] | (words >> np.uint64(32))
    passes = _passes(words)
    assert passes is None or passes <= most
    if passes is not None and n <= 65_536 and most == 8:
        assert passes == 8  # the whole input sampled: long runs aren't settled
    _check(words)
