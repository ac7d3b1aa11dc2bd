"""Ranking by a prefix of the varying bytes: keys the prefix leaves out of order
(runs settled afterwards), keys a sample of them turns away, and keys that pass
the sample and are sorted again by every byte, against numpy's order."""
import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import kernels as K
from tests.test_rank_gpu import _rank

pytestmark = pytest.mark.gpu

SAMPLE = 1 << 16


def _check(words):
    rank, first, k = _rank(words)
    u, at, inv = np.unique(words, return_index=True, return_inverse=True)
    assert k == len(u)
    assert np.array_equal(rank, inv.astype(np.uint32))
    assert np.array_equal(first, at.astype(np.uint32))


def _random(n, seed=1):
    return np.random.default_rng(seed).integers(0, 1 << 64, n, dtype=np.uint64)


def _unsampled(n):
    """Rows the sample (row i·n/65536 for each i) doesn't read."""
    rows = np.ones(n, dtype=bool)
    rows[(np.arange(SAMPLE) * n) // SAMPLE] = False
    return np.flatnonzero(rows)


@pytest.mark.parametrize("n", [300, 65536, 65537, 1 << 20, 5_000_001])
@pytest.mark.parametrize("repeats", [1, 3])
def test_random_keys(n, repeats):
    _check(np.random.default_rng(n).permutation(np.repeat(_random(n // repeats + 1), repeats))[:n].copy())


@pytest.mark.parametrize("n", [60_000, 1 << 20])
def test_heavy_keys_beside_random_ones(n):
    words = _random(n)
    words[::3] = words[0]
    words[1::5] = words[0] ^ np.uint64(1)  # the same prefix, another key
    words[2::7] = words[2]
    _check(words)


@pytest.mark.parametrize("share", [2, 50, 5000])
def test_groups_of_keys_under_one_prefix(share):
    # High halves from n / share random values, low halves random: the bytes look
    # independent, the prefixes aren't.
    n = 200_000
    rng = np.random.default_rng(share)
    high = _random(n // share, 2)[rng.integers(0, n // share, n)] & np.uint64(0xffffffff00000000)
    _check(high | rng.integers(0, 1 << 32, n, dtype=np.uint64))


@pytest.mark.parametrize("run", [2, 3, 33, 1024, 1025, 3000])
def test_runs_the_sample_misses(run):
    # One run of `run` keys under one prefix, descending, in rows the sample skips:
    # settled up to 1,024 keys, sorted again beyond.
    n = 1 << 20
    words = _random(n)
    rows = _unsampled(n)[1000:1000 + run]
    words[rows] = (words[rows[0]] & np.uint64(0xffffffff00000000)) | np.arange(run, 0, -1, dtype=np.uint64) * np.uint64(977)
    _check(words)


def test_more_runs_than_are_listed():
    n = 1 << 20
    words = _random(n)
    rows = _unsampled(n)[: 1 << 18].reshape(-1, 2)
    words[rows[:, 1]] = words[rows[:, 0]] ^ np.uint64(1)
    _check(words)


@pytest.mark.parametrize("n", [5000, 300_000])
def test_names_of_sixteen_digits(n):
    rng = np.random.default_rng(n)
    names = [f"{x:016x}" for x in rng.integers(0, 1 << 62, n)]
    picked = [names[i] for i in rng.integers(0, n, n)]
    picked[5] = None
    t = pa.record_batch([pa.array(picked)], names=["k"])
    got = K.rank_columns(K.Relation(t.schema, [t]), [0])
    order = sorted({p for p in picked if p is not None})
    place = {None: 0, **{p: i + 1 for i, p in enumerate(order)}}
    assert np.array_equal(got.rank, np.array([place[p] for p in picked], dtype=np.uint32))
    assert [picked[i] for i in got.first] == [None, *order]
