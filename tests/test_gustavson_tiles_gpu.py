"""The sparse product by tiles of 512 output columns, at the tiles' edges,
with repeated (z, y) rows, NULL factors, infinities and NaN, and beside it the
form without tiles (too many items): rows, bits and NULLs as the oracle's."""
import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import ir, kernels as K
from oracle import oracle

pytestmark = pytest.mark.gpu

E = ir.EQ
FOLD = ir.Fold([E, E, E], [ir.Operand([(0, 0), (1, 1)], 2), ir.Operand([(1, 0), (2, 1)], 2)],
               [ir.Output(0), ir.Output(2)])

CASES = {
    # distinct i, j, k; rows of a and b; share of NULL factors; special values
    "one_tile": (7, 5, 512, 40, 4000, 0.0, False),
    "a_tile_and_one": (9, 6, 513, 60, 5000, 0.05, False),
    "just_under": (3, 4, 511, 30, 9000, 0.05, True),
    "ten_tiles": (40, 11, 5000, 300, 24000, 0.02, True),
    "many_rows_an_x": (2, 90, 1500, 900, 9000, 0.02, False),
    "one_pair": (1, 1, 1, 1, 1, 0.0, False),
    "all_null": (4, 3, 1100, 30, 3000, 1.0, False),
    "few_pairs": (3000, 4000, 5000, 3500, 6000, 0.02, False),
}


def _tables(name, strings):
    ni, nj, nk, ra, rb, null, special = CASES[name]
    rng = np.random.default_rng(len(name))

    def key(n, rows, cover):
        pick = np.concatenate([np.arange(n), rng.integers(0, n, rows - n)]) if cover and rows >= n else \
            rng.integers(0, n, rows)
        ids = rng.permutation(rng.choice(1 << 40, n, replace=False))[pick]
        return ids

    def column(ids):
        return pa.array([f"{x:016x}" for x in ids]) if strings else pa.array(ids)

    js = rng.choice(1 << 40, nj, replace=False)

    def values(n):
        v = rng.standard_normal(n)
        if special:
            v[::17] = np.inf
            v[5::29] = np.nan
        return pa.array(v, mask=rng.uniform(size=n) < null)

    a = pa.record_batch([column(key(ni, ra, True)), pa.array(js[rng.integers(0, nj, ra)]), values(ra)],
                        names=["i", "j", "v"])
    b = pa.record_batch([pa.array(js[rng.integers(0, nj, rb)]), column(key(nk, rb, True)), values(rb)],
                        names=["j", "k", "v"])
    return a, b


@pytest.mark.parametrize("strings", [False, True])
@pytest.mark.parametrize("name", list(CASES))
def test_tiles_give_the_oracles_bits(name, strings):
    a, b = _tables(name, strings)
    got = K.fold(FOLD, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))
    want = oracle.fold(FOLD, a.schema, [a], b.schema, [b], None, oracle.schema(FOLD, [a.schema, b.schema]))
    if name != "one_pair" or strings:
        assert got.algorithm == K.Algorithm.DISCRIMINATE
    g, w = pa.Table.from_batches(got.batches), pa.Table.from_batches(want.batches)
    assert g.num_rows == w.num_rows
    for c in range(2):
        assert g.column(c).to_pylist() == w.column(c).to_pylist()
    gv, wv = g.column(2).combine_chunks(), w.column(2).combine_chunks()
    assert gv.null_count == wv.null_count and gv.is_valid().equals(wv.is_valid())
    x, y = (np.asarray(v.fill_null(0.0)) for v in (gv, wv))
    assert np.array_equal(np.isnan(x), np.isnan(y))
    assert np.array_equal(x[~np.isnan(x)].view(np.uint64), y[~np.isnan(y)].view(np.uint64))


def test_more_items_than_tiles_are_kept_for():
    # 600,000 x by 118 tiles: beyond 2^26 items.
    rng = np.random.default_rng(2)
    js = rng.choice(1 << 40, 60_000, replace=False)
    a = pa.record_batch([pa.array(rng.permutation(600_000) << 20), pa.array(rng.choice(js, 600_000)),
                         pa.array(rng.standard_normal(600_000))], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(js), pa.array(rng.permutation(60_000) << 20), pa.array(rng.standard_normal(60_000))],
                        names=["j", "k", "v"])
    got = K.fold(FOLD, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))
    want = oracle.fold(FOLD, a.schema, [a], b.schema, [b], None, oracle.schema(FOLD, [a.schema, b.schema]))
    assert got.algorithm == K.Algorithm.DISCRIMINATE
    g, w = pa.Table.from_batches(got.batches), pa.Table.from_batches(want.batches)
    assert g.num_rows == w.num_rows == 600_000
    for c in range(3):
        assert np.array_equal(g.column(c).to_numpy(), w.column(c).to_numpy())


@pytest.mark.parametrize("kind", ["string", "large_binary"])
@pytest.mark.parametrize("length", [1, 3, 4, 8, 12, 16, 48, "mixed", "null"])
def test_string_keys_of_one_length_and_others(length, kind):
    rng = np.random.default_rng(9)
    n = length if isinstance(length, int) else 8
    alphabet = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz", dtype=np.uint8)

    def keys(rows):
        out = [bytes(rng.choice(alphabet, n)) for _ in range(max(2, rows // 3))]
        if length == "mixed":
            out[0] = out[0][:5]
        picked = [out[i] for i in rng.integers(0, len(out), rows)]
        if length == "mixed":
            picked[3] = out[0]
        if length == "null":
            picked[3] = None
        return pa.array([None if k is None else k.decode() if kind == "string" else k for k in picked],
                        type=pa.string() if kind == "string" else pa.large_binary())

    js = pa.array(rng.integers(0, 20, 300) << 30)
    a = pa.record_batch([keys(300), js, pa.array(rng.standard_normal(300))], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(rng.integers(0, 20, 301) << 30), keys(301), pa.array(rng.standard_normal(301))],
                        names=["j", "k", "v"])
    got = K.fold(FOLD, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))
    want = oracle.fold(FOLD, a.schema, [a], b.schema, [b], None, oracle.schema(FOLD, [a.schema, b.schema]))
    g, w = pa.Table.from_batches(got.batches), pa.Table.from_batches(want.batches)
    for c in range(3):
        assert g.column(c).to_pylist() == w.column(c).to_pylist()
