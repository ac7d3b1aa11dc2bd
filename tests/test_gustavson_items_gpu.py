"""The sparse product's choice between tiles of 512 output columns (a warp an
(x, tile) item, one to four tiles a warp) and the form without, on both sides of
the number of items where it changes and of the tiles a warp takes: rows, bits
and NULLs as the oracle's."""
import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import ir, kernels as K
from oracle import oracle

pytestmark = pytest.mark.gpu

E = ir.EQ
FOLD = ir.Fold([E, E, E], [ir.Operand([(0, 0), (1, 1)], 2), ir.Operand([(1, 0), (2, 1)], 2)],
               [ir.Output(0), ir.Output(2)])


# x, y, z, rows of a and b: around 8 items an SM (1184 of 148), rows of a more and
# fewer than 32 an x, one tile and several, and enough items for two tiles a warp.
@pytest.mark.parametrize("ni,nk,nj,ra,rb", [(1100, 512, 9, 4000, 3000), (1200, 511, 9, 4000, 3000),
                                            (592, 513, 80, 30000, 9000), (591, 513, 80, 30000, 9000),
                                            (130, 5130, 60, 6000, 30000), (1500, 4700, 50, 6000, 9000)])
def test_few_and_many_items_give_the_oracles_bits(ni, nk, nj, ra, rb):
    rng = np.random.default_rng(ni + nk)

    def key(n, rows):
        pick = np.concatenate([np.arange(n), rng.integers(0, n, max(rows - n, 0))])[:max(rows, n)]
        return np.array([f"{v:016x}" for v in rng.choice(1 << 40, n, replace=False)])[rng.permutation(pick)]

    js = np.array([f"{v:016x}" for v in rng.choice(1 << 40, nj, replace=False)])

    def values(n):
        v = rng.standard_normal(n)
        v[::31] = np.inf
        v[7::53] = np.nan
        return pa.array(v, mask=rng.uniform(size=n) < 0.03)

    ak, bk = key(ni, ra), key(nk, rb)
    a = pa.record_batch([pa.array(ak), pa.array(js[rng.integers(0, nj, len(ak))]), values(len(ak))], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(js[rng.integers(0, nj, len(bk))]), pa.array(bk), values(len(bk))], names=["j", "k", "v"])
    got = K.fold(FOLD, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))
    want = oracle.fold(FOLD, a.schema, [a], b.schema, [b], None, oracle.schema(FOLD, [a.schema, b.schema]))
    assert got.algorithm == K.Algorithm.DISCRIMINATE
    g, w = pa.Table.from_batches(got.batches), pa.Table.from_batches(want.batches)
    assert g.num_rows == w.num_rows
    for c in range(2):
        assert g.column(c).equals(w.column(c))
    gv, wv = g.column(2).combine_chunks(), w.column(2).combine_chunks()
    assert gv.is_valid().equals(wv.is_valid())
    x, y = (np.asarray(v.fill_null(0.0)) for v in (gv, wv))
    assert np.array_equal(np.isnan(x), np.isnan(y))
    assert np.array_equal(x[~np.isnan(x)].view(np.uint64), y[~np.isnan(y)].view(np.uint64))
