"""Result key strings of one length: from a table of the ranks' strings where the
rows outnumber the ranks four to one (and the table is no larger than 16 bytes a
row), row by row where they don't; the rows either way."""
import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import kernels as K
from tests.launched import kernels_of
from tests.tables import matmul_fold

pytestmark = pytest.mark.gpu


# Ranks a side, x and k a shared j (its groups: per·per), bytes a key, tables built.
@pytest.mark.parametrize("ranks,shared,per,width,tables", [
    (3000, 750, 4, 16, 2), (3001, 750, 4, 16, 0), (3000, 40, 1, 16, 0), (600, 60, 10, 40, 2), (600, 60, 10, 161, 0),
    (600, 60, 10, 160, 2), (600, 60, 10, 3, 2), (5000, 0, 1, 16, 0)])
def test_tables_only_where_rows_outnumber_ranks(ranks, shared, per, width, tables):
    rng = np.random.default_rng(ranks + width)
    n = shared * per  # the rows of either side that join

    def side(base):
        names = np.array([f"{v:0{width}x}" for v in rng.choice(1 << (4 * min(width, 10)), ranks, replace=False)])
        j = base + np.arange(ranks)
        j[:n] = np.arange(n) // per
        order = rng.permutation(ranks)
        return names[order], j[order], rng.standard_normal(ranks)

    (x, ja, va), (y, jb, vb) = side(10 ** 6), side(2 * 10 ** 6)
    a = pa.record_batch([pa.array(x), pa.array(ja), pa.array(va)], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(jb), pa.array(y), pa.array(vb)], names=["j", "k", "v"])

    def run():
        return K.fold(matmul_fold(), K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))

    seen = kernels_of(run)
    assert seen is None or sum("rank_table" in name for name in seen) == tables
    got = run()
    assert got.algorithm == K.Algorithm.DISCRIMINATE
    t = pa.Table.from_batches(got.batches) if got.batches else None
    by_j = {}
    for k, j, v in zip(y, jb, vb):
        by_j.setdefault(j, []).append((k, v))
    want = sorted((i, k, va_ * v) for i, j, va_ in zip(x, ja, va) for k, v in by_j.get(j, ()))
    rows = 0 if t is None else t.num_rows
    assert rows == len(want) == shared * per * per
    if rows:
        assert t.column(0).to_pylist() == [w[0] for w in want]
        assert t.column(1).to_pylist() == [w[1] for w in want]
        assert np.array_equal(t.column(2).to_numpy(), np.array([w[2] for w in want]))
