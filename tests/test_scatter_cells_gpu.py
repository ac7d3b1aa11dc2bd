"""The placement of rows in dense matrices: tables in key order (a warp's rows on
consecutive cells, at every offset within a word), shuffled ones, NULL values
and repeated rows, over two to five keys, against the oracle's dense fold."""
import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import ir, kernels as K
from oracle import oracle

pytestmark = pytest.mark.gpu

E = ir.EQ


def _table(names, extents, seed, order, null_at=None, drop=0, repeat=False):
    rng = np.random.default_rng(seed)
    keys = np.indices(extents).reshape(len(extents), -1)
    n = keys.shape[1]
    rows = np.arange(n) if order == "sorted" else rng.permutation(n)
    rows = rows[drop:]
    if repeat:  # the last row a second time, in place of the first
        rows = np.concatenate([rows[1:], rows[-1:]])
    v = rng.uniform(-1, 1, n)
    mask = np.zeros(len(rows), dtype=bool)
    if null_at is not None:
        mask[null_at % len(rows)] = True
    cols = [pa.array(k[rows]) for k in keys] + [pa.array(v[rows], mask=mask)]
    return pa.record_batch(cols, names=list(names) + ["v"])


def _fold(nx, nz, ny):
    """SUM(a.v * b.v) over nz summed dimensions, nx of a's and ny of b's kept."""
    x, z, y = range(nx), range(nx, nx + nz), range(nx + nz, nx + nz + ny)
    a = ir.Operand([(d, i) for i, d in enumerate([*x, *z])], nx + nz)
    b = ir.Operand([(d, i) for i, d in enumerate([*z, *y])], nz + ny)
    return ir.Fold([E] * (nx + nz + ny), [a, b], [ir.Output(d) for d in [*x, *y]])


CASES = {
    # kept extents of a, summed extents, kept extents of b
    "two_keys": ([37], [53], [41]),
    "one_word_rows": ([64], [16], [32]),
    "three_keys": ([5, 7], [19], [3, 11]),
    "four_keys": ([3, 5], [7, 2], [4, 9]),
    "five_keys": ([2, 3], [5, 2, 3], [3, 7]),
    "one_row": ([1], [1], [1]),
}


@pytest.mark.parametrize("order", ["sorted", "shuffled"])
@pytest.mark.parametrize("kind", ["complete", "missing", "null_a", "repeat_a", "repeat_b"])
@pytest.mark.parametrize("name", list(CASES))
def test_placement_matches_the_oracle(name, kind, order):
    xe, ze, ye = CASES[name]
    if name == "one_row" and kind != "complete":
        pytest.skip("a single row has no other to miss or repeat")
    f = _fold(len(xe), len(ze), len(ye))
    names = [f"k{i}" for i in range(5)]
    a = _table(names[:len(xe) + len(ze)], xe + ze, 1, order, 5 if kind == "null_a" else None,
               9 if kind == "missing" else 0, kind == "repeat_a")
    b = _table(names[:len(ze) + len(ye)], ze + ye, 2, order, repeat=kind == "repeat_b")
    got = K.fold_dense(f, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]),
                       options=K.Options(precision=K.Precision.FP64))
    want = oracle.dense_fold(f, [a], [b], None, oracle.schema(f, [a.schema, b.schema]), oracle.Options())
    assert (got is None) == (want is None) == kind.startswith("repeat")
    if got is not None:
        g, w = pa.Table.from_batches(got), pa.Table.from_batches(want.batches if hasattr(want, "batches") else want)
        assert g.num_rows == w.num_rows
        for i in range(g.num_columns):
            assert g.column(i).to_pylist() == w.column(i).to_pylist()
