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


@pytest.mark.parametrize("kind", ["int8", "uint8", "int16", "uint16", "int32", "uint32", "int64", "uint64"])
@pytest.mark.parametrize("slice_at", [0, 1])
def test_key_columns_of_every_width_and_alignment(kind, slice_at):
    # 3 x 1000 and 1000 x 3 rows a table (more than one block of keys, a ragged
    # last one), columns starting at an odd element where sliced.
    import torch

    i, j = np.indices((3, 1000 if kind not in ("int8", "uint8") else 100)).reshape(2, -1)
    n = len(i)
    v = np.random.default_rng(3).uniform(-1, 1, n)

    def device(x, dtype):
        t = torch.zeros(n + 1, dtype=dtype, device="cuda")
        t[slice_at:slice_at + n] = torch.from_numpy(np.ascontiguousarray(x)).to("cuda").to(dtype)
        return t[slice_at:slice_at + n]

    dt = getattr(torch, kind)
    schema = pa.schema([("i", getattr(pa, kind)()), ("j", getattr(pa, kind)()), ("v", pa.float64())])
    a = K.DeviceRelation(schema, [device(i, dt), device(j, dt), device(v, torch.float64)])
    b = K.DeviceRelation(schema, [device(j, dt), device(i, dt), device(v, torch.float64)])
    got = K.fold_dense(_fold(1, 1, 1), a, b, options=K.Options(precision=K.Precision.FP64))
    t = pa.Table.from_batches(got)
    m = v.reshape(3, -1)
    assert t.num_rows == 9
    assert np.max(np.abs(t.column(2).to_numpy() - (m @ m.T).reshape(-1))) <= 1000 * 2.0 ** -53 * np.max(
        np.abs(m) @ np.abs(m).T)
    assert t.column(0).to_pylist() == [x for x in range(3) for _ in range(3)]


@pytest.mark.parametrize("bad", [-1, 2 ** 63])
def test_keys_that_are_no_positions_decline(bad):
    n = 5000
    col = pa.array([*range(n - 1), bad], type=pa.uint64() if bad > 0 else pa.int64())
    t = pa.record_batch([col, pa.array(np.zeros(n, np.int64)), pa.array(np.ones(n))], names=["i", "j", "v"])
    u = pa.record_batch([pa.array(np.zeros(1, np.int64)), pa.array(np.zeros(1, np.int64)), pa.array(np.ones(1))],
                        names=["j", "k", "v"])
    assert K.fold_dense(_fold(1, 1, 1), K.Relation(t.schema, [t]), K.Relation(u.schema, [u])) is None
