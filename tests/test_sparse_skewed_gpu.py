"""The sparse product of skewed keys: x with most of the pairs filled by a block of
their own, rows of one (z, y) walked side by side, both beside the ordinary
tiles: rows, bits and NULLs as the oracle's, and the same under a budget."""
import os
import subprocess
import sys

import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import kernels as K
from oracle import oracle
from tests.launched import kernels_of
from tests.tables import matmul_fold, rows_of
from tests.test_semantics_gpu import _budget_property, _fold_run

pytestmark = pytest.mark.gpu

FOLD = matmul_fold()
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _tables(nx, nz, ny, rows, sx, sz, sy, seed):
    rng = np.random.default_rng(seed)

    def keys(n, rows, s):
        pick = np.minimum(rng.zipf(s, rows) - 1, n - 1) if s else rng.integers(0, n, rows)
        return np.array([f"{v:012x}" for v in rng.choice(1 << 44, n, replace=False)]), pick

    (xs, xi), (zs, za), (ys, yi) = keys(nx, rows, sx), keys(nz, rows, sz), keys(ny, rows, sy)
    xi[:nx] = rng.permutation(nx)
    zb = keys(nz, rows, sz)[1]

    def values():
        v = rng.standard_normal(rows)
        v[::31] = np.inf
        v[7::53] = np.nan
        return pa.array(v, mask=rng.uniform(size=rows) < 0.2)

    a = pa.record_batch([pa.array(xs[xi]), pa.array(zs[za]), values()], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(zs[zb]), pa.array(ys[yi]), values()], names=["j", "k", "v"])
    return a, b


# x, z, y, rows, their Zipf exponents (0: uniform); whether some x have a block of
# their own, and whether runs of one (z, y) are gathered.
CASES = [(1300, 4, 600, 4000, 1.3, 1.3, 0, True, True), (1300, 4, 600, 4000, 0, 1.3, 1.3, False, True),
         (1300, 4, 600, 4000, 1.3, 1.3, 1.3, True, True), (700, 3, 3000, 3000, 1.5, 0, 0, True, False),
         (1300, 900, 600, 4000, 1.3, 0, 1.3, False, False), (2000, 50, 100, 3000, 2, 2, 2, True, True),
         (1300, 40, 5000, 6000, 0, 0, 0, False, False)]


@pytest.mark.parametrize("case", CASES, ids=str)
def test_skewed_keys_give_the_oracles_bits(case):
    *shape, heavy, gathered = case
    a, b = _tables(*shape, seed=len(CASES))

    def run():
        return K.fold(FOLD, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))

    names = kernels_of(run)
    assert names is None or any("gustavson<true>" in n for n in names) == heavy
    assert names is None or any("fill_tiles<true>" in n for n in names) == gathered
    got = run()
    assert got.algorithm == K.Algorithm.DISCRIMINATE
    want = oracle.fold(FOLD, a.schema, [a], b.schema, [b], None, oracle.schema(FOLD, [a.schema, b.schema]))
    g, w = pa.Table.from_batches(got.batches), pa.Table.from_batches(want.batches)
    assert g.num_rows == w.num_rows
    for c in range(2):
        assert g.column(c).equals(w.column(c))
    gv, wv = g.column(2).combine_chunks(), w.column(2).combine_chunks()
    assert gv.is_valid().equals(wv.is_valid()) and gv.null_count == wv.null_count
    x, y = (np.asarray(v.fill_null(0.0)) for v in (gv, wv))
    assert np.array_equal(np.isnan(x), np.isnan(y))
    assert np.array_equal(x[~np.isnan(x)].view(np.uint64), y[~np.isnan(y)].view(np.uint64))


def test_budgets_hold_with_heavy_x():
    a, b = _tables(*CASES[0][:7], seed=1)
    _budget_property(_fold_run(FOLD, a.schema, [a], b.schema, [b]))


SCRIPT = """
import sys
import pyarrow as pa
from einfold_b200 import kernels as K
from tests.test_sparse_skewed_gpu import CASES, FOLD, _tables
a, b = _tables(*CASES[0][:7], seed=1)
got = K.fold(FOLD, K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))
table = pa.Table.from_batches(got.batches).combine_chunks()
with pa.OSFile(sys.argv[1], "wb") as f, pa.ipc.new_file(f, table.schema) as w:
    w.write_table(table)
print(len(got.batches))
"""


def test_batches_of_groups_with_heavy_x(tmp_path):
    # (The groups a batch are read once per process.)
    tables = []
    for i, per_batch in enumerate(("", "20000")):
        path = str(tmp_path / f"{i}.arrow")
        env = dict(os.environ, **({"EINFOLD_GROUPS_PER_BATCH": per_batch} if per_batch else {}))
        r = subprocess.run([sys.executable, "-c", SCRIPT, path], env=env, capture_output=True, text=True, timeout=300, cwd=ROOT)
        assert r.returncode == 0, r.stderr[-4000:]
        assert (int(r.stdout.split()[-1]) > 1) == bool(per_batch)
        with pa.OSFile(path) as f:
            tables.append(pa.ipc.open_file(f).read_all().combine_chunks())
    (x, y) = tables
    assert x.column(0).equals(y.column(0)) and x.column(1).equals(y.column(1))
    assert x.column(2).null_count == y.column(2).null_count
    bits = [np.asarray(t.column(2).combine_chunks().fill_null(7.0)).view(np.uint64) for t in tables]
    assert np.array_equal(*bits)
