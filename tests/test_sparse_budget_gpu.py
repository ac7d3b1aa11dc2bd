"""What the sparse product asks of a budget: the run starts, counts and offsets of
its tiles where it goes by tiles, its accumulators where it doesn't, and no more
for the tiles than for the accumulators."""
import numpy as np
import pyarrow as pa
import pytest

from einfold_b200 import kernels as K
from tests.tables import matmul_fold, rows_of
from tests.test_semantics_gpu import Limit, _budget_property, _fold_run

pytestmark = pytest.mark.gpu

TILE = 512


class Ledger(Limit):
    def __init__(self):
        super().__init__(2 ** 62)
        self.asked = []

    def grow(self, nbytes):
        self.asked.append(nbytes)
        return super().grow(nbytes)


def _tables(nx, nz, ny, ra, rb):
    """Every key at least once, the z of both operands the same."""
    rng = np.random.default_rng(nx + ny)

    def keys(n, rows):
        names = np.array([f"{v:08x}" for v in rng.choice(1 << 32, n, replace=False)])
        return names, rng.permutation(np.concatenate([np.arange(n), rng.integers(0, n, rows - n)]))

    (xs, xi), (zs, zi), (ys, yi) = keys(nx, ra), keys(nz, ra), keys(ny, rb)
    zb = rng.permutation(np.concatenate([np.arange(nz), rng.integers(0, nz, rb - nz)]))
    a = pa.record_batch([pa.array(xs[xi]), pa.array(zs[zi]), pa.array(rng.standard_normal(ra))], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(zs[zb]), pa.array(ys[yi]), pa.array(rng.standard_normal(rb))], names=["j", "k", "v"])
    return a, b


# Tiles below and above their accumulators, too few items for tiles.
@pytest.mark.parametrize("nx,nz,ny,ra,rb,tiled", [(1500, 200, 700, 3000, 2000, True), (5000, 300, 5000, 9000, 9000, True),
                                                  (90_000, 90_000, 513, 100_000, 100_000, False),
                                                  (300, 200, 700, 1000, 2000, False)])
def test_asked_bytes(nx, nz, ny, ra, rb, tiled):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a, b = _tables(nx, nz, ny, ra, rb)
    run = _fold_run(matmul_fold(), a.schema, [a], b.schema, [b])
    ledger = Ledger()
    algorithm, got = run(ledger)
    assert algorithm == K.Algorithm.DISCRIMINATE
    words, n_tiles = (ny + 31) // 32, (ny + TILE - 1) // TILE
    count_blocks = min(nx, 4 * sms)
    blocks = min(count_blocks, max(sms, (64 << 20) // (ny * 8 + words * 8)))
    accumulators = blocks * ny * 8 + count_blocks * words * 8
    items = 4 * (nz * n_tiles + 1) + 12 * nx * n_tiles + 9 * nx + 8
    assert (nx * n_tiles >= 8 * sms and items <= accumulators) == tiled
    # Among the calls for the dense form's keys, the ranks and the groups.
    assert ((items if tiled else accumulators) in ledger.asked) and ((accumulators if tiled else items) not in ledger.asked)
    # Without a budget the tiles need no room of anyone: the same bits.
    free = K.fold(matmul_fold(), K.Relation(a.schema, [a]), K.Relation(b.schema, [b]))
    assert rows_of(free.batches).equals(got)
    _budget_property(run)
