"""A few queries against many keys: chunks that no row joins are left alone,
whatever they hold."""
import pytest
import torch

from einfold_b200 import autograd as A
from einfold_b200.ir import Comparison
from einfold_b200.kernels import Precision, last_call
from tests.test_attention_rows_gpu import _inputs
from tests.test_autograd_gpu import _reference

pytestmark = pytest.mark.gpu

GE, LE = Comparison.GREATER_OR_EQUAL, Comparison.LESS_OR_EQUAL
# Keys 1,400 to 1,600 after the query's position.
MIDDLE = [(GE, -1600), (LE, -1400)]


@pytest.mark.parametrize("precision", [Precision.SPLIT, Precision.FP64])
@pytest.mark.parametrize("lq,d,dv", [(1, 64, 64), (5, 16, 3), (17, 128, 128), (32, 40, 100)])
def test_chunks_that_no_row_joins_are_left_alone(lq, d, dv, precision):
    q, k, v = _inputs(3, lq, 3000, d, dv, seed=lq)
    scale = d ** -0.5
    want = _reference(q, k, v, MIDDLE, scale)
    # Chunks of 128 keys: 1,400 .. 1,631 lie in 1,280 .. 1,663.
    for t in (k, v):
        t[:, :1280], t[:, 1664:] = float("nan"), float("inf")
    out, lse = A.attention_forward(q, k, v, MIDDLE, scale, precision)
    assert last_call.kernels_launched == 2
    assert torch.isfinite(lse).all()
    s_abs = (scale * (q.abs() @ k[:, 1280:1664].abs().transpose(-1, -2))).max().item()
    tol = 4 * 2.0 ** -53 * (d * s_abs + 201) * v[:, 1280:1664].abs().max().item()
    assert (out - want).abs().max().item() <= tol


def test_rows_of_two_blocks_with_chunks_of_their_own():
    # The second block of 16 rows joins a chunk that the first doesn't, whose values
    # are tiny or large beside the others'.
    q, k, v = _inputs(2, 32, 600, 8, 4, seed=9)
    cond = [(GE, -111), (LE, -90)]  # keys x + 90 .. x + 111: 128 and beyond from row 17 on
    v[:, 128:] *= 1e150
    out, _ = A.attention_forward(q, k, v, cond, 0.5, Precision.SPLIT)
    assert last_call.kernels_launched == 2
    want = _reference(q, k, v, cond, 0.5)
    assert ((out - want).abs() <= 1e-13 * want.abs().amax(-1, keepdim=True) * 20).all()
