"""Which form a few queries against many keys take (chunks of the keys, the FP64
tensor pipe or the split form, by groups, queries, joined keys and widths), and
chunks that no row joins, which are left alone whatever they hold."""
import numpy as np
import pytest
import torch

from einfold_b200 import autograd as A, kernels as K
from einfold_b200.ir import Comparison
from einfold_b200.kernels import Precision, last_call
from tests import pipelines as P
from tests.launched import kernels_of
from tests.tables import rows_of
from tests.test_attention_rows_gpu import _inputs
from tests.test_autograd_gpu import _reference

pytestmark = pytest.mark.gpu

GE, LE = Comparison.GREATER_OR_EQUAL, Comparison.LESS_OR_EQUAL
# Keys 1,400 to 1,600 after the query's position.
MIDDLE = [(GE, -1600), (LE, -1400)]


def _kernels(f):
    f()
    seen = kernels_of(f)
    forms = ("attn_rows", "attn_fwd_f64", "attn_fwd_split")
    return f(), None if seen is None else {n for n in forms if any(n in name for name in seen)}


# Groups, queries, keys, width, conditions; the kernel in split precision.
@pytest.mark.parametrize("w,lq,lk,d,cond,kernel", [
    (1200, 8, 512, 16, [], "attn_rows"), (1184, 16, 512, 16, [], "attn_rows"), (1185, 9, 512, 16, [], "attn_fwd_f64"),
    (1200, 16, 512, 17, [], "attn_rows"), (100, 32, 600, 16, [], "attn_rows"), (333, 17, 700, 64, [], "attn_rows"),
    (334, 17, 700, 64, [], "attn_fwd_f64"), (166, 20, 1100, 64, [], "attn_rows"), (167, 20, 1100, 64, [], "attn_fwd_f64"),
    (110, 20, 1100, 32, [], "attn_fwd_f64"), (167, 20, 1100, 64, [(GE, 0)], "attn_rows"),
    (148, 17, 1025, 65, [], "attn_fwd_split"), (149, 17, 1025, 65, [], "attn_rows"), (334, 32, 512, 65, [], "attn_fwd_split"),
    (320, 32, 513, 16, [], "attn_fwd_f64"), (310, 32, 512, 16, [], "attn_rows"), (334, 32, 512, 64, [(GE, 0)], "attn_fwd_f64")])
def test_the_form_by_shape(w, lq, lk, d, cond, kernel):
    q, k, v = _inputs(w, lq, lk, d, d, seed=w + lq)
    scale = d ** -0.5
    (out, _), names = _kernels(lambda: A.attention_forward(q, k, v, cond, scale, Precision.SPLIT))
    assert names in (None, {kernel})
    (fp64, _), names = _kernels(lambda: A.attention_forward(q, k, v, cond, scale, Precision.FP64))
    assert names in (None, {kernel if kernel == "attn_rows" else "attn_fwd_f64"})
    want = _reference(q, k, v, cond, scale)
    s_abs = (scale * (q.abs() @ k.abs().transpose(-1, -2))).max().item()
    # d products a score, an exp and a sum over the keys; the split form's digits: a
    # few parts in 2^44 of the same.
    tol = 4 * 2.0 ** -53 * (d * s_abs + lk) * v.abs().max().item()
    assert (fp64 - want).abs().max().item() <= tol
    assert (out - want).abs().max().item() <= (2.0 ** 9 * tol if kernel == "attn_fwd_split" else tol)


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


@pytest.mark.parametrize("nb,slices", [(340, 0), (340, 6), (20, 0)])
def test_a_pipelines_few_queries(nb, slices):
    normal = lambda seed: lambda n: np.random.default_rng(seed).standard_normal(n)  # noqa: E731
    case = P.attention(18, d=3, nb=nb, lk=512, q_value=normal(1), k_value=normal(2), v_value=normal(3))

    def run(precision, slices=0):
        got = K.pipeline(case.pipeline, [K.Relation(*case.q), K.Relation(*case.k), K.Relation(*case.v)],
                         options=K.Options(precision=precision, slices=slices))
        t = rows_of(got.batches)
        return t.column(t.num_columns - 1).to_numpy(zero_copy_only=False), last_call.product_ops

    (got, ops), (want, _) = run(K.Precision.SPLIT, slices), run(K.Precision.FP64)
    assert (ops > 0) == (slices > 0)
    assert np.max(np.abs(got - want)) <= 1e-12 * case.v_scale
