"""The split attention where scores are large and lie close together (a common
offset in the features, of which the softmax is independent): the weights are cut
to 46 bits after the shift by the row's largest score, so the shift has to be that
score and not a bound of it. Scores here are exact in the digits, so that only
the weights and values are rounded."""
import numpy as np
import pytest

from einfold_b200 import ir, kernels as K
from tests import pipelines as P
from tests.tables import rows_of

pytestmark = pytest.mark.gpu

GE, LT = ir.Comparison.GREATER_OR_EQUAL, ir.Comparison.LESS

# A weight keeps 46 bits (half a unit: 2^-47 of the largest), a value 46 or more
# under its column's largest (2^-46), the level scheme drops 5 products of two
# digits below 2^-63 of at most 2^-4 (5·2^-46), and the sums double it.
TOL = 2.0 ** -42


def _case(power, sign, d, keys, step):
    """q and k of 128 rows with q·k = sign·2^power + step·(j mod 5), exactly."""
    import torch

    rng = np.random.default_rng(power * 8 + d)
    # d is a power of two: the offset's d equal products are exact.
    q = np.full((2, 130, d), 1.0)
    scores = sign * 2.0 ** power + step * (np.arange(keys) % 5)
    k = np.repeat((scores / d)[None, :, None], d, axis=2).repeat(2, axis=0)
    v = rng.standard_normal((2, keys, 3))
    put = lambda x: torch.tensor(np.ascontiguousarray(x), device="cuda")
    return put(q), put(k), put(v)


def _exact(q, k, v, conditions):
    """The softmax and its average in FP64 (the scores' sums are exact)."""
    import torch

    s = q @ k.transpose(-1, -2)
    x, j = torch.arange(s.shape[-2], device=s.device)[:, None], torch.arange(s.shape[-1], device=s.device)[None]
    for c, off in conditions:
        s = s.masked_fill(~{GE: x >= j + off, LT: x < j + off}[c], -torch.inf)
    w = torch.softmax(s, -1)
    return w @ v, torch.logsumexp(s, -1), w


@pytest.mark.parametrize("conditions", [(), ((GE, 0),), ((GE, 0), (LT, 1))])
@pytest.mark.parametrize("d", [1, 64, 128])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("power", [0, 8, 10, 14, 17, 20, 24, 25, 27, 30, 36])
def test_rows_of_large_close_scores(power, sign, d, conditions):
    from einfold_b200 import autograd as A
    from einfold_b200.kernels import Precision

    for step in (0.0, 0.25):  # below 2^(46 - 2): exact in the digits
        q, k, v = _case(power, sign, d, 130, step)
        out, lse = A.attention_forward(q, k, v, conditions, 1.0, Precision.SPLIT)
        want, lse_want, w = _exact(q, k, v, conditions)
        assert float((out - want).abs().max()) <= TOL * float(v.abs().max()), (power, sign, step)
        assert float((lse - lse_want).abs().max()) <= 2.0 ** -50 * 2.0 ** power + TOL
        if d > 64 or power > 30:
            continue
        # The backward's weights exp(s - lse) carry lse's rounding.
        d_out = torch_like(out, 5)
        eps = 4 * 2.0 ** -52 * 2.0 ** power + TOL
        big = float(d_out.abs().max())
        dq, dk, dv = A.attention_backward(q, k, v, out, lse, d_out, conditions, 1.0, Precision.SPLIT)
        n = q.shape[-2]
        assert float((dv - w.transpose(-1, -2) @ d_out).abs().max()) <= 2 * n * eps * big
        dp = d_out @ v.transpose(-1, -2)
        ds = w * (dp - (w * dp).sum(-1, keepdim=True))
        unit = 8 * n * eps * 3 * big * float(v.abs().max())
        assert float((dk - ds.transpose(-1, -2) @ q).abs().max()) <= unit * float(q.abs().max())
        assert float((dq - ds @ k).abs().max()) <= unit * float(k.abs().max())


def torch_like(x, seed):
    import torch

    return torch.randn(x.shape, dtype=x.dtype, generator=torch.Generator().manual_seed(seed)).to(x.device)


@pytest.mark.parametrize("power", [40, 50, 60])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_rows_of_one_score(power, sign):
    from einfold_b200 import autograd as A
    from einfold_b200.kernels import Precision

    q, k, v = _case(power, sign, 64, 130, 0.0)
    out, _ = A.attention_forward(q, k, v, (), 1.0, Precision.SPLIT)
    assert float((out - v.mean(-2, keepdim=True)).abs().max()) <= TOL * float(v.abs().max())


@pytest.mark.parametrize("scale", [ir.Scale.one(), ir.Scale.times(2.0), ir.Scale.over(4.0)])
@pytest.mark.parametrize("value", [1e4, -3e3])
def test_a_pipelines_rows_of_one_score(value, scale):
    case = P.attention(64, d=1, nb=2, weight=ir.Weight.exp(scale), q_value=lambda n: np.full(n, 1e4),
                       k_value=lambda n: np.full(n, value), v_value=lambda n: np.arange(n) % 7 - 2.0)

    def run(precision, slices=0):
        got = K.pipeline(case.pipeline, [K.Relation(*case.q), K.Relation(*case.k), K.Relation(*case.v)],
                         options=K.Options(precision=precision, slices=slices))
        t = rows_of(got.batches)
        return t.column(t.num_columns - 1).to_numpy(zero_copy_only=False)

    split, fp64 = run(K.Precision.SPLIT, 6), run(K.Precision.FP64)
    assert np.max(np.abs(split - fp64)) <= TOL * case.v_scale


@pytest.mark.parametrize("offset", [0.0, 2.0 ** 20, -2.0 ** 24])
def test_spreads_beside_an_offset_are_taken_and_refused_as_in_fp64(offset):
    import torch

    from einfold_b200 import autograd as A
    from einfold_b200.kernels import Precision

    # The lightest weight of a row with an output of 0: 2^-1021 at least.
    edge = 1021.0 * np.log(2.0)
    for spread in (1.0, edge - 200.0, edge - 30.0, edge - 1e-3, edge + 1e-3, edge + 30.0):
        q = torch.ones((1, 40, 1), dtype=torch.float64, device="cuda")
        k = (offset + torch.linspace(0.0, -spread, 65, dtype=torch.float64, device="cuda"))[None, :, None].contiguous()
        v = torch.ones((1, 65, 3), dtype=torch.float64, device="cuda")
        v[:, :, 1] = 0.0

        def outcome(precision):
            try:
                return A.attention_forward(q, k, v, (), 1.0, precision)
            except A.Declined:
                return None

        a, b = outcome(Precision.SPLIT), outcome(Precision.FP64)
        assert (a is None) == (b is None), spread
        if a is not None:
            # A key's digits leave up to 2^-46 of the largest score.
            bound = 2.0 ** -44 * (abs(offset) + spread) + TOL
            assert float((a[0] - b[0]).abs().max()) <= bound
