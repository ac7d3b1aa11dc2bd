"""Attention of a few queries against many keys (the chunked FP64 kernel),
against torch float64 and, where values or guards send a call back, against
the same groups given as ragged ones of full length (which take the other
forms)."""
import pytest
import torch

from einfold_b200 import autograd as A
from einfold_b200.ir import Comparison
from einfold_b200.kernels import Precision, last_call
from tests.test_autograd_gpu import _reference

pytestmark = pytest.mark.gpu


def _inputs(b, lq, lk, d, dv, seed, sd=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    return r(b, lq, d) * sd, r(b, lk, d) * sd, r(b, lk, dv)


CASES = {
    # groups, queries, keys, d, dv, conditions
    "one_query": (3, 1, 8191, 64, 64, []),
    "least_keys": (2, 2, 512, 16, 5, []),
    "odd_widths": (2, 3, 1025, 7, 63, []),
    "wide": (2, 5, 700, 128, 128, []),
    "wide_odd": (1, 9, 640, 127, 101, A.window(600)),
    "two_row_blocks": (2, 17, 1000, 40, 64, []),
    "most_queries": (5, 32, 513, 64, 100, [(Comparison.GREATER_OR_EQUAL, -500)]),
    "rows_without_keys": (2, 20, 512, 64, 64, [(Comparison.GREATER_OR_EQUAL, 10)]),
}


@pytest.mark.parametrize("precision", [Precision.SPLIT, Precision.FP64])
@pytest.mark.parametrize("name", list(CASES))
def test_few_queries_match_torch_float64(name, precision):
    b, lq, lk, d, dv, cond = CASES[name]
    q, k, v = _inputs(b, lq, lk, d, dv, seed=len(name))
    scale = d ** -0.5
    out, lse = A.attention_forward(q, k, v, cond, scale, precision)
    assert last_call.product_ops == 0 and last_call.kernels_launched == 2
    want = _reference(q, k, v, cond, scale)
    seen = ~torch.isnan(want)
    assert torch.equal(seen, ~torch.isnan(out))
    # Both form d products a score (relative to Σ|q||k|), an exp and a sum over the keys.
    s_abs = (scale * (q.abs() @ k.abs().transpose(-1, -2))).max().item()
    tol = 4 * 2.0 ** -53 * (d * s_abs + lk) * v.abs().max().item()
    assert (out[seen] - want[seen]).abs().max().item() <= tol
    rows = seen.any(-1)
    x, j = torch.arange(lq, device="cuda")[:, None], torch.arange(lk, device="cuda")[None, :]
    allowed = torch.ones(lq, lk, dtype=torch.bool, device="cuda")
    for c, off in cond:
        allowed &= x >= j + off if c == Comparison.GREATER_OR_EQUAL else x <= j + off
    ref = torch.logsumexp((scale * (q @ k.transpose(-1, -2))).masked_fill(~allowed, float("-inf")), -1)
    assert (lse[rows] - ref[rows]).abs().max().item() <= 4 * 2.0 ** -53 * (d * s_abs + lk)


def _both(q, k, v, cond, scale, precision):
    def run(**lengths):
        try:
            return A.attention_forward(q, k, v, cond, scale, precision, **lengths)[0]
        except A.Declined:
            return None

    full = dict(q_lengths=[q.shape[1]] * q.shape[0], k_lengths=[k.shape[1]] * q.shape[0])
    return run(), run(**full)


@pytest.mark.parametrize("precision", [Precision.SPLIT, Precision.FP64])
@pytest.mark.parametrize("what", ["v_inf", "v_nan", "k_inf", "q_nan", "huge_scores", "v_tiny", "v_largest"])
def test_values_the_kernel_sends_back(what, precision):
    q, k, v = _inputs(2, 3, 600, 16, 8, seed=3)
    if what == "v_inf":
        v[1, 77, 3] = float("inf")
    elif what == "v_nan":
        v[0, 599, 0] = float("nan")
    elif what == "k_inf":
        k[0, 100, 5] = float("inf")
    elif what == "q_nan":
        q[1, 2, 0] = float("nan")
    elif what == "huge_scores":
        q *= 1e155
        k *= 1e155
    elif what == "v_tiny":
        v *= 1e-307
    else:
        v[0, 5, 1] = 1.7e308
        v[0, 6, 1] = 1.7e308
    got, want = _both(q, k, v, [], 0.25, precision)
    assert (got is None) == (want is None)
    if got is not None:
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        fin = torch.isfinite(want)
        assert torch.equal(got[~fin].nan_to_num(7.0), want[~fin].nan_to_num(7.0))
        if fin.any():
            scale = want[fin].abs().max().item()
            assert (got[fin] - want[fin]).abs().max().item() <= 1e-11 * scale
