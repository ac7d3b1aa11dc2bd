"""The split attention's operands prepared in one reading each (row digits,
column digits, exponent ranges, value statistics, D): at the edges of the
64-row chunks, of the lanes' four columns and of the 64 and 128 columns the
digits hold, ragged or not; operands whose powers of two leave the normal
range, and ones that aren't finite, through the same calls (the tile kernels
launched before the host knows). Against plain FP64 softmax attention."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    # lq, lk, d, dv, batches
    (1, 1, 1, 1, 1),
    (63, 65, 7, 3, 2),
    (64, 64, 64, 64, 3),
    (129, 127, 33, 62, 2),
    (200, 130, 65, 64, 1),
    (66, 200, 128, 130, 2),
    (300, 300, 6, 65, 2),
]


def _reference(torch, q, k, v, g, scale, ql, kl):
    lq, lk = q.shape[1], k.shape[1]
    dev = q.device
    i, j = torch.arange(lq, device=dev)[:, None], torch.arange(lk, device=dev)[None]
    ok = (i >= j)[None] & (i[None] < ql[:, None, None]) & (j[None] < kl[:, None, None])
    s = (q @ k.transpose(1, 2)) * scale
    s = torch.where(ok, s, -torch.inf)
    m = s.max(-1, keepdim=True).values
    p = torch.where(ok, torch.exp(s - torch.where(torch.isinf(m), 0.0, m)), 0.0)
    z = p.sum(-1, keepdim=True)
    w = torch.where(z > 0, p / z, 0.0)
    out = w @ v
    dead = (z == 0).squeeze(-1)
    d = (g * out).sum(-1, keepdim=True)
    ds = w * (g @ v.transpose(1, 2) - d)
    return out, dead, scale * ds @ k, scale * ds.transpose(1, 2) @ q, w.transpose(1, 2) @ g


def _bounds(q, k, v, g, scale):
    # Six digits keep a product of two rows to n·2^(3-48) of their largest
    # magnitudes. A score's error turns into a relative one of the weights
    # (twice: numerator and sum); FP64 sums add n·2^-53, far below.
    u = 2.0 ** -45
    (lq, d), (lk, dv) = q.shape[1:], v.shape[1:]
    mq, mk, mv, mg = (float(x.abs().max()) for x in (q, k, v, g))
    weight = 2 * (d + 1) * u * abs(scale) * mq * mk + 64 * 2.0 ** -53
    dp = dv * mg * mv
    ds = 2 * dp * (weight + u)  # of a weight's share of dS
    out = mv * (weight + lk * u)
    dq = abs(scale) * mk * (ds + 2 * dp * lk * u)
    dk = abs(scale) * mq * lq * (ds + 2 * dp * u)
    return out, dq, dk, mg * lq * (weight + u)


@pytest.mark.parametrize("ragged", [False, True])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_prepared_operands(shape, ragged):
    import torch

    from einfold_b200 import autograd as A
    from einfold_b200.kernels import Precision

    lq, lk, d, dv, batches = shape
    gen = torch.Generator(device="cuda").manual_seed(lq * 1000 + d)

    def normal(n, c, sd):
        return torch.randn(batches, n, c, dtype=torch.float64, device="cuda", generator=gen) * sd

    q, k, v, g = normal(lq, d, 0.5), normal(lk, d, 0.5), normal(lk, dv, 1.0), normal(lq, dv, 1.0)
    full = torch.tensor([lq] * batches, device="cuda"), torch.tensor([lk] * batches, device="cuda")
    ql, kl = full
    if ragged:
        ql = torch.tensor([(lq, max(lq // 2, 1), 1)[w % 3] for w in range(batches)], device="cuda")
        kl = torch.tensor([(max(lk - 1, 1), lk, 0)[w % 3] for w in range(batches)], device="cuda")
    lengths = dict(q_lengths=ql, k_lengths=kl) if ragged else {}
    conditions = A.causal()

    def run(q, k, v, g, scale, precision=Precision.SPLIT):
        out, lse = A.attention_forward(q, k, v, conditions, scale, precision, **lengths)
        if ragged:  # rows without keys are NaN; their D must not spread
            out = torch.nan_to_num(out, nan=0.0)
            g = torch.where(torch.arange(lq, device="cuda")[None, :, None] < ql[:, None, None], g, 0.0)
        return (out, lse) + A.attention_backward(q, k, v, out, lse, g, conditions, scale, precision, **lengths)

    def check(got, q, k, v, g, scale):
        if ragged:
            g = torch.where(torch.arange(lq, device="cuda")[None, :, None] < ql[:, None, None], g, 0.0)
        want = _reference(torch, q, k, v, g, scale, ql, kl)
        out = torch.where(want[1][..., None], 0.0, torch.nan_to_num(got[0], nan=0.0))
        for a, b, bound in zip((out,) + got[2:], (want[0],) + want[2:], _bounds(q, k, v, g, scale)):
            assert float((a - b).abs().max()) <= bound

    first = run(q, k, v, g, 0.7)
    check(first, q, k, v, g, 0.7)
    again = run(q, k, v, g, 0.7)  # its schedule known: launched before the host knows the ranges
    for a, b in zip(first, again):
        assert np.array_equal(a.cpu().numpy().view(np.uint64), b.cpu().numpy().view(np.uint64))
    # Powers of two below the normal range: the same scores by a large scale,
    # and v·d_out below it too.
    t = 2.0 ** -520
    check(run(q * t, k * t, v, g, 0.7 * 2.0 ** 1000), q * t, k * t, v, g, 0.7 * 2.0 ** 1000)
    # One value that isn't finite: what the FP64 form gives.
    for n, x in enumerate((q, k, v, g)):
        y = [q, k, v, g]
        y[n] = x.clone()
        y[n][0, 0, 0] = float("nan")
        got, want = run(*y, 0.7), run(*y, 0.7, Precision.FP64)
        clean = _bounds(q, k, v, g, 0.7)
        for a, b, bound in zip((got[0],) + got[2:], (want[0],) + want[2:], clean):
            assert torch.equal(torch.isnan(a), torch.isnan(b))
            assert not torch.isnan(a - b).ne(torch.isnan(a)).any()
            assert float(torch.nan_to_num(a - b, nan=0.0).abs().max()) <= bound
    # Scores beyond the split form's reach: taken or refused as by the FP64 form.
    big = 2.0 ** 505

    def outcome(precision):
        try:
            return A.attention_forward(q * big, k * big, v, conditions, 1.0, precision, **lengths)[0].cpu().numpy()
        except Exception as e:
            return type(e).__name__

    a, b = outcome(Precision.SPLIT), outcome(Precision.FP64)
    assert type(a) is type(b) and (a == b if isinstance(a, str) else np.array_equal(a, b, equal_nan=True))
