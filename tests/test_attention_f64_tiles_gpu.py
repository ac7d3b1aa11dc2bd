"""Tiles of 16 or 32 keys in the FP64 forward, by the blocks an SM and whether
they are of one length, against torch float64."""
import pytest
import torch

from einfold_b200 import autograd as A
from einfold_b200.ir import Comparison
from einfold_b200.kernels import Precision
from tests.launched import kernels_of
from tests.test_attention_rows_gpu import _inputs
from tests.test_autograd_gpu import _reference

pytestmark = pytest.mark.gpu

CAUSAL = [(Comparison.GREATER_OR_EQUAL, 0)]


# Groups of one block of 64 rows (or of four, under a causal mask) on 148 SMs.
@pytest.mark.parametrize("w,l,cond,lengths,keys", [
    (296, 64, [], False, 32), (297, 64, [], False, 16), (444, 64, [], False, 16), (445, 64, [], False, 32),
    (592, 50, [], False, 32), (593, 64, [], False, 16), (592, 64, [], True, 16),
    (92, 200, CAUSAL, False, 32), (93, 256, CAUSAL, False, 16), (130, 256, CAUSAL, False, 16),
    (130, 256, A.window(40), False, 32)])
def test_tiles_by_blocks(w, l, cond, lengths, keys):
    d = 24
    q, k, v = _inputs(w, l, l, d, 10, seed=w)
    scale = d ** -0.5
    full = dict(q_lengths=[l] * w, k_lengths=[l] * w) if lengths else {}
    run = lambda: A.attention_forward(q, k, v, cond, scale, Precision.FP64, **full)  # noqa: E731
    seen = kernels_of(run)
    names = [name for name in seen or [] if "attn_fwd_f64" in name]
    out, _ = run()
    if seen is not None and torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert len(names) == 1 and f", {keys}, " in names[0]
    want = _reference(q, k, v, cond, scale)
    s_abs = (scale * (q.abs() @ k.abs().transpose(-1, -2))).max().item()
    # d products a score, an exp and a rescaled sum over the keys.
    tol = 4 * 2.0 ** -53 * (d * s_abs + l + l // 16) * v.abs().max().item()
    assert (out - want).abs().max().item() <= tol
