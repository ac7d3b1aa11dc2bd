"""Split products' operands sliced by rows (half a warp, a warp or a block a row,
values held or read again) and by columns, and both gradients of a product in
one call: against einfold_split_gemm on transposed arrays, bit for bit, and
against FP64 within the digits' bound."""
import numpy as np
import pytest

from einfold_b200 import _lib

pytestmark = pytest.mark.gpu

# batches, m, n, k: each is a contraction of one of the products, across the
# slicers' limits (64, 128, 512 and 8192 values) and off the 16-byte alignment.
SHAPES = [(1, 1, 1, 1), (2, 63, 64, 65), (3, 127, 129, 128), (1, 511, 130, 513), (2, 40, 515, 200), (1, 5, 8195, 33),
          (1, 8200, 3, 7)]


def _product(torch, lib, ctx, a, b, transposed, slices):
    *_, m, k = a.shape
    n = b.shape[1] if transposed else b.shape[2]
    c = torch.empty(a.shape[0], m, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.einfold_split_gemm(ctx, a.data_ptr(), b.data_ptr(), c.data_ptr(), a.shape[0], m, n, k, transposed, slices,
                                  None) == _lib.OK
    return c


@pytest.mark.parametrize("slices", [2, 6, 7])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_gradients_are_the_two_products(shape, slices):
    import torch

    batches, m, n, k = shape
    lib, ctx = _lib.load(), _lib.context(0)
    gen = torch.Generator(device="cuda").manual_seed(m + 10 * n + 100 * k)
    a, b, g = (torch.randn(batches, *s, dtype=torch.float64, device="cuda", generator=gen) for s in ((m, k), (k, n), (m, n)))
    a[:, 0] *= 2.0 ** 40  # rows and columns under powers of two of their own
    g[..., -1] *= 2.0 ** -200
    d_a, d_b = torch.empty_like(a), torch.empty_like(b)
    torch.cuda.synchronize()

    def gradients(x, y):
        return lib.einfold_split_gemm_gradients(ctx, a.data_ptr(), b.data_ptr(), g.data_ptr(), x.data_ptr() if x is not None
                                                else None, y.data_ptr() if y is not None else None, batches, m, n, k, slices,
                                                None)

    assert gradients(d_a, d_b) == _lib.OK
    at = a.transpose(1, 2).contiguous()
    want_a, want_b = _product(torch, lib, ctx, g, b, 1, slices), _product(torch, lib, ctx, at, g, 0, slices)
    for x, y in ((d_a, want_a), (d_b, want_b)):
        assert np.array_equal(x.cpu().numpy().view(np.uint64), y.cpu().numpy().view(np.uint64))
    # Each alone.
    for i in range(2):
        only = torch.empty_like((a, b)[i])
        assert gradients(*((only, None), (None, only))[i]) == _lib.OK
        assert np.array_equal(only.cpu().numpy().view(np.uint64), (d_a, d_b)[i].cpu().numpy().view(np.uint64))
    # A product of S digits each keeps n·(S+1)·2^(2-8S) of its row's and column's
    # largest magnitudes (the dropped levels and the digits' rounding), FP64 n·2^-53.
    for x, left, right in ((d_a, g, b.transpose(1, 2)), (d_b, at, g)):
        count = left.shape[2]
        bound = left.abs().amax(2)[:, :, None] * right.abs().amax(1)[:, None, :] * count * \
            ((slices + 1) * 2.0 ** (2 - 8 * slices) + 2.0 ** -52)
        assert bool(((x - left @ right).abs() <= bound).all())
    # A value that isn't finite refuses the call.
    g[0, 0, 0] = float("inf")
    torch.cuda.synchronize()
    assert gradients(d_a, d_b) == _lib.INVALID


@pytest.mark.parametrize("shape", [(0, 3, 4, 5), (2, 0, 4, 5), (2, 3, 0, 5), (2, 3, 4, 0)])
def test_empty_extents_give_empty_or_zero_gradients(shape):
    import torch

    from einfold_b200 import autograd as A

    batches, m, n, k = shape
    a = torch.ones(batches, m, k, dtype=torch.float64, device="cuda", requires_grad=True)
    b = torch.ones(batches, k, n, dtype=torch.float64, device="cuda", requires_grad=True)
    d_a, d_b = torch.autograd.grad(A.matmul(a, b), (a, b), torch.ones(batches, m, n, dtype=torch.float64, device="cuda"))
    assert d_a.shape == a.shape and d_b.shape == b.shape
    assert not d_a.any() and not d_b.any()
