"""Rows of a split product between a warp's and a long row's: cut with as many
values held as they have, to the digits that the same rows padded with zeros to
a long row's get."""
import numpy as np
import pytest

from einfold_b200 import _lib
from tests.launched import kernels_of
from tests.test_gemm_gradients_gpu import _product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slices", [2, 6, 7])
@pytest.mark.parametrize("k,held", [(513, 1), (1000, 1), (1023, 1), (1024, 1), (1025, 2), (2047, 2), (2048, 2), (2049, 4),
                                    (4096, 4), (4097, 8), (8193, 8)])
def test_rows_keep_their_digits(k, held, slices):
    import torch

    lib, ctx = _lib.load(), _lib.context(0)
    gen = torch.Generator(device="cuda").manual_seed(k)
    a, b = (torch.randn(2, r, k, dtype=torch.float64, device="cuda", generator=gen) for r in (70, 33))
    a[:, ::7] *= 2.0 ** 40
    a[:, 5], b[:, 3, :k - 1] = 0.0, 0.0
    a[:, 9, k - 1] = 2.0 ** 300  # a row's largest value last
    product = lambda: _product(torch, lib, ctx, a, b, 1, slices)  # noqa: E731
    seen = kernels_of(product)
    names = [name for name in seen or [] if "row_digits" in name]
    got = product()
    assert seen is None or len(names) == 1 and f"{slices}, 256, {held}>" in names[0]
    long = 8256
    want = _product(torch, lib, ctx, *(torch.nn.functional.pad(x, (0, long - k)) for x in (a, b)), 1, slices)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want.cpu().numpy().view(np.uint64))
