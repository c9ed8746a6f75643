"""The float products in groups of K: every tile height, ragged rows, outputs and columns, groups with
CTAs of their own and groups that one CTA walks, and the property all of them share - a row's bits
depend neither on how many rows there are nor on where it lies."""

import pytest
import torch

from test_kernels_gpu import close, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(128, 128), (1024, 1024), (1000, 516), (33, 2308), (4608, 260), (130, 4)])
def test_float_products_and_their_rows(n, k):
    t = ops()
    w, bias = rnd((n, k), torch.float32, 1), rnd((n,), torch.float32, 2)
    x = rnd((1300, k), torch.float32, 3)
    want = x.double() @ w.double().T
    full = t.linear(x.cuda(), w.cuda(), torch.float32)
    # (rounding of a sum of k products: at most k 2^-24 of the sum of their magnitudes, and about the root of k of
    # it where signs are random; one float unit of the largest result per 64 columns stands far above that)
    close(full, want, torch.float32, f"float product {n} x {k}", rel32=1e-6 * (1 + k / 64) ** 0.5 * 4)
    simple = t.linear_simple(x.cuda(), w.cuda(), torch.float32)
    assert (full.cpu().double() - want).norm() <= 1.05 * (simple.cpu().double() - want).norm()  # no less exact than one long chain
    for a, rows in ((5, 1), (0, 8), (31, 9), (64, 32), (700, 33), (3, 96), (100, 300), (1299, 1)):
        part = t.linear(x[a : a + rows].contiguous().cuda(), w.cuda(), torch.float32, bias.cuda())
        assert torch.equal(part, full[a : a + rows] + bias.cuda()), (n, k, a, rows)
