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


@pytest.mark.parametrize("n,k,rows", [(4608, 260, 1280), (4608, 4608, 630), (512, 4096, 4160), (128, 16384, 700)])
def test_one_cta_for_all_groups_gives_the_bits_of_many(n, k, rows):
    """Eight rows a thread: tiles enough for one CTA to walk several groups (the first two), groups whose sums
    would take more room than is set aside (the third: 272 MB), and as many groups as there are (the last)."""
    t = ops()
    w, x = rnd((n, k), torch.float32, 1).cuda(), rnd((rows, k), torch.float32, 3).cuda()
    groups = lambda r: t.library().shiso_gemm_float_groups(x.data_ptr(), w.data_ptr(), x.data_ptr(), r, n, k, t._sm_count())
    full = t.linear(x, w, torch.float32)
    assert groups(64) >= 2 and groups(rows) == (128 if k == 16384 else 0)
    for a, part in ((0, 64), (5, 1), (100, 20), (300, 250)):
        assert torch.equal(t.linear(x[a : a + part].contiguous(), w, torch.float32), full[a : a + part]), (a, part)
