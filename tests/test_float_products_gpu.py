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


@pytest.mark.parametrize("n,k,rows", [(64, 256, 1), (127, 264, 15), (129, 1032, 17), (300, 520, 65), (1024, 4608, 129), (4608, 1024, 257)])
def test_float_products_on_the_tensor_cores(n, k, rows):
    """Edges of the tiles of 128 outputs, 16 to 128 rows and 64 columns; operands of very different sizes.  The
    pieces' products lose 2^-22 of a product's magnitude at most and a chunk's five additions, which cut off, as much
    again: 2^-21 of the products' magnitudes, and less than the K roundings of a chain."""
    t = ops()
    w, x = rnd((n, k), torch.float32, 11), rnd((rows, k), torch.float32, 12)
    x = x * torch.exp2(torch.randint(-20, 20, (rows, 1), generator=torch.Generator().manual_seed(3)).float())
    w[:, ::7] *= 1e-6
    assert t.library().shiso_gemm_float_tc_supported(16, 16, 16, rows, n, k)
    got = t.linear(x.cuda(), w.cuda(), torch.float32).cpu().double()
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((got - want).abs() <= 2.0 ** -21 * size).all()
    chain = t.linear_simple(x.cuda(), w.cuda(), torch.float32).cpu().double()
    scale = want.norm(dim=1, keepdim=True)
    assert ((got - want) / scale).norm() <= 1.05 * ((chain - want) / scale).norm()  # no less exact than one long chain


@pytest.mark.parametrize("rows", [3, 200])
def test_float_products_that_are_not_finite(rows):
    """Infinities, NaN and overflow come out as from a chain of multiply-adds, and touch no other row."""
    t = ops()
    n, k = 256, 1024
    w, x = rnd((n, k), torch.float32, 13), rnd((rows, k), torch.float32, 14)
    clean = t.linear(x.cuda(), w.cuda(), torch.float32).cpu()
    w2, x2 = w.clone(), x.clone()
    w2[5, 70] = float("inf")
    w2[9] = w2[9].bfloat16().float()  # (its lower pieces are zeros)
    x2[1, 3], x2[2, 900] = float("-inf"), float("nan")
    x2[0, :2], w2[77, :2] = 1e30, 1e30
    got = t.linear(x2.cuda(), w2.cuda(), torch.float32).cpu()
    chain = t.linear_simple(x2.cuda(), w2.cuda(), torch.float32).cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(chain)) and torch.equal(torch.isinf(got), torch.isinf(chain))
    assert torch.equal(got[torch.isinf(got)], chain[torch.isinf(chain)])
    keep = torch.ones(n, dtype=torch.bool)
    keep[[5, 9, 77]] = False
    assert torch.equal(got[3:][:, keep], clean[3:][:, keep])


@pytest.mark.parametrize("k", [256, 1032, 4608])
def test_float_products_whose_errors_do_not_average_out(k):
    """Operands of one sign, and ones whose pieces leave as much as they can behind: most where they are rounded (1 + 2^-8 - 2^-17), and most
    where they would be cut off (1 + 2^-7 - 2^-23).  What is left out of a product is below 2^-24 of it, and the 24 instructions of
    a chunk cut off a unit of its sum at most in each of the last four, and of a 2^7th of it before: below 2^-21 of the result,
    with the chunk sums' own rounding, K / 64 2^-25 of it on average."""
    t = ops()
    n, rows = 128, 40
    w, x = rnd((n, k), torch.float32, 21).abs() + 0.1, rnd((rows, k), torch.float32, 22).abs() + 0.1
    w[3], x[5] = 1 + 2.0 ** -7 - 2.0 ** -23, 1 + 2.0 ** -7 - 2.0 ** -23
    w[4], x[6] = 1 + 2.0 ** -8 - 2.0 ** -17, -(1 + 2.0 ** -8 - 2.0 ** -17)
    for part in (x, x[:9]):  # rows in pieces ahead of the product, and split by its own CTAs
        got = t.linear(part.cuda().contiguous(), w.cuda(), torch.float32).cpu().double()
        want = part.double() @ w.double().T
        assert ((got - want) / want).abs().max() <= 2.0 ** -21 + k / 64 * 2.0 ** -25
        if k > 1000:
            chain = t.linear_simple(part.cuda().contiguous(), w.cuda(), torch.float32).cpu().double()
            assert (got - want).norm() <= 1.05 * (chain - want).norm()


def test_float_products_that_one_product_dominates():
    """One column beside zeros, and beside columns 2^-40 as large: below 2^-24 of the product is left out and less than two units
    cut off, 2^-22 together."""
    t = ops()
    n, k, rows = 192, 512, 24
    w, x = rnd((n, k), torch.float32, 23), torch.zeros(rows, k)
    x[:, 70] = rnd((rows,), torch.float32, 24)
    x[rows // 2 :, 1:64] = rnd((rows - rows // 2, 63), torch.float32, 25) * 2.0 ** -40
    got = t.linear(x.cuda(), w.cuda(), torch.float32).cpu().double()
    want = x.double() @ w.double().T
    large = want.abs() > 1e-3 * want.abs().max()  # (beside a tiny product the small columns are no longer small)
    assert (((got - want) / want).abs()[large] <= 2.0 ** -22).all()


@pytest.mark.parametrize("rows", [12, 24, 40])
def test_floats_that_are_infinite_as_bfloat16(rows):
    """Above 3.39e38 a float rounds up to an infinite bfloat16; beside infinities and NaN its results are formed again, and no other row is touched."""
    t = ops()
    n, k = 256, 1024
    w, x = rnd((n, k), torch.float32, 13), rnd((rows, k), torch.float32, 14)
    clean = t.linear(x.cuda(), w.cuda(), torch.float32).cpu()
    x2 = x.clone()
    x2[0] = 0.0
    x2[0, 5], x2[1, 3], x2[2, 900] = 3.4e38, float("-inf"), float("nan")
    w2 = w.clone()
    w2[5, 70], w2[6] = float("inf"), w2[6].clamp(-0.9, 0.9)
    got = t.linear(x2.cuda(), w2.cuda(), torch.float32).cpu()
    chain = t.linear_simple(x2.cuda(), w2.cuda(), torch.float32).cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(chain)) and torch.equal(torch.isinf(got), torch.isinf(chain))
    assert torch.equal(got[0, 6], chain[0, 6]) and torch.isfinite(got[0, 6])  # one product of a huge float and zeros: the chain's bits
    keep = torch.ones(n, dtype=torch.bool)
    keep[[5, 6]] = False
    assert rows > 4 and torch.equal(got[3:][:, keep], clean[3:][:, keep])


@pytest.mark.parametrize("n,k,rows", [(128, 16384, 20), (300, 4608, 130), (129, 1032, 17), (4608, 520, 65)])
def test_groups_with_ctas_of_their_own_have_the_bits_of_one_cta(n, k, rows):
    t = ops()
    lib, sums = t.library(), {}
    w, x, bias = rnd((n, k), torch.float32, 1).cuda(), rnd((rows, k), torch.float32, 3).cuda(), rnd((n,), torch.float32, 2).cuda()
    group = -(-lib.shiso_gemm_float_group_columns(n, k) // 64) * 64
    pieces = torch.empty(3, rows, k, dtype=torch.bfloat16, device="cuda")
    for split in (False, True):
        sums[split] = torch.empty(rows, n, device="cuda")
        partial = torch.empty(-(-k // group), rows, n, device="cuda")
        assert lib.shiso_gemm_float_tc(x.data_ptr(), w.data_ptr(), bias.data_ptr(), sums[split].data_ptr(), partial.data_ptr() if split else 0,
                                       pieces.data_ptr(), rows, n, k, group, torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(sums[False], sums[True]) and torch.equal(sums[True], t.linear(x, w, torch.float32, bias))


@pytest.mark.parametrize("n,k,rows", [(4608, 4612, 630), (512, 4100, 4600), (128, 16388, 700)])
def test_products_that_stay_with_the_multiply_adds(n, k, rows):
    """Columns of 4 modulo 8 are no whole bfloat16 words: groups that one CTA walks, groups whose sums would take more room than is set
    aside, and as many groups as there are, with the bits of the other form."""
    t = ops()
    w, x = rnd((n, k), torch.float32, 1).cuda(), rnd((rows, k), torch.float32, 3).cuda()
    assert not t.library().shiso_gemm_float_tc_supported(x.data_ptr(), w.data_ptr(), x.data_ptr(), rows, n, k)
    groups = lambda r: t.library().shiso_gemm_float_groups(x.data_ptr(), w.data_ptr(), x.data_ptr(), r, n, k, t._sm_count())
    full = t.linear(x, w, torch.float32)
    assert groups(64) >= 2 and (groups(rows) > 0) == (k == 16388)
    for a, part in ((0, 64), (5, 1), (100, 20), (300, 250)):
        assert torch.equal(t.linear(x[a : a + part].contiguous(), w, torch.float32), full[a : a + part]), (a, part)
