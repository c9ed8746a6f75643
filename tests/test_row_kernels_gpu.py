"""Row kernels that choose among variants by size: every variant, its ragged ends and the hand-over to the general kernel."""

import pytest
import torch

import fake_kernels as ref
from test_kernels_gpu import close, make_step, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("pool", [1, 3, 16, 17, 32, 33, 64])
def test_pooled_blocks(pool, dtype):
    """Blocks on either side of the rows a CTA looks through and of the positions it asks for together, ends in neighbouring rows."""
    q_lens, starts, page, kv_heads, dim, vdim = [70, 1, 1, 40], [0, pool - 1, 2 * pool - 1, 130], 8, 2, 24, 40
    pages = sum(-(-(s + n) // page) for s, n in zip(starts, q_lens)) + 3
    cpu, gpu, table = make_step(q_lens, starts, page, pages, 7)
    k, v = rnd((pages, page, kv_heads, dim), dtype, 1), rnd((pages, page, kv_heads, vdim), dtype, 2)
    pk, pv = torch.zeros(pages, page, kv_heads, dim), torch.zeros(pages, page, kv_heads, vdim)
    got_k, got_v = pk.cuda(), pv.cuda()
    ref.pool_kv(k, v, table, pk, pv, table, page, pool, cpu)
    ops().pool_kv(k.cuda(), v.cuda(), table.cuda(), got_k, got_v, table.cuda(), page, pool, gpu)
    # (a sum of `pool` numbers of about one, added one after the other: pool 2^-24 of the sum of their magnitudes at most, per block of `pool`)
    close(got_k, pk, torch.float32, f"pooled keys {pool}", rel32=2e-6)
    close(got_v, pv, torch.float32, f"pooled values {pool}", rel32=2e-6)
    assert (pk != 0).any()
