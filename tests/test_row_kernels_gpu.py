"""Row kernels that choose among variants by size: every variant, its ragged ends and the hand-over to the general kernel."""

import pytest
import torch

import fake_kernels as ref
from test_kernels_gpu import close, make_step, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1032, 2048, 4096, 4104, 4608, 8448, 10240, 16384, 16392, 32768, 32776, 50008])
def test_polynorm_widths(width):
    """Pieces of eight a thread: 1, 2, 4, 5 and 8, with 128, 256 and 512 threads, and wider rows, read twice; rows off 16-byte
    boundaries take the general kernel, whose sums run in another order."""
    z, c = rnd((5, width + 8), torch.bfloat16, width), torch.tensor([0.7, -0.4, 0.2, 0.1])
    for first in (0, 1):  # (a column range that starts off a 16-byte boundary)
        view = z[:, first : first + width]
        got = ops().polynorm(z.cuda()[:, first : first + width], c.cuda(), 1e-5, torch.bfloat16)
        close(got, ref.polynorm(view.float(), c, 1e-5, torch.float32), torch.bfloat16, f"polynorm {width} from column {first}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("copies", [2, 3, 4])
@pytest.mark.parametrize("hidden", [512, 516, 1028, 2044, 2048, 2052])
def test_stream_copies_widths(hidden, copies, dtype):
    """Four columns a thread, one, two and four times, with a last one that is partly out of the row; three copies and wider
    rows take the general kernel.  A first read, a write into copies that stand, in place, and the sum that closes."""
    t, T = ops(), 5
    x, y1, y2 = rnd((T, hidden), torch.float32, 1), rnd((T, hidden), dtype, 2), rnd((T, hidden), dtype, 3)
    read, write = [rnd((copies,), torch.float32, s) for s in (4, 5, 6)], [rnd((copies,), torch.float32, s) for s in (7, 8)]
    mix, weight = [rnd((copies, copies), torch.float32, s) for s in (9, 10)], rnd((hidden,), torch.float32, 11)
    lanes = x.double()[None].repeat(copies, 1, 1)
    wants = []
    for step, y in enumerate((None, y1, y2)):
        if y is not None:
            lanes = torch.einsum("sr,std->rtd", mix[step - 1].double(), lanes) + write[step - 1].double()[:, None, None] * y.double()[None]
        u = torch.einsum("s,std->td", read[step].double(), lanes)
        wants.append(u * torch.rsqrt(u.pow(2).mean(-1, keepdim=True) + 1e-5) * weight.double())
    x, y1, y2, weight = x.cuda(), y1.cuda(), y2.cuda(), weight.cuda()
    read, write, mix = [a.cuda() for a in read], [a.cuda() for a in write], [a.cuda() for a in mix]
    none, first = t.hyper_mix_read(x, None, None, None, copies, read[0], weight, 1e-5, dtype)
    held, second = t.hyper_mix_read(x, y1, mix[0], write[0], copies, read[1], weight, 1e-5, dtype)
    total = t.hyper_mix_sum(held.clone(), y2, mix[1], write[1])
    same, third = t.hyper_mix_read(held, y2, mix[1], write[1], copies, read[2], weight, 1e-5, dtype)
    assert none is None and same.data_ptr() == held.data_ptr()
    for got, want, what in zip((first, second, third), wants, ("first read", "write and read", "in place")):
        close(got, want, dtype, f"{what} {copies} x {hidden}", rel32=4e-6)
    close(same, lanes, torch.float32, f"copies {copies} x {hidden}", rel32=4e-6)
    close(total, lanes.sum(0), torch.float32, f"sum {copies} x {hidden}", rel32=4e-6)


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
