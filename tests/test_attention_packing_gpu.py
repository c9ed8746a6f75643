"""Prompt attention in tensor memory with one query head a tile and with all heads of a key head: which of the two runs
depends on the step's shape and changes no bit."""

import pytest
import torch

from test_kernels_gpu import close, make_step, ops, ref, rnd

pytestmark = pytest.mark.gpu


def step_of(q_lens, starts, page, pages):
    cpu, gpu, table = make_step(q_lens, starts, page, pages, 9)
    gpu.h_q_start, gpu.max_q_len, gpu.all_decode = cpu.q_start.tolist(), max(q_lens), False
    cpu.max_q_len = max(q_lens)
    return cpu, gpu, table


def test_tiles_hold_a_group_where_requests_decode_beside_a_portion():
    tile = ops().library().shiso_prefill_attention_tc_tile
    assert [tile(32, 8, t, s) for t, s in ((1088, 33), (1088, 9), (1088, 8), (2048, 1), (128, 1), (129, 1))] == [32, 32, 128, 128, 32, 128]
    # heads of a key head: none shared, tiles of 25, three and two tokens, more than half a tile
    assert [tile(g, 1, 64, 2) for g in (1, 5, 42, 43, 64, 65, 128, 129)] == [128, 25, 3, 2, 2, 128, 128, 128]
    assert tile(7, 2, 64, 2) == 128


@pytest.mark.parametrize("heads,kv_heads", [(8, 2), (40, 1), (63, 1), (96, 1), (6, 6)])
@pytest.mark.parametrize("window,keep", [(0, 0), (100, 0), (100, 5)])
def test_a_portion_has_the_same_bits_alone_and_beside_decoding_requests(heads, kv_heads, window, keep):
    t, page, d = ops(), 16, 64
    q_lens, starts = [330, 1, 1, 1, 1], [70, 300, 0, 63, 64]
    pages = sum(-(-(s + n) // page) for s, n in zip(starts, q_lens)) + 2
    cpu, beside, table = step_of(q_lens, starts, page, pages)
    k, v = rnd((pages, page, kv_heads, d), torch.bfloat16, 1), rnd((pages, page, kv_heads, d), torch.bfloat16, 2)
    q = rnd((cpu.num_tokens, heads * d), torch.bfloat16, 3)
    _, alone, _ = step_of(q_lens[:1], starts[:1], page, pages)
    args = (k.cuda(), v.cuda())
    size = window or 1 << 30

    def run(rows, step, tables):
        return t.masked_attention(rows.cuda(), heads, *args, tables.cuda().contiguous(), page, 0.125, "window", size, keep, step)

    together, single = run(q, beside, table), run(q[:330].contiguous(), alone, table[:1])
    t.check_kernel_status()
    assert torch.equal(together[:330], single)
    want = ref.masked_attention(q, heads, k, v, table, page, 0.125, "window", size, keep, cpu)
    close(together, want, torch.bfloat16, f"{heads} / {kv_heads} heads, window {window} + {keep}")
