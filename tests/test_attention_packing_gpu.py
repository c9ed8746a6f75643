"""Prompt attention in tensor memory with all heads of a key head in a tile and with one: the bits of a row depend neither on that nor on
what it shares the step with."""

import pytest
import torch

from test_kernels_gpu import close, make_step, ops, ref, rnd

pytestmark = pytest.mark.gpu


def step_of(q_lens, starts, page, pages):
    cpu, gpu, table = make_step(q_lens, starts, page, pages, 9)
    gpu.h_q_start, gpu.max_q_len, gpu.all_decode = cpu.q_start.tolist(), max(q_lens), False
    cpu.max_q_len = max(q_lens)
    return cpu, gpu, table


def test_tiles_hold_a_group_while_they_have_two_tokens():
    tile = ops().library().shiso_prefill_attention_tc_tile
    # heads of a key head: none shared, tiles of 32, 25, three and two tokens, more than half a tile
    assert [tile(g, 1) for g in (1, 4, 5, 42, 43, 64, 65, 128, 129)] == [128, 32, 25, 3, 2, 2, 128, 128, 128]
    assert tile(32, 8) == 32 and tile(7, 2) == 128


@pytest.mark.parametrize("heads,kv_heads", [(8, 2), (40, 1), (63, 1), (96, 1), (6, 6)])
@pytest.mark.parametrize("window,keep", [(0, 0), (100, 0), (100, 5)])
def test_a_portion_has_the_same_bits_packed_or_not_alone_or_beside_decoding_requests(heads, kv_heads, window, keep):
    t, page, d = ops(), 16, 64
    q_lens, starts = [330, 1, 1, 1, 1], [70, 300, 0, 63, 64]
    pages = sum(-(-(s + n) // page) for s, n in zip(starts, q_lens)) + 2
    cpu, beside, table = step_of(q_lens, starts, page, pages)
    k, v = rnd((pages, page, kv_heads, d), torch.bfloat16, 1), rnd((pages, page, kv_heads, d), torch.bfloat16, 2)
    q = rnd((cpu.num_tokens, heads * d), torch.bfloat16, 3)
    _, alone, _ = step_of(q_lens[:1], starts[:1], page, pages)
    size = window or 1 << 30

    def run(rows, step, tables, keys, values):
        return t.masked_attention(rows.cuda(), heads, keys.cuda(), values.cuda(), tables.cuda().contiguous(), page, 0.125, "window", size, keep, step)

    together, single = run(q, beside, table, k, v), run(q[:330].contiguous(), alone, table[:1], k, v)
    spread = [x.repeat_interleave(heads // kv_heads, dim=2) for x in (k, v)]  # a key head for every query head: one head a tile
    unpacked = run(q, beside, table, *spread)
    t.check_kernel_status()
    assert torch.equal(together[:330], single) and torch.equal(together, unpacked)
    want = ref.masked_attention(q, heads, k, v, table, page, 0.125, "window", size, keep, cpu)
    close(together, want, torch.bfloat16, f"{heads} / {kv_heads} heads, window {window} + {keep}")
