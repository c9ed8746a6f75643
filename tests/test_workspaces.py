"""Rules on the host that no GPU is needed for: which steps the walk of long portions takes, and that what an
engine sets aside for a step covers the workspaces of its kernels."""

import json
from types import SimpleNamespace

import pytest
import torch

from shiso_llm_b200.cli import preset_path
from shiso_llm_b200.config import plan_from_document
from shiso_llm_b200.engine import core
from shiso_llm_b200.kernels.library import library

AT = 0x7F0000000000  # an address on every boundary; nothing is read there


def walk_takes(**change):
    a = dict(dtype=1, q=AT, k=AT, v=AT, q_ld=256, k_ld=256, v_ld=256, state=AT, stride=3 * 64 * 64, logits=0, logits_ld=0, rotary=64,
             tokens=300, seqs=3, dim=64, vdim=64)
    assert set(change) <= set(a)
    return library().shiso_decay_walk_takes(*{**a, **change}.values())


def test_which_steps_the_walk_takes():
    assert walk_takes() == 1 and walk_takes(dtype=0) == 1
    assert walk_takes(logits=AT, logits_ld=192, rotary=0) == 1
    for vdim, takes in ((64, 1), (128, 1), (192, 1), (256, 1), (320, 0), (32, 0), (96, 0)):
        assert walk_takes(vdim=vdim) == takes, vdim
    assert walk_takes(dim=32) == walk_takes(dim=128) == 0
    # four activations are read at a time: 8 bytes in bfloat16, 16 in float32
    for name in ("q", "k", "v"):
        assert walk_takes(**{name: AT + 8}) == 1 and walk_takes(**{name: AT + 8, "dtype": 0}) == 0
        assert walk_takes(**{name: AT + 6}) == 0 and walk_takes(**{name + "_ld": 258}) == 0
    assert walk_takes(state=AT + 8) == 0 and walk_takes(stride=64 * 64 + 2) == 0
    assert walk_takes(logits=AT + 8, logits_ld=192, rotary=0) == 0 and walk_takes(logits=AT, logits_ld=190, rotary=0) == 0
    for rotary, takes in ((0, 1), (8, 1), (16, 1), (2, 0), (20, 0), (36, 0)):
        assert walk_takes(rotary=rotary) == takes, rotary
    # what a grid has no room for stays with the general kernel
    assert walk_takes(tokens=1, seqs=65535) == 1 and walk_takes(tokens=128, seqs=65535) == 0
    assert walk_takes(tokens=128 * 65534 + 127, seqs=1) == 1 and walk_takes(tokens=128 * 65535, seqs=1) == 0


@pytest.mark.parametrize("sm_count", [148, 132])
def test_float_products_stay_within_what_is_set_aside(sm_count):
    groups_of = lambda t, n, k: library().shiso_gemm_float_groups(AT, AT, AT, t, n, k, sm_count)
    split = 0
    for k in (128, 256, 516, 1024, 4608, 16384):
        for t in (1, 8, 9, 24, 100, 300, 1000, 2048, 2300, 5000, 20000):
            room = core.float_product_room_bytes(t, k)
            for n in (1, 100, 128, 256, 512, 900, 1024, 2048, 4608, 9216, 65536):
                groups = groups_of(t, n, k)
                assert groups >= 0 and 4 * groups * t * n <= room, (t, n, k, groups)
                split += groups > 0
    assert split > 100
    assert groups_of(300, 1024, 1026) == -1  # rows of no multiple of four: the other kernel


@pytest.mark.parametrize("preset", ["filulix-1b", "filulix-350m"])
@pytest.mark.parametrize("rows", [64, 2048, 16384])
def test_recurrences_are_set_aside_for(preset, rows):
    with open(preset_path(preset)) as f:
        _, _, plan = plan_from_document(json.load(f))
    options = SimpleNamespace(max_num_batched_tokens=rows, max_num_seqs=8)
    # 16 heads of 64 x 128 and 32 of 64 x 64 (half as many in the smaller model): outputs in float32, two states per 128 rows
    heads = 32 if preset == "filulix-1b" else 16
    need = 4 * (rows * heads * 64 + 2 * (rows // 128) * heads * 64 * 64)
    assert core.recurrence_room_bytes(plan, rows) == need
    plain = core.step_buffer_bytes(SimpleNamespace(hidden_size=plan.hidden_size, vocab_size=plan.vocab_size, layers=[]), options, torch.bfloat16)
    assert core.step_buffer_bytes(plan, options, torch.bfloat16) >= plain + need
