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
