"""Steps that run kernel by kernel while the device is still busy with the ones before: a step's data comes from a kernel that loads it
from the host's memory, and nothing of the step may read it earlier.  (A device that idles between launches hides such a read: the
steps here wait behind long products, so that every launch of a step is in the queue when its first kernel starts.)"""

import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu

# heads of 64: single tokens and long portions take the kernels that read step data ahead of their wait
DOC = {**helpers.TINY_A, "hidden_size": 256, "num_attention_heads": 4, "num_key_value_heads": 2, "num_hidden_layers": 3,
       "layer_types": ["full_attention", "conv", "full_attention"]}


def test_steps_queued_behind_work_give_the_bits_of_steps_one_at_a_time(tmp_path):
    helpers.make_folder(tmp_path, DOC, 5)
    prompts = {"a": helpers.random_prompt(330, DOC["vocab_size"], 1), "b": helpers.random_prompt(460, DOC["vocab_size"], 2)}
    steps = [[("a", prompts["a"][:200])], [("b", prompts["b"][:300])]]
    for i in range(130):  # contexts cross the borders of pages and key tiles, alone and together
        entries = [("a", [prompts["a"][200 + i]])] if i % 3 != 1 else []
        entries += [("b", [prompts["b"][300 + i]])] if i % 3 != 2 else []
        steps.append(entries)
    steps.append([("b", prompts["b"][430:]), ("c", prompts["a"][:150])])
    got = {}
    for queued in (False, True):
        engine = helpers.make_engine(tmp_path, "bfloat16", page_size=16, kv_cache_tokens=2048, ctx=512, max_num_seqs=4,
                                     max_num_batched_tokens=512, cuda_graphs=False)
        big = torch.zeros(8192, 8192, dtype=torch.bfloat16, device="cuda")
        rows = []
        for entries in steps:
            if queued:
                torch.mm(big, big)
                torch.mm(big, big)
            rows.append(engine.step([helpers.StepEntry(r, tokens, [len(tokens) - 1]) for r, tokens in entries]).clone())
            if not queued:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        engine.env.ops.check_kernel_status()
        got[queued] = rows
    for i, (one, other) in enumerate(zip(got[False], got[True])):
        assert torch.isfinite(one).all() and torch.equal(one, other), f"step {i}: {steps[i]}"
