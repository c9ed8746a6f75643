"""Rules of the kernel files that no run shows reliably: what happens when they are broken depends on how far two
kernels overlap.  (common.cuh states them, where it explains dependent launches.)"""

import os
import re

import pytest

from shiso_llm_b200.kernels import build

SOURCES = {os.path.basename(p): open(p, encoding="utf-8").read() for p in build.sources()}

# Pointers that may be __restrict__ const: weights and other tensors that no kernel writes.
WEIGHTS = {"q_w", "k_w", "inv_freq", "w", "bias", "b", "pair_table", "coefficients", "norm_w", "taps", "mu", "correction", "mix", "write", "read"}


def kernels(text):
    """(name, parameters) of every kernel of a file."""
    pattern = re.compile(r"__global__\s+void\s*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^{]*?)\)\s*\{")
    return [(m.group(1), re.sub(r"\s+", " ", m.group(2))) for m in pattern.finditer(text)]


def test_nothing_a_kernel_writes_is_read_through_restrict_const():
    found = []
    for name, text in SOURCES.items():
        for kernel, parameters in kernels(text):
            for kind, what in re.findall(r"const ([\w ]+)\* __restrict__ (\w+)", parameters):
                if what not in WEIGHTS and not (what == "table" and kind == "WT"):
                    found.append((name, kernel, what))
            # read and written in place
            found += [(name, kernel, what) for what in re.findall(r"(?<!const )\b\w+\* __restrict__ (residual|proj|logits|state|x)\b", parameters)
                      if not re.search(r"const [\w ]+\* __restrict__ " + what, parameters)]
    assert sum(len(kernels(t)) for t in SOURCES.values()) > 60 and not found, found


def test_a_steps_first_kernel_is_launched_in_full_order():
    """What uploads a step's data lets its successor start early, and kernels read step data ahead of their wait."""
    for name, kernel in (("elementwise.cu", "embed_kernel"), ("stream_copies.cu", "embed_hashed_pair_kernel")):
        launches = re.findall(r"(launch_\w+)\(" + kernel + "<", SOURCES[name])
        assert launches == ["launch_in_order"] * 2, (name, launches)


@pytest.mark.parametrize("name", ["attention_prefill_tc.cu", "differential_attention_tc.cu"])
def test_attention_leaves_at_the_first_wait_that_runs_out(name):
    """Every wait is the condition of a way out of its loop; only the last ones of a role just note that they failed."""
    text = SOURCES[name]
    text = text[text.index("__global__"):]
    text = text[: text.index("\n}\n")]
    carried_on = [line.strip() for line in text.splitlines() if re.search(r"mbar_wait\(.*\)\) failed = true;", line)]
    assert [line for line in carried_on if "products_done" not in line and "q_full" not in line] == []
    waits = len(re.findall(r"(?<!auto )\bwait\(&|mbar_wait\(", text))
    ways_out = len(re.findall(r"if \(failed\) break;|return false;|&& landed;|&& !failed|if \(!failed\) failed|products_done, 0\)|q_full, 0\)|break;", text))
    assert waits >= 10 and ways_out >= waits - 3, (waits, ways_out)


@pytest.mark.parametrize("name", ["attention_prefill_tc.cu", "differential_attention_tc.cu", "gemm_float_tc.cu"])
def test_tensor_memory_is_taken_behind_the_wait_for_the_kernel_before(name):
    text = SOURCES[name]
    text = text[text.index("tcgen05.relinquish") - 2500 : text.index("tcgen05.relinquish")]
    assert "pdl_wait();" in text[: text.index("tcgen05.alloc")], name


@pytest.mark.parametrize("name", ["gemm_tcgen05_prompt.cu", "gemm_tcgen05_pair.cu"])
def test_products_let_their_successor_start_behind_their_main_loop(name):
    """Not from lanes without a role, which come to the kernel's end at once."""
    lines = [line.strip() for line in SOURCES[name].splitlines() if "pdl_trigger()" in line]
    assert len(lines) == 1 and lines[0].startswith("if (tile + ") and ">= num_tiles) pdl_trigger();" in lines[0], lines


def test_a_pair_takes_and_gives_back_its_tensor_memory_when_nothing_else_does():
    """Ahead of the wait for the kernel before, one CTA's allocation could stand for ever.  Both CTAs free theirs before either ends."""
    assert [name for name, t in SOURCES.items() if "tcgen05.alloc.cta_group::2" in t] == ["gemm_tcgen05_pair.cu"]
    text = SOURCES["gemm_tcgen05_pair.cu"]
    text = text[text.index("gemm_pair_kernel("):]
    order = [text.index(x) for x in ("cluster_sync_all();", "pdl_wait();", "tcgen05.alloc.cta_group::2", "// ---- producer", "// ---- epilogue",
                                     "nobody signals into", "tcgen05.relinquish_alloc_permit.cta_group::2", "tcgen05.dealloc.cta_group::2")]
    assert order == sorted(order)
    behind = text[order[-1]:]
    assert "cluster_sync_all();" in behind[: behind.index("\n}\n")]


def test_the_streaming_product_begins_no_wait_behind_one_that_ran_out():
    waits = [line.strip() for line in SOURCES["gemm_stream.cu"].splitlines() if "mbar_wait(&" in line]
    assert len(waits) == 3 and all("!timed_out && !mbar_wait(" in line or line.endswith("break;") for line in waits), waits
