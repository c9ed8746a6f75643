"""Rules of the kernel files that no run shows reliably: what happens when they are broken depends on how far two
kernels overlap.  (common.cuh states them, where it explains dependent launches.)"""

import os
import re

from shiso_llm_b200.kernels import build

SOURCES = {os.path.basename(p): open(p, encoding="utf-8").read() for p in build.sources()}


def test_a_steps_first_kernel_is_launched_in_full_order():
    """What uploads a step's data lets its successor start early, and kernels read step data ahead of their wait."""
    for name, kernel in (("elementwise.cu", "embed_kernel"), ("stream_copies.cu", "embed_hashed_pair_kernel")):
        launches = re.findall(r"(launch_\w+)\(" + kernel + "<", SOURCES[name])
        assert launches == ["launch_in_order"] * 2, (name, launches)
