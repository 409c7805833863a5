# SPDX-License-Identifier: Apache-2.0
"""A warp leaves an abandoned mbarrier wait as one. Lanes that see different answers when a wait runs out (one the barrier's
phase, another the abort flag) would part ways before warp-aligned instructions and hang there, so every role of the tensor-core
kernels waits through the voted form. Read from the sources: a wait that runs out is not provoked on a GPU."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "core_scheduler_b200", "csrc", "kernels")


@pytest.mark.parametrize("name", ["gemm_tcgen05.cu", "attention_tcgen05.cu"])
def test_every_wait_of_a_role_is_voted_on(name):
    with open(os.path.join(KERNELS, name)) as f:
        source = re.sub(r"//[^\n]*", "", f.read())
    definition = re.search(r"bool mbar_wait_warp\([^{]*\{.*?\n\}", source, re.S)
    assert definition and definition.group(0).count("__all_sync") == 2
    rest = source.replace(definition.group(0), "")
    rest = re.sub(r"__device__ __forceinline__ bool mbar_(?:try_)?wait\([^{]*\{.*?\n\}", "", rest, flags=re.S)
    assert rest.count("mbar_wait_warp(") >= 5
    assert not re.findall(r"\bmbar_(?:try_)?wait\(", rest)
