# SPDX-License-Identifier: Apache-2.0
"""The tensor maps that attention and GEMM launches take: one cache, whose entries are told apart by every field."""
import os
import re
import subprocess

from core_scheduler_b200 import build as native_build

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "core_scheduler_b200", "csrc", "kernels")


def test_cached_maps_are_told_apart_by_every_field():
    program = [e for e in native_build.build_cpp_tests() if e.endswith("test_tensor_map")][0]
    out = subprocess.run([program], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "2 tests ran, 0 failed" in out.stdout, out.stdout[-3000:] + out.stderr[-3000:]


def test_kernels_keep_no_cache_of_their_own():
    for name in ("attention_tcgen05.cu", "gemm_tcgen05.cu"):
        with open(os.path.join(KERNELS, name)) as f:
            source = f.read()
        assert "get_tensor_map(" in source and not re.search(r"unordered_map|\bstd::map\b", source), name
