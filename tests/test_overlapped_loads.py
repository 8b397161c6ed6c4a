"""A kernel launched to overlap the one before it is resident while that one still writes, so what it
reads of the stream's data must go through ld_stream: a non-coherent load (__ldg, or a plain one
through a const __restrict__ pointer) is for memory that nothing writes while the kernel lives."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neural_wavelet_prt_demo_b200", "csrc")

# Read-only pointers that may be non-coherent: the weights, which only host-synchronous copies write,
# and the arguments of sh.cu's SH dot product, whose kernels are launched as usual.
MAY_BE_READ_ONLY = {"relight_tc.cu": {"table"}, "relight_common.cu": {"emb"}, "sh.cu": {"T", "Lg", "L"}}
LDG_OF = {"relight_tc.cu": {"lvl"}}  # the hash table's levels


def _sources():
    files = {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith(".cu")}
    return {f: s for f, s in files.items() if "launch_overlapped(" in s}


def test_the_overlapped_kernels_are_where_they_are_looked_for():
    assert {"env_rotate.cu", "haar_topk.cu", "relight_common.cu", "relight_tc.cu", "sh.cu",
            "tonemap.cu"} == set(_sources())


@pytest.mark.parametrize("name", ["env_rotate.cu", "haar_topk.cu", "relight_common.cu", "relight_tc.cu", "sh.cu",
                                  "tonemap.cu"])
def test_stream_data_is_not_read_by_non_coherent_loads(name):
    src = re.sub(r"//[^\n]*", "", _sources()[name])
    read_only = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", src))
    assert read_only <= MAY_BE_READ_ONLY.get(name, set()), read_only
    ldg = set(re.findall(r"__ldg\s*\(\s*(\w+)", src))
    assert ldg <= LDG_OF.get(name, set()), ldg
