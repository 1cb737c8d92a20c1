"""Rules of the CUDA sources that no run can show."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kitbase.jl_gb300", "csrc")


def _sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as s:
                yield f, re.sub(r"//[^\n]*", "", s.read())


def test_overlapping_kernels_hold_no_input_read_only():
    """A kernel that waits on the one before it (pdl_wait) is resident while that
    one writes its input: neither its parameters nor the distributions that it
    reads are const __restrict__, and it reads none of it by __ldg."""
    seen = 0
    for f, src in _sources():
        for m in re.finditer(r"__global__[^;{]*?(k_\w+)\s*\(([^{;]*?)\)\s*\{", src):
            body = src[m.end():src.find("__global__", m.end())]
            if "pdl_wait()" in body:
                seen += 1
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", m.group(2)), (f, m.group(1))
        assert not re.search(r"const\s+R\s*\*\s*__restrict__\s*(H|Bq|q|hin|bin)\b", src), f
        for x in re.findall(r"__ldg\(([^)]*)", src):  # tables that no step writes
            assert re.match(r"d\.(step_rec|step_geo32|cell_iarea)\b", x.strip()), (f, x)
    assert seen >= 12
