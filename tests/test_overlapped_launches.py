"""Kernels that are set up while their predecessor in the stream still runs (``host::launch_overlapped``, the local launches
of the fused kernel): what they read may still be written until ``grid_dependency_wait()`` returns. So the sources hold no
access ahead of it and no read-only load (``__ldg``, ``const __restrict__``), which a compiler may move ahead of it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mm_rs_with_catlass_b200", "csrc")
# files whose kernels (and device functions) all belong to overlapped launches
WHOLE = ["kernels/flash_attn.cu", "kernels/flash_decode.cu", "kernels/mla_rows.cu", "kernels/mx_quant.cu", "kernels/launch.cu",
         "include/catcoc/fused_gemm.cuh", "include/catcoc/double_tile.cuh", "include/catcoc/softmax_row.cuh"]
FILES = WHOLE + ["kernels/blas_prims.cu"]


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


def _closed(s, i, opening, closing):
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == opening) - (s[j] == closing)
        if depth == 0 and s[j] == closing:
            return j
    raise AssertionError("unbalanced source")


def _kernels(s):
    """(name, parameters, body) of every kernel definition."""
    for m in re.finditer(r"__global__\s+void\s+", s):
        i = m.end()
        if s.startswith("__launch_bounds__", i):
            i = _closed(s, s.index("(", i), "(", ")") + 1
        name = re.match(r"\s*(\w+)\s*\(", s[i:])
        par = i + name.end() - 1
        end = _closed(s, par, "(", ")")
        brace = s.index("{", end)
        yield name.group(1), s[par + 1:end], s[brace:_closed(s, brace, "{", "}") + 1]


@pytest.mark.parametrize("name", FILES)
def test_nothing_is_read_ahead_of_the_wait(name):
    s = _source(name)
    seen = 0
    for kernel, params, body in _kernels(s):
        if "grid_dependency_wait" not in body:
            # launched the ordinary way
            assert re.search(kernel + r"\s*(<[^;(]*?>)?\s*<<<", s), "%s neither waits nor is launched by itself" % kernel
            continue
        seen += 1
        assert "__restrict__" not in params, kernel
        assert "__ldg" not in body and "ldg_v4" not in body, kernel
        before = body[:body.rindex("grid_dependency_wait")]
        for p in params.split(","):
            if "*" in p:
                assert not re.search(r"(?<!\.)\b%s\b" % re.search(r"(\w+)\s*$", p).group(1), before), (kernel, p)
        assert not re.search(r"\breturn\b", re.sub(r"\[&\][^;]*?\{.*?\};", "", before, flags=re.S)), "%s may end without the wait" % kernel
    assert seen > 0 or name.endswith("softmax_row.cuh")
    if name in WHOLE:
        assert "__ldg" not in s and "__ldcg" not in s
