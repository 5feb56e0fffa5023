"""Block-scaled products of at most 128 rows whose units are cut along K: half of every tile of rows lies outside the matrix, its
scales too."""
import pytest
import torch

import mm_rs_with_catlass_b200 as catcoc
from mm_rs_with_catlass_b200.ops import mx


def test_rule():
    assert mx._cut(16, 256, 12288) and mx._cut(128, 8192, 28672) and mx._cut(129, 8192, 28672)
    assert mx._cut(43, 8192, 7168) is None and mx._cut(16, 8192, 1024) is None


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(16, 256, 12288), (1, 1000, 16384), (31, 200, 12320), (127, 384, 12288), (128, 2000, 16384)])
def test_against_uncut(m, n, k, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(m)
    ops = []
    for rows in (m, n):
        q, s = catcoc.quantize_mxf8(torch.randn(rows, k, device="cuda", generator=g), "e4m3")
        ops += [q, catcoc.pack_scales(s)]
    assert mx._cut(m, n, k) is not None
    whole = torch.full((m + 1, n), 7.0, device="cuda")
    catcoc.mxf8_matmul(*ops, out=whole[:m], out_dtype=torch.float32)
    monkeypatch.setattr(mx, "_cut", lambda *a: None)
    mx._blocks.clear()
    want = catcoc.mxf8_matmul(*ops, out_dtype=torch.float32)
    mx._blocks.clear()
    # the same products summed in another order: fp32 rounding of sums of k terms of size sqrt(k) at most
    assert (whole[:m] - want).abs().max().item() <= 2.0 ** -23 * k and bool((whole[m] == 7).all())
