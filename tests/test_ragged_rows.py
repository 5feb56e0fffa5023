"""Outputs whose rows begin at any element: the same bits as in an aligned buffer, nothing written beside them."""
import pytest
import torch

import mm_rs_with_catlass_b200 as catcoc
from mm_rs_with_catlass_b200.tiling.config import TilingConfig

TILINGS = {"single": dict(bn=64, cta_pair=1), "pair": dict(bn=256, cta_pair=2),
           "double": dict(bn=64, cta_pair=2, twice=True), "swapped": dict(bn=64, cta_pair=2, twice=True, swap=True)}


@pytest.mark.gpu
@pytest.mark.parametrize("tiling", sorted(TILINGS))
@pytest.mark.parametrize("kind", ["bf16", "bf16_to_fp32", "int8_to_int32"])
def test_rows_at_any_element(tiling, kind):
    g = torch.Generator().manual_seed(7)
    k, rows, cols = 144, 301, 330
    if kind == "int8_to_int32":
        a, b = (torch.randint(-127, 128, s, generator=g, dtype=torch.int8).cuda() for s in ((rows, k), (cols, k)))
    else:
        a, b = (torch.randn(s, generator=g).cuda().bfloat16() for s in ((rows, k), (cols, k)))
    dt = {"bf16": torch.bfloat16, "bf16_to_fp32": torch.float32, "int8_to_int32": torch.int32}[kind]
    t = TilingConfig(swizzle=2, **TILINGS[tiling])
    for m, n in ((1, 1), (7, 2), (33, 63), (255, 64), (64, 65), (301, 97), (300, 127), (257, 128), (31, 129), (129, 250), (301, 323)):
        want = catcoc.matmul(a[:m], b[:n], trans_b=True, tiling=t, out=torch.empty(m, 336, device="cuda", dtype=dt)[:, :n])
        for pitch, first in ((336, 0), (336, 1), (335, 0), (335, 3), (334, 0), (334, 1), (332, 2), (336, 4)):
            first = min(first, pitch - n)
            whole = torch.full((m, pitch), 77, device="cuda", dtype=dt)
            catcoc.matmul(a[:m], b[:n], trans_b=True, tiling=t, out=whole[:, first:first + n])
            assert torch.equal(whole[:, first:first + n], want), (m, n, pitch, first)
            assert bool((whole[:, :first] == 77).all()) and bool((whole[:, first + n:] == 77).all()), (m, n, pitch, first)
