"""Attention with the keys cut into slices: slices that a tile, or a row, sees nothing of, a short last slice, packed heads, moving
maxima; the rule cuts only where tiles are few and keys are many."""
import pytest
import torch

from mm_rs_with_catlass_b200 import _native as N
from test_attention_gpu import _run

# b, hq, hk, sq, sk, causal
CUT = [(1, 32, 4, 131, 3404, True), (1, 8, 8, 170, 5000, False), (2, 4, 1, 200, 3000, True), (1, 1, 1, 300, 4096, True), (1, 2, 2, 257, 2500, True),
       (1, 8, 2, 160, 1930, True), (1, 2, 1, 1900, 1900, True), (1, 1, 1, 2300, 2301, True), (4, 32, 8, 64, 4096, True), (1, 4, 2, 300, 2049, False), (3, 5, 5, 129, 4096, True)]


def _scratch(b, hq, hk, sq, sk, d, causal):
    return int(N.lib().catcoc_flash_attention_workspace_bytes(b, hq, hk, sq, sk, d, int(causal)))


def test_the_rule():
    for d in (64, 128):
        for b, hq, hk, sq, sk, causal in CUT:
            need, rows = _scratch(b, hq, hk, sq, sk, d, causal), b * hq * sq
            assert need > 0 and need % (rows * (d + 2) * 4) == 0 and 2 <= need // (rows * (d + 2) * 4) <= 16
        for case in ((1, 32, 8, 8192, 8192, True), (16, 32, 8, 300, 4096, True), (1, 32, 32, 128, 128, False), (1, 8, 2, 160, 1290, True)):
            assert _scratch(*case[:5], d, case[5]) == 0
    assert _scratch(1, 3, 2, 100, 4096, 128, True) == 0 and _scratch(0, 8, 8, 100, 4096, 128, True) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("case", CUT)
def test_against_the_reference(case, d):
    for dtype in (torch.bfloat16, torch.float16):
        _run(*case[:5], d, dtype, case[5], seed=case[3])


@pytest.mark.gpu
@pytest.mark.parametrize("gain", [(0.0, 6.0), (6.0, 0.0)])
def test_moving_reference_maxima(gain):
    for d in (64, 128):
        _run(1, 8, 2, 160, 3000, d, torch.bfloat16, True, seed=5, key_gain=gain)
