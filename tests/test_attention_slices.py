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


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("b,h,sq,sk,first", [(1, 1, 2300, 2301, 1280), (1, 2, 1900, 1900, 896), (2, 1, 1500, 4096, 3200)])
def test_values_behind_a_tile_do_not_reach_its_rows(b, h, sq, sk, first, bad):
    """Values that are no numbers from key ``first`` on, over several slices: tiles of 128 rows that see none of these keys give the
    bits that they give without them, as they do where the keys are not cut. A query that is no number still shows."""
    import mm_rs_with_catlass_b200 as catcoc
    for d in (64, 128):
        assert _scratch(b, h, h, sq, sk, d, True) > 0
        g = torch.Generator(device="cuda").manual_seed(d)
        q, k, v = (torch.randn(b, h, s, d, device="cuda", generator=g).bfloat16() for s in (sq, sk, sk))
        want = catcoc.flash_attention(q, k, v, causal=True)
        v[:, :, first:] = bad
        got = catcoc.flash_attention(q, k, v, causal=True)
        clean = sum(1 for t in range(0, sq, 128) if min(sk, t + 128 + sk - sq) <= first) * 128
        assert 0 < clean < sq and torch.equal(got[:, :, :clean], want[:, :, :clean])
        assert not got[:, :, -1].isfinite().any()
        q[:, :, 5] = float("nan")
        assert catcoc.flash_attention(q, k, v, causal=True)[:, :, 5].isnan().all()


# D = 64: launches on either side of the line between the two forms of a block's wait: one wave, more, masks over much and over little
WAITS = [(2, 32, 8, 300, 600, True), (8, 32, 8, 300, 1200, True), (3, 32, 8, 600, 1200, True), (6, 32, 8, 1000, 1000, False), (1, 4, 4, 130, 300, False)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", WAITS)
def test_both_forms_of_the_wait(case):
    assert _scratch(*case[:5], 64, case[5]) == 0
    _run(*case[:5], 64, torch.bfloat16, case[5], seed=case[3])
