"""The latent-attention kernel with chunks of 64 query rows, and with more than 128 rows: rows below, at and above a chunk and
half a chunk (each half has a warpgroup of its own), runs that end inside sequences, masked and stale keys, moving maxima."""
import pytest
import torch

from test_mla_rows_gpu import _case

pytestmark = pytest.mark.gpu
LENS = [0, 700, 129, 1, 2050, 0, 128, 17, 300]


def _spare_pages(rows, lens):
    """Pages a sequence may have beyond these lengths, so that chunks of 64 rows are taken."""
    chunks = -(-rows // 32)
    return -(-24 * 148 // (chunks * len(lens))) + 1


@pytest.mark.parametrize("q_len,heads", [(1, 64), (1, 33), (3, 21), (1, 65), (1, 96), (1, 97), (4, 32), (4, 33), (2, 128), (4, 128)])
@pytest.mark.parametrize("wide", [False, True])
def test_rows_and_the_causal_mask(q_len, heads, wide):
    for causal in (False, True):
        lens = [max(n, q_len) if n else 0 for n in LENS]
        _case(q_len, heads, lens, torch.bfloat16, causal=causal, seed=heads, extra_pages=_spare_pages(q_len * heads, lens) if wide else 0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", [[700] * 150, [100] * 140, [(37 * i) % 900 for i in range(70)], [9000, 20, 4000]])
def test_runs_of_pages(lens, dtype):
    for heads in (64, 80, 256):
        _case(1, heads, lens, dtype, seed=sum(lens) + heads, extra_pages=_spare_pages(heads, lens) if len(lens) < 100 else 20)


@pytest.mark.parametrize("heads", [64, 128])
@pytest.mark.parametrize("gain", [(0.0, 40.0), (40.0, 0.0)])
def test_moving_reference_maxima(heads, gain):
    _case(1, heads, [3000, 1100, 40], torch.bfloat16, gain=gain, seed=3, extra_pages=_spare_pages(heads, [1] * 3))


@pytest.mark.parametrize("heads", [64, 192])
def test_stale_cache_slots(heads):
    _case(1, heads, [131, 300, 17, 1, 255], torch.bfloat16, seed=4, stale=True, extra_pages=_spare_pages(heads, [1] * 5))
