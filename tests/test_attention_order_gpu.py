"""Order and packing of the attention kernel's query tiles: heads of a KV head packed into tiles (rows of two heads in one
tile, a last tile that is not full, positions with and without a cache offset), and causal launches whose heads are walked
in several blocks, the last of them short."""
import pytest
import torch

from test_attention_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,hq,hk,sq,sk", [(2, 32, 4, 50, 50), (40, 32, 4, 33, 300), (20, 16, 2, 100, 1000), (12, 32, 8, 129, 129),
                                           (9, 24, 8, 255, 400), (16, 32, 4, 300, 300), (8, 8, 1, 520, 520)])
@pytest.mark.parametrize("causal", [False, True])
def test_packed_heads(b, hq, hk, sq, sk, causal):
    _run(b, hq, hk, sq, sk, 128, torch.bfloat16, causal, seed=sq + sk)
    _run(b, hq, hk, sq, sk, 64, torch.float16, causal, seed=sq + sk + 1)


def test_heads_in_blocks():
    # keys and values of 8.4 MB a head: blocks of 8 heads, the last one of 4
    _run(1, 20, 20, 300, 16384, 128, torch.bfloat16, True, seed=1)
    _run(1, 12, 3, 600, 33000, 64, torch.float16, True, seed=2)
