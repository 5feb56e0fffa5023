"""The attention kernel for few query rows per key / value head, where its plan can go wrong: runs of key blocks that
end inside a sequence, exactly at its end, or hold several sequences; one block in all; odd and even block counts per
run (the two accumulators); rows that fill one lane quarter, several, or the whole tile; causal rows of a packed group."""
import pytest
import torch

from test_attention_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,hq,hk,sq,sk", [
    (1, 1, 1, 1, 1), (1, 8, 1, 1, 128), (1, 8, 1, 1, 129), (1, 4, 1, 2, 257), (1, 32, 4, 4, 5000),   # few CTAs, cut sequences
    (37, 8, 4, 1, 384), (37, 8, 4, 1, 385), (30, 16, 8, 2, 700), (75, 8, 4, 4, 130),                 # whole sequences / cut ones
    (160, 4, 2, 1, 1000), (2, 2, 2, 128, 1024), (3, 4, 4, 97, 333), (1, 16, 4, 32, 2049),            # many runs, full tiles
])
@pytest.mark.parametrize("causal", [False, True])
def test_runs_of_key_blocks(b, hq, hk, sq, sk, causal):
    _run(b, hq, hk, sq, sk, 128, torch.bfloat16, causal, seed=sk + b)
    _run(b, hq, hk, sq, sk, 64, torch.float16, causal, seed=sk + b + 1)


@pytest.mark.parametrize("gain", [(0.2, 6.0), (6.0, 0.2)])
def test_accumulators_with_different_maxima_merge(gain):
    # growing keys: the later block of every pair and the later run dominate; shrinking: the earlier ones
    _run(2, 8, 2, 1, 4096, 128, torch.bfloat16, True, seed=3, key_gain=gain)
    _run(1, 8, 8, 3, 1500, 64, torch.float16, True, seed=4, key_gain=gain)
