"""The tile choice for launches over groups of rows: legal for every dtype and size, pairs only where the groups' padding
allows them, narrower tiles where wide ones leave most SMs idle."""
import pytest
import torch

from mm_rs_with_catlass_b200.tiling import chooser
from mm_rs_with_catlass_b200.tiling.chooser import grouped


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.int8])
@pytest.mark.parametrize("groups", [1, 8, 64])
def test_choice_is_legal(dtype, groups):
    for rows in (1, 3, 100, 129, 256, 300, 2000):
        for n in (8, 64, 200, 1408, 4096):
            for per in (rows, rows + 0.5):
                t = grouped(int(groups * per), per, n, dtype).validate()
                assert t.cta_pair == 1 or (per > 64 and t.effective_bn >= 128)
                assert dtype != torch.int8 or t.effective_bn // (2 if t.cta_pair == 2 else 1) >= 128


def test_choice_follows_the_waves():
    assert grouped(8 * 1024, 1024, 8192, torch.bfloat16).cta_pair == 2          # whole 256-row tiles
    assert grouped(14080, 440.0, 4096, torch.bfloat16).cta_pair == 1            # half a tile of padding in each of 32 groups
    assert grouped(148, 18.5, 1408, torch.bfloat16).effective_bn < 256          # 48 wide tiles for 148 SMs
    # an exact row count and an equal mean are different questions, in either order
    assert [grouped(8 * 512, r, 8192, torch.bfloat16).cta_pair for r in (512.0, 512, 512.0)] == [
        grouped(8 * 512, float(512), 8192, torch.bfloat16).cta_pair, 2, grouped(8 * 512, 512.0, 8192, torch.bfloat16).cta_pair]
    assert grouped(14080, 440, 4096, torch.bfloat16) is not grouped(14080, 440.0, 4096, torch.bfloat16)


@pytest.mark.parametrize("case,order", list(enumerate([("1", None), (None, "1"), ("1", "2"), ("2", "1")])))
def test_choices_follow_the_forced_cta_count(monkeypatch, case, order):
    """A choice made with CATCOC_CTA_PAIR set is not kept for calls without it, nor the other way round."""
    tokens = 14080 + 64 * case             # sizes of its own: what an earlier order left behind serves no later one
    rules = {"ranges along K": lambda: chooser.slice_k_groups(32, 2048, 4096, tokens, torch.bfloat16),
             "groups of rows": lambda: chooser.token_groups(tokens, 32, 4096, 2048, torch.bfloat16),
             "one product": lambda: chooser.choose("matmul", 4096 + tokens, 4096, 4096, 1, torch.bfloat16, tails=True, doubles=True)}
    for name, rule in rules.items():
        seen = []
        for forced in order:
            if forced is None:
                monkeypatch.delenv("CATCOC_CTA_PAIR", raising=False)
            else:
                monkeypatch.setenv("CATCOC_CTA_PAIR", forced)
            seen.append(rule())
        for forced, t in zip(order, seen):
            assert (t.cta_pair == 1) == (forced == "1"), (name, order, t)
