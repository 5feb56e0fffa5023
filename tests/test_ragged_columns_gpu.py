"""Products with a B stored [K, N] whose last 128-byte column block is ragged: whole blocks come through one map, tiles
that touch the ragged block through another. Column counts around block and tile edges, one column of tiles and several."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [72, 120, 136, 200, 264, 328, 504, 520, 1000, 1696])
@pytest.mark.parametrize("m,pair", [(100, 1), (300, 2), (520, 2)])
def test_ragged_last_block(n, m, pair):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    from mm_rs_with_catlass_b200.tiling.config import TilingConfig
    from mm_rs_with_catlass_b200.utils.verify import assert_close
    g = torch.Generator(device="cuda").manual_seed(n + m)
    k = 200
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    # the operand ends with its last element, and what follows in memory must not reach a result
    store = torch.full((k * n + 64,), float("nan"), device="cuda", dtype=torch.bfloat16)
    b = store[: k * n].view(k, n)
    b.copy_(torch.randn(k, n, device="cuda", generator=g))
    for bn in (64, 128, 256):
        if pair == 2 and bn == 64:
            continue
        out = catcoc.matmul(a, b, tiling=TilingConfig(bn=bn, cta_pair=pair))
        torch.cuda.synchronize()
        raise_on_status(local_status(a.device), "ragged columns")
        assert_close(out, a.float() @ b.float(), k=k, dtype=torch.bfloat16, what="n=%d bn=%d" % (n, bn))
    n8 = max(16, n // 16 * 16)
    x1 = torch.randint(-127, 128, (m, 208), device="cuda", dtype=torch.int8, generator=g)
    x2 = torch.randint(-127, 128, (208, n8), device="cuda", dtype=torch.int8, generator=g)
    gold = (x1.double() @ x2.double()).int()                 # whole numbers below 2^53
    assert torch.equal(catcoc.matmul(x1, x2, tiling=TilingConfig(bn=256, cta_pair=pair)), gold)
