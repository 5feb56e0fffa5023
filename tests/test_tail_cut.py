"""Local products whose last wave of pair tiles is cut along K: ragged last tiles among the cut ones, all tiles cut, a
short last slice, every epilogue; results against the direct kernel (GPU). The rule gives a valid cut for every shape (CPU)."""
import pytest
import torch


def _both(monkeypatch, cut, bn, a, b, **kw):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops import gemm
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    from mm_rs_with_catlass_b200.tiling import chooser
    from mm_rs_with_catlass_b200.tiling.config import TilingConfig
    gemm._plans.clear()
    tiling = TilingConfig(bn=bn, cta_pair=2, swizzle=4)
    direct = catcoc.matmul(a, b, tiling=tiling, **kw)
    monkeypatch.setattr(chooser, "split_k", lambda *x: None)
    monkeypatch.setattr(chooser, "choose", lambda *x, **y: tiling)
    monkeypatch.setattr(chooser, "tail_cut", lambda *x: (1.0, cut))
    res = catcoc.matmul(a, b, **kw)
    assert torch.equal(res, catcoc.matmul(a, b, **kw))        # the planned call
    gemm._plans.clear()
    torch.cuda.synchronize()
    raise_on_status(local_status(a.device), "tail")
    return direct, res


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,bn,first,slices,ks", [
    (300, 700, 1100, 256, 4, 3, 384), (512, 1024, 2048, 256, 0, 2, 1024), (513, 136, 1000, 128, 5, 4, 256), (1000, 520, 1280, 192, 7, 5, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_cut_tiles_match_the_direct_product(monkeypatch, m, n, k, bn, first, slices, ks, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    for trans_b in ((True,) if bn == 192 else (True, False)):
        b = torch.randn(*((n, k) if trans_b else (k, n // 8 * 8)), device="cuda", generator=g).to(dtype)
        direct, cut = _both(monkeypatch, (first, slices, ks), bn, a, b, trans_b=trans_b, out_dtype=torch.float32)
        # both are fp32 sums of exact products, in another order: k * 2^-24 relative to the sum of magnitudes (about sqrt(k))
        assert (direct - cut).abs().max().item() < k * 2.0 ** -24 * 4 * k ** 0.5


@pytest.mark.gpu
def test_epilogues(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(7)
    m, n, k = 600, 520, 1536
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = (torch.randn(k, n, device="cuda", generator=g) * 0.05).bfloat16()
    c = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g)
    for kw in (dict(), dict(activation="gelu"), dict(alpha=0.5, beta=2.0, c=c, bias_f32=bias), dict(bias_f32=bias, activation="relu")):
        direct, cut = _both(monkeypatch, (5, 3, 512), 256, a, b, **kw)
        # one bf16 rounding of values that differ by the order of an fp32 sum: neighbouring bf16 numbers at most
        assert ((direct.float() - cut.float()).abs() <= 2.0 ** -7 * direct.float().abs() + 1e-3).all()
    # int8: the sums are whole numbers, so the results are the same bits
    x1 = torch.randint(-127, 128, (m, k), device="cuda", dtype=torch.int8, generator=g)
    x2 = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8, generator=g)
    s1, s2 = torch.rand(m, device="cuda", generator=g) * 0.02, torch.rand(n, device="cuda", generator=g) * 0.01
    ib = torch.randint(-1000, 1000, (n,), device="cuda", dtype=torch.int32, generator=g)
    for kw in (dict(), dict(bias=ib), dict(scale_m=s1, scale_n=s2, bias=ib), dict(scale_m=s1, scale_n=s2, out_dtype=torch.float16), dict(scale_n=s2)):
        direct, cut = _both(monkeypatch, (4, 3, 512), 256, x1, x2, trans_b=True, **kw)
        assert torch.equal(direct, cut)


def test_rule_cuts_whole_stages_that_cover_k():
    from mm_rs_with_catlass_b200.tiling import chooser
    hits = 0
    for m in (300, 512, 1024, 8144):
        for n in (1696, 5120, 8192):
            for k in (520, 5120, 6148, 28672):
                for elt in (1, 2):
                    for bn in (128, 192, 256):
                        waves, cut = chooser.tail_cut(m, n, k, elt, bn)
                        if cut is not None:
                            first, s, ks = cut
                            tiles = -(-m // 256) * -(-n // bn)
                            assert 0 <= first < tiles and s >= 2 and (ks * elt) % 256 == 0 and ks * (s - 1) < k <= ks * s
                            hits += 1
    assert hits > 10
