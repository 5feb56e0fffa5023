"""Local products whose K range is cut into slices: the rule gives a valid cut for every shape (CPU), and the two launches
give the direct kernel's result for ragged rows and columns, a short last slice and every epilogue (GPU)."""
import pytest
import torch


def test_rule_gives_whole_stages_that_cover_k():
    from mm_rs_with_catlass_b200.tiling import chooser
    hits = 0
    for m in (1, 17, 100, 128, 200, 512, 4096):
        for n in (64, 130, 1696, 8192, 28672):
            for k in (48, 512, 3584, 6148, 28672):
                for elt, dt in ((2, torch.bfloat16), (1, torch.int8)):
                    cut = chooser.split_k(m, n, k, elt, chooser.heuristic("matmul", m, n, k, 1, dt))
                    if cut is None:
                        continue
                    s, ks, bn = cut
                    assert s >= 2 and (ks * elt) % 256 == 0 and ks * (s - 1) < k <= ks * s and bn in (128, 256)
                    hits += 1
    assert hits > 20
    assert chooser.split_k(8192, 8192, 8192, 2, chooser.heuristic("matmul", 8192, 8192, 8192, 1, torch.bfloat16)) is None


def _both(monkeypatch, cut, a, b, **kw):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops import gemm
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    from mm_rs_with_catlass_b200.tiling import chooser
    res = []
    for c in (None, cut):
        monkeypatch.setattr(chooser, "split_k", lambda *a, c=c: c)
        gemm._plans.clear()
        first = catcoc.matmul(a, b, **kw)
        again = catcoc.matmul(a, b, **kw)                    # the planned call
        assert torch.equal(first, again)
        res.append(first)
    gemm._plans.clear()
    torch.cuda.synchronize()
    raise_on_status(local_status(a.device), "split-K matmul")
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 64, 1024), (33, 130, 1100), (128, 512, 2048), (129, 1000, 4000), (300, 72, 520)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_slices_match_the_direct_product(monkeypatch, m, n, k, trans_a, trans_b, dtype):
    if trans_a:
        m = (m + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(*((k, m) if trans_a else (m, k)), device="cuda", generator=g).to(dtype)
    b = torch.randn(*((n, k) if trans_b else (k, n)), device="cuda", generator=g).to(dtype)
    for s, ks, bn in ((2, -(-k // 2 // 128) * 128, 128), (-(-k // 256), 256, 256)):
        if ks * (s - 1) >= k or s < 2:
            continue
        direct, cut = _both(monkeypatch, (s, ks, bn), a, b, trans_a=trans_a, trans_b=trans_b, out_dtype=torch.float32)
        # both are fp32 sums of exact products, in another order: k * 2^-24 relative to the sum of magnitudes (about sqrt(k))
        assert (direct - cut).abs().max().item() < k * 2.0 ** -24 * 4 * k ** 0.5


@pytest.mark.gpu
def test_epilogues(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(5)
    m, n, k = 70, 264, 3000
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = (torch.randn(k, n, device="cuda", generator=g) * 0.05).bfloat16()
    c = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g)
    for kw in (dict(activation="gelu"), dict(activation="silu"), dict(alpha=0.5, beta=2.0, c=c, bias_f32=bias), dict(bias_f32=bias, activation="relu")):
        direct, cut = _both(monkeypatch, (3, 1024, 128), a, b, **kw)
        # one bf16 rounding of values that differ by the order of an fp32 sum: neighbouring bf16 numbers at most
        assert ((direct.float() - cut.float()).abs() <= 2.0 ** -7 * direct.float().abs() + 1e-3).all()
    # int8: the sums are whole numbers, so the results are the same bits
    x1 = torch.randint(-127, 128, (m, k), device="cuda", dtype=torch.int8, generator=g)
    x2 = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8, generator=g)
    s1, s2 = torch.rand(m, device="cuda", generator=g) * 0.02, torch.rand(n, device="cuda", generator=g) * 0.01
    ib = torch.randint(-1000, 1000, (n,), device="cuda", dtype=torch.int32, generator=g)
    k = 2992
    x1, x2 = x1[:, :k].contiguous(), x2[:, :k].contiguous()
    for kw in (dict(), dict(bias=ib), dict(scale_m=s1, scale_n=s2, bias=ib), dict(scale_m=s1, scale_n=s2, out_dtype=torch.float16), dict(scale_n=s2)):
        direct, cut = _both(monkeypatch, (3, 1024, 256), x1, x2, trans_b=True, **kw)
        assert torch.equal(direct, cut)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 32, 33, 64, 65])                      # planes up to 64 rows leave from the registers
@pytest.mark.parametrize("n", [32, 136, 1001, 1024])                    # whole and partial 32-column pieces, padded pitch
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.int8])
def test_planes_of_few_rows(monkeypatch, m, n, dtype):
    k = 2048
    g = torch.Generator(device="cuda").manual_seed(m + n)
    if dtype == torch.int8:
        a = torch.randint(-127, 128, (m, k), device="cuda", generator=g, dtype=dtype)
        b = torch.randint(-127, 128, (n, k), device="cuda", generator=g, dtype=dtype)
        kw = dict(scale_m=torch.rand(m, device="cuda", generator=g), scale_n=torch.rand(n, device="cuda", generator=g))
    else:
        a, b = (torch.randn(r, k, device="cuda", generator=g).to(dtype) for r in (m, n))
        kw = dict(out_dtype=torch.float32)
    for cut in ((4, 512, 128), (8, 256, 256)):
        direct, sliced = _both(monkeypatch, cut, a, b, trans_b=True, **kw)
        if dtype == torch.int8:
            assert torch.equal(direct, sliced)                          # the planes hold whole numbers
        else:
            # fp32 sums of exact products in another order: k * 2^-24 relative to the sum of magnitudes (about sqrt(k))
            assert (direct - sliced).abs().max().item() < k * 2.0 ** -24 * 4 * k ** 0.5
