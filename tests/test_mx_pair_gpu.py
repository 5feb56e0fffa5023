"""Block-scaled fp8 products on 2-CTA tiles of 256 x 192: tile columns that start in the middle of a scale block, ragged
last tiles in both directions, an odd number of K-blocks (a stage holds two), scales that differ from block to block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(129, 192, 128), (256, 384, 256), (300, 200, 384), (512, 1000, 1184), (1000, 576, 160), (130, 64, 96)])
@pytest.mark.parametrize("fmt", ["e4m3", "e5m2"])
def test_pair_tiles(m, n, k, fmt):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    from mm_rs_with_catlass_b200.ops.mx import dequantize_mxf8
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    # rows and K-blocks of very different magnitude, so that a scale applied to the wrong place is off by a factor of two or more
    x = torch.randn(m, k, device="cuda", generator=g) * torch.exp2(torch.randint(-6, 7, (m, 1), device="cuda", generator=g).float())
    w = torch.randn(n, k, device="cuda", generator=g) * torch.exp2(torch.randint(-6, 7, (n, 1), device="cuda", generator=g).float())
    ramp = torch.exp2((torch.arange(k, device="cuda") // 32 % 7 - 3).float())
    xq, xs = catcoc.quantize_mxf8((x * ramp).bfloat16(), fmt)
    wq, ws = catcoc.quantize_mxf8((w / ramp).bfloat16(), fmt)
    out = catcoc.mxf8_matmul_reduce_scatter(xq, catcoc.pack_scales(xs), wq, catcoc.pack_scales(ws))
    torch.cuda.synchronize()
    raise_on_status(local_status(out.device), "mx pair")
    a, b = dequantize_mxf8(xq, xs).double(), dequantize_mxf8(wq, ws).double()
    gold, mag = a @ b.t(), a.abs() @ b.abs().t()
    # one rounding to bf16 (2^-9 relative) and an fp32 sum (k * 2^-24 of the magnitudes)
    assert ((out.double() - gold).abs() <= 2.0 ** -8 * gold.abs() + k * 2.0 ** -23 * mag).all()


@pytest.mark.parametrize("m,n,k", [(256, 192 * 74, 288), (200, 192 * 74 + 8, 288), (300, 192 * 80 - 40, 160), (700, 192 * 50, 416)])
def test_one_wave_of_units_and_more(m, n, k):
    # on 74 pairs: the last launch whose units are one to a pair (one accumulator each), the first with more, and double tiles
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    from mm_rs_with_catlass_b200.ops.mx import dequantize_mxf8
    g = torch.Generator(device="cuda").manual_seed(n)
    ramp = torch.exp2((torch.arange(k, device="cuda") // 32 % 7 - 3).float())
    rows = torch.exp2(torch.randint(-6, 7, (n, 1), device="cuda", generator=g).float())
    xq, xs = catcoc.quantize_mxf8((torch.randn(m, k, device="cuda", generator=g) * ramp).bfloat16())
    wq, ws = catcoc.quantize_mxf8((torch.randn(n, k, device="cuda", generator=g) * rows / ramp).bfloat16())
    out = catcoc.mxf8_matmul(xq, catcoc.pack_scales(xs), wq, catcoc.pack_scales(ws), out_dtype=torch.float32)
    torch.cuda.synchronize()
    raise_on_status(local_status(out.device), "mx units")
    a, b = dequantize_mxf8(xq, xs).double(), dequantize_mxf8(wq, ws).double()
    gold, mag = a @ b.t(), a.abs() @ b.abs().t()
    assert ((out.double() - gold).abs() <= k * 2.0 ** -23 * mag).all()      # an fp32 sum
