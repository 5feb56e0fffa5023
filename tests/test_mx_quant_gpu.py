"""The block-scaled quantisation and scale-packing kernels against the same functions in PyTorch (the CPU path of
``quantize_mxf8`` / ``pack_scales``). Values and scales are compared as bytes: every step (amax, log2, the power-of-two
scale, the rounding to fp8) is exact or correctly rounded, so nothing may differ."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["e4m3", "e5m2"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,k", [(1, 32), (3, 96), (129, 256), (5, 4128), (1000, 7168)])
def test_quantisation_is_byte_identical(rows, k, dtype, fmt, device):
    from mm_rs_with_catlass_b200.ops.mx import pack_scales, quantize_mxf8
    g = torch.Generator(device=device)
    g.manual_seed(rows + k)
    # magnitudes over the whole exponent range of the scale, exact fp8 limits, an all-zero block, infinities and NaNs
    x = torch.randn(rows, k, device=device, generator=g)
    x = (x * torch.exp2(torch.randint(-20, 14, (rows, k // 32, 1), device=device, generator=g).float()).expand(-1, -1, 32)
         .reshape(rows, k)).to(dtype)
    x[0, :32] = 0
    if k >= 96:
        x[-1, 32], x[-1, 40] = 448.0, -57344.0 if dtype != torch.float16 else -448.0
        x[-1, 64], x[-1, 70], x[-1, 75] = float("inf"), 3.0, -1000.0
    if rows > 2:
        x[1, 0], x[1, 5], x[1, 7], x[1, 9] = float("nan"), 500.0, -464.0, 61440.0 if dtype != torch.float16 else 60000.0
    q, s = quantize_mxf8(x, fmt)
    qr, sr = quantize_mxf8(x.cpu(), fmt)
    nan = torch.isnan(qr.float())
    assert torch.equal(s.cpu(), sr)
    assert torch.equal(torch.isnan(q.float()).cpu(), nan)
    assert torch.equal(q.cpu().view(torch.uint8)[~nan], qr.view(torch.uint8)[~nan])
    assert torch.equal(pack_scales(s).cpu(), pack_scales(sr))


@pytest.mark.parametrize("rows,kb", [(1, 1), (127, 3), (128, 4), (129, 5), (300, 34), (2, 224)])
def test_scale_packing(rows, kb, device):
    from mm_rs_with_catlass_b200.ops.mx import pack_scales
    s = torch.randint(0, 255, (rows, kb), device=device, dtype=torch.int32).to(torch.uint8)
    assert torch.equal(pack_scales(s).cpu(), pack_scales(s.cpu()))
