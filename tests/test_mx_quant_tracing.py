"""``quantize_mxf8`` and ``pack_scales`` where a kernel cannot stand in for the PyTorch passes: an input that carries a gradient
(reverse or forward mode), a batched one under ``vmap``, and inputs that are only traced."""
import pytest
import torch


def _x(device, rows=6, k=96):
    g = torch.Generator().manual_seed(rows + k)
    return (torch.randn(rows, k, generator=g) * 3).to(device)


def test_fake_tensors_trace_without_a_gpu():
    from torch._subclasses.fake_tensor import FakeTensorMode
    from mm_rs_with_catlass_b200.ops.mx import pack_scales, quantize_mxf8
    with FakeTensorMode():
        q, s = quantize_mxf8(torch.empty(200, 256, device="cuda", dtype=torch.bfloat16), "e5m2")
        p = pack_scales(s)
    assert (tuple(q.shape), q.dtype, q.device.type) == ((200, 256), torch.float8_e5m2, "cuda")
    assert (tuple(s.shape), s.dtype) == ((200, 8), torch.uint8) and (tuple(p.shape), p.dtype) == ((2, 2, 512), torch.uint8)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradients_are_those_of_the_cpu(dtype):
    from mm_rs_with_catlass_b200.ops.mx import quantize_mxf8
    grads = []
    for device in ("cpu", "cuda"):
        x = _x(device).to(dtype).requires_grad_()
        q, s = quantize_mxf8(x)
        assert q.requires_grad and not s.requires_grad
        weight = torch.tensor([1.0, -2.0, 0.5], device=device).repeat(32)     # (a gradient of fp8 values is fp8 as well)
        (q.float() * weight).sum().backward()
        grads.append(x.grad.cpu())
        with torch.no_grad():
            assert not quantize_mxf8(x)[0].requires_grad
        assert not quantize_mxf8(x.detach())[0].requires_grad
    assert torch.equal(*grads) and bool((grads[0] != 0).all())


@pytest.mark.gpu
def test_transforms_and_tracers_see_the_passes():
    import torch.autograd.forward_ad as fwad
    from torch.fx.experimental.proxy_tensor import make_fx
    from mm_rs_with_catlass_b200.ops.mx import pack_scales, quantize_mxf8
    x = _x("cuda", 4, 64)
    q, s = quantize_mxf8(x)
    batched = torch.stack([x, x * 5, x - 1])
    qb, sb = torch.vmap(quantize_mxf8)(batched)
    assert torch.equal(qb[0].float(), q.float()) and torch.equal(sb[0], s)
    with fwad.dual_level():
        dual = quantize_mxf8(fwad.make_dual(x, torch.ones_like(x)))[0]
        assert fwad.unpack_dual(dual).tangent is not None

    def both(t):
        v, w = quantize_mxf8(t)
        return v.float(), pack_scales(w)

    graph = make_fx(both)(x)
    y = x * 7 - 2
    for got, want in zip(graph(y), both(y)):
        assert torch.equal(got, want)
    traced = torch.jit.trace(lambda t: both(t)[0], x, check_trace=False)
    assert torch.equal(traced(y), both(y)[0])
