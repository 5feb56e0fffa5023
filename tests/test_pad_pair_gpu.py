"""Both operands of a product re-pitched by one launch: odd widths and bases, each storage order, the smallest sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,off", [(1, 3, 1, 0), (20, 868, 607, 0), (129, 257, 67, 1), (7, 1001, 2051, 3), (600, 30, 333, 0)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.int8])
def test_both_operands_padded(m, n, k, off, trans_a, trans_b, dtype):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops._common import _tma_legal, as_operands, local_status, raise_on_status
    g = torch.Generator(device="cuda").manual_seed(m * n + k)

    def stored(rows, cols):
        if dtype == torch.int8:
            flat = torch.randint(-127, 128, (rows * cols + off,), device="cuda", generator=g, dtype=dtype)
        else:
            flat = torch.randn(rows * cols + off, device="cuda", generator=g).to(dtype)
        return flat[off:].view(rows, cols)

    a, b = stored(*((k, m) if trans_a else (m, k))), stored(*((n, k) if trans_b else (k, n)))
    with torch.cuda.device(a.device):
        pads = as_operands(a, trans_a, b, trans_b)
    for x, o in zip((a, b), pads):
        assert o.ptr % 16 == 0 and (o.ld * x.element_size()) % 16 == 0
        if not _tma_legal(a) and not _tma_legal(b):
            row = torch.zeros(x.shape[0], o.ld, dtype=dtype, device="cuda")
            row[:, : x.shape[1]] = x
            start = o.ptr - o.tensor.data_ptr()
            copy = o.tensor.flatten()[start:start + row.numel() * row.element_size()]
            assert torch.equal(copy, row.view(torch.uint8).flatten())     # bytes stay the same, the padding is zero
    out = catcoc.matmul(a, b, trans_a=trans_a, trans_b=trans_b)
    torch.cuda.synchronize()
    raise_on_status(local_status(a.device), "padded pair")
    la, lb = (a.t() if trans_a else a), (b.t() if trans_b else b)
    ref = la.cpu().double() @ lb.cpu().double()
    if dtype == torch.int8:
        assert torch.equal(out.cpu().double(), ref)
    else:
        # one rounding to fp16 (2^-11 relative) after an fp32 sum of k exact products (k * 2^-24 of their magnitudes)
        bound = ref.abs() * 2.0 ** -11 + (la.cpu().double().abs() @ lb.cpu().double().abs()) * k * 2.0 ** -24 + 1e-7
        assert bool(((out.cpu().double() - ref).abs() <= bound).all())
