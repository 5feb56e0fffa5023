"""Activations of the GEMM epilogues value by value: the whole range, infinities and NaN among ordinary neighbours, in every
tile form."""
import math

import pytest
import torch

import mm_rs_with_catlass_b200 as catcoc
from mm_rs_with_catlass_b200.tiling.config import TilingConfig

TILINGS = {"single": dict(bn=64, cta_pair=1), "pair": dict(bn=128, cta_pair=2),
           "double": dict(bn=64, cta_pair=2, twice=True), "swapped": dict(bn=64, cta_pair=2, twice=True, swap=True)}


@pytest.mark.gpu
@pytest.mark.parametrize("tiling", sorted(TILINGS))
@pytest.mark.parametrize("act", ["relu", "silu", "gelu"])
def test_values(tiling, act):
    x = torch.cat([torch.linspace(-100, 100, 301), torch.linspace(-2, 2, 64), torch.tensor([0.0, math.inf, -5.0, -math.inf, math.nan, 1e38, -1e38, 1e-38])])
    x = x[torch.randperm(x.numel(), generator=torch.Generator().manual_seed(1))].bfloat16()
    n, m, k = x.numel(), 70, 16
    a, b = torch.zeros(m, k, dtype=torch.bfloat16), torch.zeros(k, n, dtype=torch.bfloat16)
    a[:, 0], b[0] = 1, x                                     # the accumulator of column j is x[j], exactly
    tb = tiling == "double"                                  # halves of 64 columns take B with K along its rows
    out = catcoc.matmul(a.cuda(), (b.t().contiguous() if tb else b).cuda(), trans_b=tb, activation=act, out_dtype=torch.float32,
                        tiling=TilingConfig(swizzle=2, **TILINGS[tiling])).cpu()
    assert torch.equal(out.isnan(), out.isnan()[:1].expand_as(out)) and torch.equal(out.nan_to_num(), out.nan_to_num()[:1].expand_as(out))
    got, v = out[0].double(), x.double()
    if act == "relu":
        fin = ~v.isnan()
        assert torch.equal(got[fin], v[fin].clamp_min(0))
        return
    if act == "silu":
        want = v / (1 + torch.exp(-v))
        # exp in hardware: 2 + 1.173 |x| units of 2^-23, the sum and the quotient one each; below 2^-125 only the size
        tol = want.abs() * (4 + 1.173 * v.abs()) * 2.0 ** -23 + 2.0 ** -119
    else:
        want = 0.5 * v * (1 + torch.tanh(0.7978845608028654 * v * (1 + 0.044715 * v * v)))
        tol = 0.5 * v.abs() * 2.0 ** -10                     # hardware tanh: a relative error of 2^-11
    bad = v.isnan() | (v == -math.inf)                       # -inf / inf, -inf * 0
    assert bool(got[v.isnan()].isnan().all()) and bool(got[v == -math.inf].isnan().all() or (got[v == -math.inf] == 0).all())
    ok = ~bad & v.isfinite() & (want.abs() < 1e37)
    assert bool(((got - want).abs()[ok] <= tol[ok]).all()), ((got - want).abs() - tol)[ok].max()
    assert bool((got[v == math.inf] == math.inf).all())


@pytest.mark.gpu
@pytest.mark.parametrize("tiling", sorted(TILINGS))
def test_silu_keeps_the_sign_of_zero(tiling):
    # minus one times an accumulator of zero, and a bias: minus zero where the bias is
    x = torch.tensor([-0.0, 0.0, -1e-38, 1e-38, -2.0, -0.0, 3.0, -0.0] * 12).cuda()
    m, n, k = 40, x.numel(), 16
    a, b = torch.zeros(m, k, device="cuda", dtype=torch.bfloat16), torch.zeros(n, k, device="cuda", dtype=torch.bfloat16)
    out = catcoc.matmul(a, b, trans_b=True, activation="silu", out_dtype=torch.float32, alpha=-1.0, bias_f32=x,
                        tiling=TilingConfig(swizzle=2, **TILINGS[tiling]))
    assert torch.equal(out.signbit(), x.signbit().expand(m, n))
