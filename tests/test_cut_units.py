"""Double tiles whose last units are cut along K: the launch, its workspace and its fold agree on the units, or the call is
refused."""
import ctypes as C

import pytest
import torch

from mm_rs_with_catlass_b200 import _native as N
from mm_rs_with_catlass_b200.tiling.config import TilingConfig


def _args(m, n, k, in_fmt, **tiling):
    args = N.OpArgs()
    args.mode, args.in_fmt, args.M, args.N, args.K = N.MODE_LOCAL, in_fmt, m, n, k
    args.trans_b, args.lda, args.ldb, args.ldc = 1, k, k, n
    args.out_fmt = args.partial_fmt = N.FMT_F32
    args.W, args.sf_k_blocks = 1, -(-k // 128)
    args.tiling.cta_pair, args.tiling.twice = 2, 1
    for name, value in tiling.items():
        setattr(args.tiling, name, value)
    for name in ("a", "b", "out", "sfa", "sfb", "status"):
        setattr(args, name, 1 << 20)              # never read: the calls below are refused ahead of any launch
    return args


@pytest.mark.parametrize("bn", [64, 128, 160, 256])
def test_block_scaled_units_of_another_width_are_refused(bn):
    # the kernel's units are 192 columns whatever bn says; planes sized for 64 columns are too small for them
    for fmt in (N.IN_MXE4M3, N.IN_MXE5M2):
        args = _args(1024, 8192, 3072, fmt, bn=bn, cut_slices=3, cut_k=1024)
        assert N.lib().catcoc_double_workspace_bytes(C.byref(args)) == -1
        code = N.lib().catcoc_double_launch(C.byref(args), 1 << 20, None)
        assert code == -4 and b"192 columns" in N.lib().catcoc_last_error(), code


@pytest.mark.parametrize("num_ctas", [1, 2, 3])
def test_one_cta_is_a_pair(num_ctas):
    # 3 x 4 units of 256 x 192 on one pair: nothing is left over to cut; on a grid of no pair the deal divided by zero
    args = _args(700, 700, 1024, N.IN_BF16, bn=192, cut_slices=2, cut_k=512, num_ctas=num_ctas)
    assert N.lib().catcoc_double_workspace_bytes(C.byref(args)) == 0


def test_a_refused_workspace_is_an_error():
    from mm_rs_with_catlass_b200.ops import _common as cm
    args = _args(700, 700, 1024, N.IN_MXE4M3, bn=64, cut_slices=2, cut_k=512)
    with pytest.raises(ValueError, match="no workspace"):
        cm.launch_double(args, torch.device("cpu"))


@pytest.mark.gpu
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("num_ctas", [1, 2, 3, 14])
def test_few_ctas(num_ctas, swap):
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(num_ctas)
    a, b = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((600, 1024), (700, 1024)))
    t = dict(bn=160, cta_pair=2, twice=True, swap=swap, num_ctas=num_ctas)
    got = catcoc.matmul(a, b, trans_b=True, out_dtype=torch.float32, tiling=TilingConfig(cut_slices=2, cut_k=512, **t))
    want = catcoc.matmul(a, b, trans_b=True, out_dtype=torch.float32, tiling=TilingConfig(**t))
    torch.cuda.synchronize()
    # the same products summed in another order: fp32 rounding of sums of k terms of size sqrt(k) at most
    assert (got - want).abs().max().item() <= 2.0 ** -24 * 1024 * 4 * 32
