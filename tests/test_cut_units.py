"""Double tiles whose last units are cut along K: the launch, its workspace and its fold agree on the units, or the call is
refused."""
import ctypes as C

import pytest

from mm_rs_with_catlass_b200 import _native as N


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
