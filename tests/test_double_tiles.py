"""Double tiles (256 x 2 bn on a CTA pair): the plan covers the output once and deals it out evenly, the rule's choices are
legal (CPU); results are the bits of the one-accumulator kernel, whose products run in the same order along K (GPU)."""
import ctypes as C

import pytest
import torch

from mm_rs_with_catlass_b200 import _native as N
from mm_rs_with_catlass_b200.tiling import chooser
from mm_rs_with_catlass_b200.tiling.config import TilingConfig


@pytest.mark.parametrize("workers", [1, 7, 74])
@pytest.mark.parametrize("slices", [0, 3])
def test_plan_covers_the_output_once_and_evenly(workers, slices):
    buf = (C.c_int32 * (6 * 4096))()
    for m in (1, 257, 600, 2365, 8192):
        for n in (64, 200, 300, 700, 1696, 5120):
            for bn in (64, 192, 256):
                rt, ct = -(-m // 256), -(-n // bn)
                seen, cut, loads = {}, {}, []
                for w in range(workers):
                    cnt = N.lib().catcoc_double_plan_replay(m, n, bn, 4, workers, slices, w, 4096, buf)
                    load = 0
                    for kind, m0, n0, rows, cols, s in (buf[6 * i:6 * i + 6] for i in range(cnt)):
                        assert m0 % 256 == 0 and n0 % bn == 0 and rows == min(256, m - m0) and cols == min(bn * (2 if kind == 1 else 1), n - n0)
                        units = [(m0, n0)] + ([(m0, n0 + bn)] if kind == 1 else [])
                        assert kind != 1 or cols > bn                      # no half of a double tile is empty
                        for u in units:
                            if kind == 3:
                                cut.setdefault(u, []).append(s)
                            else:
                                seen[u] = seen.get(u, 0) + 1
                        load += 0 if kind == 3 else len(units)
                    loads.append(load)
                assert all(v == 1 for v in seen.values()) and all(sorted(v) == list(range(slices)) for v in cut.values())
                assert len(seen) + len(cut) == rt * ct and not (set(seen) & set(cut))
                assert len(cut) == (rt * ct % workers if slices else 0)
                assert max(loads) == -(-len(seen) // workers)              # no worker has more than its share


def test_choices_are_legal():
    hits = 0
    for m in (1, 64, 129, 300, 1024, 2365, 8144):
        for n in (8, 200, 1696, 8192, 28672):
            for k in (64, 520, 5120, 28672):
                for dt in (torch.bfloat16, torch.int8):
                    for major in (False, True):
                        for swap in (False, True):
                            t = chooser.choose("matmul", m, n, k, 1, dt, b_k_major=major, tails=True, doubles=True, swap=swap).validate()
                            assert swap or not t.swap
                            if t.twice:
                                hits += 1
                                assert major or t.swap or t.bn == 256
                                if t.cut_slices:
                                    assert t.cut_k * dt.itemsize % 128 == 0 and t.cut_k * (t.cut_slices - 1) < k <= t.cut_k * t.cut_slices
                            # a caller that does not ask for them gets what it got
                            old = chooser.choose("matmul", m, n, k, 1, dt, b_k_major=major, tails=True)
                            assert not old.twice and old == chooser.heuristic("matmul", m, n, k, 1, dt, major, True)
    assert hits > 100
    for bad in (dict(twice=True, bn=256), dict(twice=True, bn=100, cta_pair=2), dict(swap=True), dict(cut_slices=2, cut_k=64),
                dict(twice=True, bn=256, cta_pair=2, cut_slices=1, cut_k=64)):
        with pytest.raises(ValueError):
            TilingConfig(**bad).validate()
    with pytest.raises(ValueError):
        TilingConfig(twice=True, bn=256, cta_pair=2).validate(local=False)


def _check(what):
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    torch.cuda.synchronize()
    raise_on_status(local_status(torch.device("cuda", 0)), what)


def _operand(g, dtype, *shape):
    if dtype == torch.int8:
        return torch.randint(-127, 128, shape, device="cuda", dtype=dtype, generator=g)
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.int8])
@pytest.mark.parametrize("m,n,k,bn", [
    (1, 64, 64, 64),            # one unit, one K block
    (256, 512, 128, 256),       # one whole double tile, two K blocks: no block between the two ends of the tile
    (300, 1000, 72, 224),       # ragged everywhere; half a window behind the last whole one of a half
    (513, 336, 1296, 160), (1040, 2064, 520, 96), (2000, 40, 640, 128)])
def test_matches_the_single_accumulator_kernel(dtype, m, n, k, bn):
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    if dtype == torch.int8:
        m, n, k = (-(-x // 16) * 16 for x in (m, n, k))
    for ta in (False, True):
        for tb in (False, True):
            a, b = _operand(g, dtype, *((k, m) if ta else (m, k))), _operand(g, dtype, *((n, k) if tb else (k, n)))
            for out_dtype in ((torch.int32,) if dtype == torch.int8 else (dtype, torch.float32)):
                want = catcoc.matmul(a, b, trans_a=ta, trans_b=tb, out_dtype=out_dtype, tiling=TilingConfig(bn=256, cta_pair=1))
                for swap in (False, True):
                    out = torch.full_like(want, 7)
                    catcoc.matmul(a, b, trans_a=ta, trans_b=tb, out=out, tiling=TilingConfig(bn=bn, cta_pair=2, twice=True, swap=swap, swizzle=2))
                    _check("double tiles")
                    assert torch.equal(out, want), (ta, tb, out_dtype, swap)


@pytest.mark.gpu
@pytest.mark.parametrize("swap", [False, True])
def test_epilogues(swap):
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(3)
    m, n, k = 600, 1216, 768
    t, ref = TilingConfig(bn=224, cta_pair=2, twice=True, swap=swap), TilingConfig(bn=256, cta_pair=1)
    a, b = _operand(g, torch.bfloat16, m, k), _operand(g, torch.bfloat16, k, n) * 0.05
    c, bias = _operand(g, torch.bfloat16, m, n), torch.randn(n, device="cuda", generator=g)
    for kw in (dict(activation="gelu"), dict(alpha=0.5, bias_f32=bias), dict(alpha=-2.0, bias_f32=bias, activation="silu"), dict(alpha=0.5, beta=2.0, c=c)):
        if swap and "c" in kw:
            with pytest.raises(RuntimeError, match="without C"):
                catcoc.matmul(a, b, tiling=t, **kw)
            continue
        got, want = catcoc.matmul(a, b, tiling=t, **kw), catcoc.matmul(a, b, tiling=ref, **kw)
        _check("epilogues")
        # the same operations on the same sums, which the compiler may contract differently: one bf16 rounding apart at most
        assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 1e-3).all(), kw
    x, w = _operand(g, torch.int8, m, k), _operand(g, torch.int8, k, n)
    s1, s2 = torch.rand(m, device="cuda", generator=g) * 0.02, torch.rand(n, device="cuda", generator=g) * 0.01
    ib = torch.randint(-1000, 1000, (n,), device="cuda", dtype=torch.int32, generator=g)
    for kw in (dict(bias=ib), dict(scale_m=s1, scale_n=s2, bias=ib), dict(scale_n=s2, out_dtype=torch.float16), dict(scale_m=s1, out_dtype=torch.float32)):
        got, want = catcoc.matmul(x, w, tiling=t, **kw), catcoc.matmul(x, w, tiling=ref, **kw)
        _check("dequantisation")
        assert torch.equal(got, want), kw


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,bn,slices,cut_k", [(300, 700, 1104, 160, 3, 384), (1024, 2368, 2048, 128, 4, 512), (4000, 5008, 1024, 224, 2, 512)])
@pytest.mark.parametrize("swap", [False, True])
def test_cut_units(m, n, k, bn, slices, cut_k, swap):
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(m)
    t = TilingConfig(bn=bn, cta_pair=2, twice=True, swap=swap, cut_slices=slices, cut_k=cut_k)
    for tb in (True, False):
        a, b = _operand(g, torch.bfloat16, m, k), _operand(g, torch.bfloat16, *((n, k) if tb else (k, n)))
        got = catcoc.matmul(a, b, trans_b=tb, out_dtype=torch.float32, tiling=t)
        assert torch.equal(got, catcoc.matmul(a, b, trans_b=tb, out_dtype=torch.float32, tiling=t))      # the planned call
        want = catcoc.matmul(a, b, trans_b=tb, out_dtype=torch.float32, tiling=TilingConfig(bn=256, cta_pair=1))
        _check("cut units")
        # both are fp32 sums of exact products, in another order: k * 2^-24 relative to the sum of magnitudes (about sqrt(k))
        assert (got - want).abs().max().item() < k * 2.0 ** -24 * 4 * k ** 0.5
        x, w = _operand(g, torch.int8, m // 16 * 16, k), _operand(g, torch.int8, *((n, k) if tb else (k, n)))
        assert torch.equal(catcoc.matmul(x, w, trans_b=tb, tiling=t), catcoc.matmul(x, w, trans_b=tb, tiling=TilingConfig(bn=256, cta_pair=1)))
        _check("cut units")


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(130, 200, 128), (300, 584, 1056), (1024, 1536, 640)])
def test_block_scaled_cut_units(monkeypatch, m, n, k):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops import mx
    g = torch.Generator(device="cuda").manual_seed(k)
    ops, scaled = [], []
    for rows in (m, n):
        q, s = catcoc.quantize_mxf8(torch.randn(rows, k, device="cuda", generator=g), "e4m3")
        ops += [q, catcoc.pack_scales(s)]
        scaled.append((q, s))
    res = []
    for cut in (None, (2, -(-k // 256) * 128)) if k > 128 else (None,):
        monkeypatch.setattr(mx, "double_plan", lambda *a: (0.0, cut))
        mx._blocks.clear()
        res.append(catcoc.mxf8_matmul(*ops, out_dtype=torch.float32))
        _check("block-scaled")
    # fp32 sums in another order, as above; the operands' magnitudes are about one
    assert (res[0] - res[-1]).abs().max().item() < k * 2.0 ** -24 * 4 * k ** 0.5
    a, b = (catcoc.ops.mx.dequantize_mxf8(*x).double() for x in scaled)
    assert all((r - a @ b.t()).abs().max().item() < k * 2.0 ** -24 * 4 * k ** 0.5 for r in res)


@pytest.mark.gpu
@pytest.mark.parametrize("ends", [[0, 1, 70, 70, 333, 900], [900], [64, 128, 900]])
def test_weight_gradients(ends):
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(9)
    for m, n in ((256, 512), (264, 520), (520, 1408)):
        a, b = _operand(g, torch.bfloat16, 900, m), _operand(g, torch.bfloat16, 900, n)
        want = catcoc.grouped_matmul_slice_k(a, b, ends, tiling=TilingConfig(bn=256, cta_pair=1))
        got = catcoc.grouped_matmul_slice_k(a, b, ends, tiling=TilingConfig(bn=256, cta_pair=2, twice=True))
        _check("weight gradients")
        assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.int8])
@pytest.mark.parametrize("sizes", [
    [0, 1, 31, 32, 33, 160, 161, 192, 0], [512, 513, 0, 1025, 300], [777], [3] * 128, [0, 0, 256, 0]])
def test_token_groups(dtype, sizes):
    # groups at the edges of the widths (32, the single unit of 160, one tile of 512), empty ones, the most groups; their order
    # by width is the kernel's own affair
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    total, n, k = sum(sizes), 336, 256
    ends = torch.tensor(sizes).cumsum(0).to(torch.int32).cuda()
    t, ref = TilingConfig(bn=256, cta_pair=2, twice=True, swap=True), TilingConfig(bn=256, cta_pair=1)
    for tb in (False, True):
        a, b = _operand(g, dtype, total, k), _operand(g, dtype, *((len(sizes), n, k) if tb else (len(sizes), k, n)))
        if dtype == torch.int8:
            s1, s2 = torch.rand(total, device="cuda", generator=g), torch.rand(len(sizes), n, device="cuda", generator=g)
            res = [catcoc.grouped_quant_matmul(a, b, s1, s2, ends, trans_b=tb, tiling=x) for x in (t, ref)]
        else:
            res = [catcoc.grouped_matmul(a, b, ends, trans_b=tb, tiling=x) for x in (t, ref)]
            res += [catcoc.grouped_matmul(a, b, ends, trans_b=tb, out_dtype=torch.float32, tiling=x) for x in (t, ref)]
        _check("token groups")
        assert all(torch.equal(x, y) for x, y in zip(res[::2], res[1::2])), tb


@pytest.mark.gpu
def test_malformed_group_lists_stay_inside_the_output():
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(2)
    a, b = _operand(g, torch.bfloat16, 300, 128), _operand(g, torch.bfloat16, 4, 128, 256)
    ends = torch.tensor([200, 100, 1000, -5], dtype=torch.int32, device="cuda")      # decreasing, past the end, negative
    out = [catcoc.grouped_matmul(a, b, ends, out=torch.zeros(300, 256, device="cuda", dtype=torch.bfloat16), tiling=t)
           for t in (TilingConfig(bn=256, cta_pair=2, twice=True, swap=True), TilingConfig(bn=256, cta_pair=1))]
    _check("group lists")
    assert torch.equal(out[0], out[1])


def test_token_group_choice():
    for groups in (1, 8, 64, 200):
        for rows in (1, 100, 440, 3000):
            for n, k in ((1408, 1024), (4096, 4096), (8, 64)):
                for dt in (torch.bfloat16, torch.int8):
                    t = chooser.token_groups(groups * rows, groups, n, k, dt).validate()
                    assert not t.twice or (t.swap and t.bn == 256 and groups <= 128 and rows >= 128)
    assert chooser.token_groups(14080, 32, 4096, 2048, torch.bfloat16).swap
    assert not chooser.token_groups(1158, 64, 1408, 2048, torch.bfloat16).twice


@pytest.mark.gpu
def test_kept_argument_blocks_serve_other_buffers():
    # the same layouts at other addresses, at an address TMA cannot take, and back; contents of their own each time
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops import blas, mx
    g = torch.Generator(device="cuda").manual_seed(12)
    ends = torch.tensor([100, 130, 300], dtype=torch.int32, device="cuda")
    for kept in (blas._group_blocks, blas._slice_k_blocks, mx._blocks):
        kept.clear()
    for shift in (0, 0, 4, 0):
        a = torch.randn(300 * 256 + shift, device="cuda", generator=g).bfloat16()[shift:].view(300, 256)
        b = torch.randn(3, 256, 384, device="cuda", generator=g).bfloat16()
        want = torch.cat([a[x:y].float() @ b[i].float() for i, (x, y) in enumerate(((0, 100), (100, 130), (130, 300)))])
        got = catcoc.grouped_matmul(a, b, ends)
        assert (got.float() - want).abs().max().item() < 2.0 ** -7 * want.abs().max().item()
        x1, x2 = _operand(g, torch.int8, 300, 256), _operand(g, torch.int8, 3, 256, 384)
        s1, s2 = torch.rand(300, device="cuda", generator=g), torch.rand(3, 384, device="cuda", generator=g)
        deq = torch.cat([(x1[x:y].double() @ x2[i].double()) * s2[i] * s1[x:y, None] for i, (x, y) in enumerate(((0, 100), (100, 130), (130, 300)))])
        got = catcoc.grouped_quant_matmul(x1, x2, s1, s2, ends)
        assert (got.double() - deq).abs().max().item() < 2.0 ** -7 * deq.abs().max().item()
        c = torch.randn(300, 128, device="cuda", generator=g).bfloat16()
        want = torch.stack([a[x:y].float().t() @ c[x:y].float() for x, y in ((0, 10), (10, 10), (10, 300))])
        got = catcoc.grouped_matmul_slice_k(a, c, [10, 10, 300])
        assert (got.float() - want).abs().max().item() < 2.0 ** -7 * want.abs().max().item()
        qs = [catcoc.quantize_mxf8(torch.randn(r, 256, device="cuda", generator=g)) for r in (200, 96)]
        want = catcoc.ops.mx.dequantize_mxf8(*qs[0]) @ catcoc.ops.mx.dequantize_mxf8(*qs[1]).t()
        got = catcoc.mxf8_matmul(qs[0][0], catcoc.pack_scales(qs[0][1]), qs[1][0], catcoc.pack_scales(qs[1][1]))
        assert (got.float() - want).abs().max().item() < 2.0 ** -7 * want.abs().max().item()
        _check("kept blocks")
    assert blas._group_blocks and blas._slice_k_blocks and mx._blocks


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("m,n,k,bn", [(1, 64, 64, 64), (300, 1008, 208, 224), (513, 336, 1296, 160), (256, 512, 256, 256)])
def test_fp8(fmt, m, n, k, bn):
    # by an explicit tiling alone: no rule sends fp8 without block scales here
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(m + n)
    s1, s2 = torch.rand(m, device="cuda", generator=g) + 0.5, torch.rand(n, device="cuda", generator=g) + 0.5
    for tb in (True, False):
        a, b = _operand(g, fmt, m, k), _operand(g, fmt, *((n, k) if tb else (k, n)))
        for kw in (dict(out_dtype=torch.float32), dict(scale_m=s1, scale_n=s2)):
            got, want = (catcoc.matmul(a, b, trans_b=tb, tiling=TilingConfig(bn=x, cta_pair=p, twice=p == 2), **kw) for x, p in ((bn, 2), (256, 1)))
            _check("fp8")
            assert torch.equal(got, want), (tb, kw.keys())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.int8])
@pytest.mark.parametrize("bn", [96, 256])
def test_groups_of_rows_without_swapped_roles(dtype, bn):
    # ragged and uniform groups, by an explicit tiling alone; bn 96 leaves half a window behind the last whole one
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(bn)
    t, ref = TilingConfig(bn=bn, cta_pair=2, twice=True), TilingConfig(bn=256, cta_pair=1)
    sizes = [0, 1, 31, 300, 256, 0, 513]
    total, n, k = sum(sizes), 848, 256
    ends = torch.tensor(sizes).cumsum(0).to(torch.int32).cuda()
    for tb in (False, True):
        a, b = _operand(g, dtype, total, k), _operand(g, dtype, *((len(sizes), n, k) if tb else (len(sizes), k, n)))
        s1, s2 = torch.rand(total, device="cuda", generator=g), torch.rand(len(sizes), n, device="cuda", generator=g)
        got, want = (catcoc.grouped_quant_matmul(a, b, s1, s2, ends, trans_b=tb, tiling=x) if dtype == torch.int8 else
                     catcoc.grouped_matmul(a, b, ends, trans_b=tb, tiling=x) for x in (t, ref))
        _check("groups of rows")
        assert torch.equal(got, want), tb
        for ta in (False, True):
            a = _operand(g, dtype, *((3, k, 304) if ta else (3, 304, k)))
            got, want = (catcoc.batched_matmul(a, b[:3].contiguous(), trans_a=ta, trans_b=tb, tiling=x) for x in (t, ref))
            _check("uniform groups")
            assert torch.equal(got, want), (ta, tb)


@pytest.mark.gpu
@pytest.mark.parametrize("swap", [False, True])
def test_infinities_beside_a_group_or_behind_k_stay_outside(swap):
    import mm_rs_with_catlass_b200 as catcoc
    g = torch.Generator(device="cuda").manual_seed(21)
    t = TilingConfig(bn=256, cta_pair=2, twice=True, swap=swap)
    # groups of rows: those of one group
    sizes, n, k = [70, 200, 33, 300], 336, 200
    ends, bounds = torch.tensor(sizes).cumsum(0).to(torch.int32).cuda(), [0, 70, 270, 303, 603]
    a, b = _operand(g, torch.bfloat16, 640, k), _operand(g, torch.bfloat16, len(sizes), n, k)     # (K is no whole number of MMAs)
    a[603:] = float("inf")                                     # rows of no group
    want = catcoc.grouped_matmul(a, b, ends, trans_b=True, tiling=t)[:603].clone()
    assert want.isfinite().all()
    for i in range(len(sizes)):
        x = a.clone()
        x[bounds[i]:bounds[i + 1]] = float("inf")
        got = catcoc.grouped_matmul(x, b, ends, trans_b=True, tiling=t)
        for j in range(len(sizes)):
            if j != i:
                assert torch.equal(got[bounds[j]:bounds[j + 1]], want[bounds[j]:bounds[j + 1]]), (i, j)
    # ranges along K: those of one range, which end inside a K block
    if not swap:
        a, b = _operand(g, torch.bfloat16, 640, 264), _operand(g, torch.bfloat16, 640, 520)
        want = catcoc.grouped_matmul_slice_k(a, b, bounds[1:], tiling=t)
        for i in range(len(sizes)):
            x, y = a.clone(), b.clone()
            x[bounds[i]:bounds[i + 1]] = float("inf")
            y[bounds[i]:bounds[i + 1]] = float("nan")
            got = catcoc.grouped_matmul_slice_k(x, y, bounds[1:], tiling=t)
            assert all(torch.equal(got[j], want[j]) for j in range(len(sizes)) if j != i), i
    # columns behind K of operands inside wider buffers, whole and in slices
    for k in (72, 1096):
        wide = [torch.full((r, 1280), float("inf"), device="cuda", dtype=torch.bfloat16) for r in (600, 700)]
        for w in wide:
            w[:, :k] = _operand(g, torch.bfloat16, w.shape[0], k)
        for cut in (dict(), dict(cut_slices=3, cut_k=384)) if k > 72 else (dict(),):
            tc = TilingConfig(bn=96, cta_pair=2, twice=True, swap=swap, **cut)
            got, want = (catcoc.matmul(x, y, trans_b=True, out_dtype=torch.float32, tiling=tc)
                         for x, y in ([w[:, :k] for w in wide], [w[:, :k].contiguous() for w in wide]))
            assert want.isfinite().all() and torch.equal(got, want), (k, cut)
    _check("infinities")
