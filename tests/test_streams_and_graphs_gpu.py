"""Calls that take scratch of their own and run as two overlapped launches: two streams at once never share it, and a
captured call replays on new contents of its inputs."""
import pytest
import torch

from mm_rs_with_catlass_b200.tiling.config import TilingConfig

pytestmark = pytest.mark.gpu


def _randn(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g).bfloat16()


def _call(name, seed):
    """(inputs to be rewritten, the call) of one route."""
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.tiling import chooser
    g = torch.Generator(device="cuda").manual_seed(seed)
    if name == "flash_decode":                       # sequences that are spread over several CTAs
        q, k, v = _randn(g, 2, 16, 2, 128), _randn(g, 2, 4, 3000, 128), _randn(g, 2, 4, 3000, 128)
        return [q, k], lambda: catcoc.flash_attention(q, k, v, causal=True)
    if name == "mla_rows":
        q, r, ckv, kr = _randn(g, 6, 16, 512), _randn(g, 6, 16, 64), _randn(g, 60, 128, 512), _randn(g, 60, 128, 64)
        table = torch.randperm(60, device="cuda", generator=g).view(6, 10).int()
        lens = torch.tensor([1280, 5, 700, 0, 129, 1000], device="cuda", dtype=torch.int32)
        return [q, ckv], lambda: catcoc.mla_decode(q, r, ckv, kr, table, lens)
    if name == "slice_k":
        a, b = _randn(g, 700, 512), _randn(g, 700, 256)
        return [a, b], lambda: catcoc.grouped_matmul_slice_k(a, b, [100, 100, 431, 700])
    if name == "attention_cut":                      # few tiles of queries over many keys
        from mm_rs_with_catlass_b200 import _native as N
        assert N.lib().catcoc_flash_attention_workspace_bytes(1, 8, 2, 160, 3000, 128, 1) > 0
        q, k, v = _randn(g, 1, 8, 160, 128), _randn(g, 1, 2, 3000, 128), _randn(g, 1, 2, 3000, 128)
        return [q, k], lambda: catcoc.flash_attention(q, k, v, causal=True)
    if name == "token_groups":
        a, b = _randn(g, 2000, 512), _randn(g, 8, 512, 1024)
        ends = torch.tensor([10, 300, 300, 800, 1001, 1500, 1600, 2000], device="cuda", dtype=torch.int32)
        t = TilingConfig(bn=256, cta_pair=2, twice=True, swap=True)
        return [a, b], lambda: catcoc.grouped_matmul(a, b, ends, tiling=t)
    if name == "mx_cut":
        from mm_rs_with_catlass_b200.ops import mx
        assert mx._cut(100, 1000, 16384) is not None
        x, w = _randn(g, 100, 16384), _randn(g, 1000, 16384)
        wq, ws = catcoc.quantize_mxf8(w)
        ws = catcoc.pack_scales(ws)

        def quantised():
            q, s = catcoc.quantize_mxf8(x)
            return catcoc.mxf8_matmul(q, catcoc.pack_scales(s), wq, ws)
        return [x], quantised
    if name.startswith("double_cut"):
        a, b = _randn(g, 1024, 2048), _randn(g, 2368, 2048)
        t = TilingConfig(bn=128, cta_pair=2, twice=True, swap=name.endswith("swapped"), cut_slices=4, cut_k=512)
        return [a, b], lambda: catcoc.matmul(a, b, trans_b=True, tiling=t)
    m, n, k = {"split_k": (64, 1024, 8192), "tail_cut": (1024, 5120, 6144), "padded_a": (200, 1000, 601),
               "padded_both": (200, 999, 601)}[name]
    a, b = _randn(g, m, k), _randn(g, k, n)
    tiling = chooser.choose("matmul", m, n, k, 1, a.dtype, tails=True)
    if name == "split_k":
        assert chooser.split_k(m, n, k, 2, tiling) is not None
    if name == "tail_cut":
        assert chooser.split_k(m, n, k, 2, tiling) is None and chooser.tail_cut(m, n, k, 2, tiling.effective_bn)[1] is not None
    return [a, b], lambda: catcoc.matmul(a, b)


ROUTES = ["split_k", "tail_cut", "padded_a", "padded_both", "flash_decode", "mla_rows", "slice_k", "double_cut", "double_cut_swapped",
          "attention_cut", "token_groups", "mx_cut"]


def _status():
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    torch.cuda.synchronize()
    raise_on_status(local_status(torch.device("cuda", 0)), "streams and graphs")


@pytest.mark.parametrize("name", ROUTES)
def test_two_streams(name):
    calls = [_call(name, seed)[1] for seed in (1, 2)]
    want = [c().clone() for c in calls]
    _status()
    streams = [torch.cuda.Stream() for _ in calls]
    got = [[], []]
    for _ in range(12):
        for s, c, out in zip(streams, calls, got):
            with torch.cuda.stream(s):
                out.append(c())
    _status()
    for w, out in zip(want, got):
        assert all(torch.equal(o, w) for o in out)


@pytest.mark.parametrize("name", ROUTES)
def test_captured_calls_replay_on_new_contents(name):
    inputs, call = _call(name, 3)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        first = call()
        second = call()                              # its scratch may be the first call's: behind it in the stream
    for scale in (1.0, 0.5, -2.0):
        for x in inputs:
            x.mul_(scale)
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        a, b = first.clone(), second.clone()
        want = call()
        assert torch.equal(a, want) and torch.equal(b, want)
    _status()
    del graph
