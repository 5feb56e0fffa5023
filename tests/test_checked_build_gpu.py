"""The bounds-checked build of the library (``CATCOC_CHECKED=1``): every workspace, peer, output
and accumulator offset of the kernels is compared with the extent of its buffer; an offset
outside is recorded in the status block (site, limit, offset) and the access is skipped. The
tests run it in child processes (the build is chosen when the library is loaded): the small-case
matrix must pass under it without a report, and an output whose extent is understated (the
buffer itself is large enough, so nothing is ever written out of bounds) must be reported with
its site and left untouched beyond the stated extent."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _child(code: str, env_extra=None, timeout=600):
    env = dict(os.environ, CATCOC_CHECKED="1", PYTHONPATH=REPO)
    env.update(env_extra or {})
    proc = subprocess.run([sys.executable, "-c", textwrap.dedent(code)], capture_output=True, text=True, env=env,
                          timeout=timeout, cwd=REPO)
    assert proc.returncode == 0, "child failed:\n%s\n%s" % (proc.stdout[-3000:], proc.stderr[-3000:])
    return [json.loads(l) for l in proc.stdout.splitlines() if l.startswith("{")]


def test_local_kernels_pass_under_the_checked_build():
    out = _child("""
        import json, torch
        import mm_rs_with_catlass_b200 as catcoc
        from mm_rs_with_catlass_b200 import _native as N
        from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
        from mm_rs_with_catlass_b200.utils.verify import assert_close
        assert N.lib().catcoc_is_checked_build() == 1
        dev = torch.device("cuda:0")
        for (m, n, k, pair, bn) in [(256, 512, 384, 1, 256), (23, 45, 68 + 4, 1, 64), (1000, 328, 136, 1, 128),
                                    (512, 512, 256, 2, 256), (300, 200, 264, 2, 128)]:
            a = torch.randn(m, k, device=dev).bfloat16()
            b = (torch.randn(k, n, device=dev) * 0.1).bfloat16()
            o = catcoc.matmul(a, b, tiling=catcoc.TilingConfig(bn=bn, cta_pair=pair))
            assert_close(o, a.float() @ b.float(), k=k, dtype=torch.bfloat16, what="%dx%dx%d" % (m, n, k))
        x1 = torch.randint(-127, 128, (200, 256), device=dev, dtype=torch.int32).to(torch.int8)
        x2 = torch.randint(-127, 128, (256, 384), device=dev, dtype=torch.int32).to(torch.int8)
        o = catcoc.matmul(x1, x2)
        assert torch.equal(o.cpu().long(), x1.cpu().long() @ x2.cpu().long())
        torch.cuda.synchronize()
        raise_on_status(local_status(dev), "checked build")
        print(json.dumps({"ok": True}))
    """)
    assert out and out[-1]["ok"]


def test_double_tiles_pass_under_the_checked_build():
    out = _child("""
        import json, torch
        import mm_rs_with_catlass_b200 as catcoc
        from mm_rs_with_catlass_b200 import _native as N
        from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
        from mm_rs_with_catlass_b200.utils.verify import assert_close
        T = catcoc.TilingConfig
        assert N.lib().catcoc_is_checked_build() == 1
        dev = torch.device("cuda:0")
        def r(*s):
            return torch.randn(*s, device=dev).bfloat16()
        def i8(*s):
            return torch.randint(-127, 128, s, device=dev, dtype=torch.int32).to(torch.int8)
        for swap in (False, True):
            for (m, n, k, bn, kw) in [(256, 512, 128, 256, {}), (300, 1001, 72, 224, {}), (1, 64, 64, 64, {}), (1024, 2368, 2048, 128, dict(cut_slices=4, cut_k=512)),
                                      (700, 703, 1024, 96, dict(cut_slices=2, cut_k=512, num_ctas=14))]:
                a, b = r(m, k), r(n, k) * 0.1
                t = T(bn=bn, cta_pair=2, twice=True, swap=swap, **kw)
                for dt in (torch.bfloat16, torch.float32):
                    assert_close(catcoc.matmul(a, b, trans_b=True, tiling=t, out_dtype=dt), a.float() @ b.float().t(), k=k, dtype=dt, what=str((m, n, k, swap)))
                x, w = i8(m, -(-k // 16) * 16), i8(n, -(-k // 16) * 16)
                assert torch.equal(catcoc.matmul(x, w, trans_b=True, tiling=t).cpu().long(), x.cpu().long() @ w.cpu().long().t())
            sizes = [0, 1, 33, 300, 256, 513]
            ends = torch.tensor(sizes).cumsum(0).to(torch.int32).to(dev)
            a, b = r(sum(sizes), 256), r(len(sizes), 256, 336) * 0.1
            got, at = catcoc.grouped_matmul(a, b, ends, tiling=T(bn=256, cta_pair=2, twice=True, swap=swap)), 0
            for i, s in enumerate(sizes):
                if s:
                    assert_close(got[at:at + s], a[at:at + s].float() @ b[i].float(), k=256, dtype=torch.bfloat16, what="group %d" % i)
                at += s
        a, b = r(900, 264), r(900, 520) * 0.1
        got = catcoc.grouped_matmul_slice_k(a, b, [70, 70, 900], tiling=T(bn=256, cta_pair=2, twice=True))
        for i, (x, y) in enumerate(((0, 70), (70, 900))):
            assert_close(got[2 * i], a[x:y].float().t() @ b[x:y].float(), k=900, dtype=torch.bfloat16, what="range %d" % i)
        assert not got[1].any()
        for m, n, k in ((300, 584, 1056), (100, 1000, 16384), (300, 15320, 160)):
            qs = [catcoc.quantize_mxf8(torch.randn(s, k, device=dev)) for s in (m, n)]
            want = catcoc.ops.mx.dequantize_mxf8(*qs[0]) @ catcoc.ops.mx.dequantize_mxf8(*qs[1]).t()
            assert_close(catcoc.mxf8_matmul(qs[0][0], catcoc.pack_scales(qs[0][1]), qs[1][0], catcoc.pack_scales(qs[1][1])), want, k=k, dtype=torch.bfloat16, what="mx")
        torch.cuda.synchronize()
        raise_on_status(local_status(dev), "checked build")
        print(json.dumps({"ok": True}))
    """)
    assert out and out[-1]["ok"]


@pytest.mark.parametrize("swap", [0, 1])
def test_double_tiles_report_an_understated_output_extent(swap):
    out = _child("""
        import json, torch
        from mm_rs_with_catlass_b200 import _native as N
        from mm_rs_with_catlass_b200.ops import _common as cm
        dev = torch.device("cuda:0")
        m, n, k = 512, 512, 128
        a, b = (torch.randn(m, k, device=dev).bfloat16() for _ in range(2))
        out = torch.full((m, n), 7.0, device=dev, dtype=torch.bfloat16)
        status = torch.zeros(8, dtype=torch.int32, device=dev)
        args = N.OpArgs()
        args.mode, args.in_fmt = N.MODE_LOCAL, N.IN_BF16
        args.M, args.N, args.K = m, n, k
        args.trans_b = 1
        args.a, args.lda, args.b, args.ldb = a.data_ptr(), k, b.data_ptr(), k
        args.out, args.ldc, args.out_fmt, args.partial_fmt = out.data_ptr(), n, N.FMT_BF16, N.FMT_BF16
        args.tiling.bn, args.tiling.cta_pair, args.tiling.twice, args.tiling.swap = 128, 2, 1, %d
        args.rank, args.W = 0, 1
        args.status = status.data_ptr()
        args.limit[N.LIM_OUT] = 256 * n * 2            # the caller claims half of the rows
        cm.launch(args, dev)
        torch.cuda.synchronize()
        print(json.dumps({"status": status.cpu().tolist(), "tail_untouched": bool((out[256:] == 7.0).all().item()),
                          "head_written": bool((out[:256] != 7.0).any().item())}))
    """ % swap, {"CATCOC_OUT_TMA": "0"})
    r = out[-1]
    assert r["status"][0] == 7 and r["status"][2] == 13 and r["status"][3] == 256 * 512 * 2, r
    assert r["tail_untouched"] and r["head_written"], r


def test_an_understated_output_extent_is_reported_and_nothing_is_written_past_it():
    out = _child("""
        import ctypes as C, json, torch
        import mm_rs_with_catlass_b200 as catcoc
        from mm_rs_with_catlass_b200 import _native as N
        from mm_rs_with_catlass_b200.ops import _common as cm
        dev = torch.device("cuda:0")
        m, n, k = 256, 256, 128
        a = torch.randn(m, k, device=dev).bfloat16()
        b = torch.randn(k, n, device=dev).bfloat16()
        out = torch.full((m, n), 7.0, device=dev, dtype=torch.bfloat16)
        status = torch.zeros(8, dtype=torch.int32, device=dev)
        args = N.OpArgs()
        args.mode, args.in_fmt = N.MODE_LOCAL, N.IN_BF16
        args.M, args.N, args.K = m, n, k
        args.a, args.lda, args.b, args.ldb = a.data_ptr(), k, b.data_ptr(), n
        args.out, args.ldc, args.out_fmt, args.partial_fmt = out.data_ptr(), n, N.FMT_BF16, N.FMT_BF16
        args.tiling.bn = 128
        args.rank, args.W = 0, 1
        args.status = status.data_ptr()
        args.limit[N.LIM_OUT] = 128 * n * 2            # the caller claims half of the rows
        cm.launch(args, dev)
        torch.cuda.synchronize()
        st = status.cpu().tolist()
        print(json.dumps({"status": st, "tail_untouched": bool((out[128:] == 7.0).all().item()),
                          "head_written": bool((out[:128] != 7.0).any().item())}))
    """, {"CATCOC_OUT_TMA": "0"})
    r = out[-1]
    assert r["status"][0] == 7, r            # STATUS_OUT_OF_RANGE
    assert r["status"][2] == 13, r           # SITE_OUT_STORE
    assert r["status"][3] == 128 * 256 * 2, r
    assert r["tail_untouched"] and r["head_written"], r


def test_register_stores_of_short_k_ranges_respect_the_extent():
    out = _child("""
        import ctypes as C, json, torch
        from mm_rs_with_catlass_b200 import _native as N
        from mm_rs_with_catlass_b200.ops import _common as cm
        dev = torch.device("cuda:0")
        m, n, k = 256, 256, 128
        a = torch.randn(k, m, device=dev).bfloat16()
        b = torch.randn(k, n, device=dev).bfloat16()
        out = torch.full((2, m, n), 7.0, device=dev, dtype=torch.bfloat16)
        status = torch.zeros(8, dtype=torch.int32, device=dev)
        args = N.OpArgs()
        args.mode, args.in_fmt = N.MODE_LOCAL, N.IN_BF16
        args.M, args.N, args.K = 2 * m, n, k
        args.trans_a = 1
        args.a, args.lda, args.b, args.ldb = a.data_ptr(), m, b.data_ptr(), n
        args.out, args.ldc, args.out_fmt, args.partial_fmt = out.data_ptr(), n, N.FMT_BF16, N.FMT_BF16
        args.tiling.bn = 128
        args.rank, args.W = 0, 1
        args.num_groups, args.group_rows, args.g_a_row_back = 2, m, m
        args.a_rows_total, args.a_k_total, args.b_n_total, args.b_k_total = m, k, n, k
        args.status = status.data_ptr()
        args.limit[N.LIM_OUT] = m * n * 2              # the caller claims the first group's output alone
        cm.launch_slice_k(args, [0, 64, 64, 128], dev)
        torch.cuda.synchronize()
        print(json.dumps({"status": status.cpu().tolist(), "second_untouched": bool((out[1] == 7.0).all().item()),
                          "first_written": bool((out[0] != 7.0).any().item())}))
    """, {"CATCOC_OUT_TMA": "0"})
    r = out[-1]
    assert r["status"][0] == 7 and r["status"][2] == 13 and r["status"][3] == 256 * 256 * 2, r
    assert r["second_untouched"] and r["first_written"], r


def test_the_launcher_refuses_a_tensor_map_over_an_understated_output():
    out = _child("""
        import json, torch
        from mm_rs_with_catlass_b200 import _native as N
        from mm_rs_with_catlass_b200.ops import _common as cm
        dev = torch.device("cuda:0")
        m, n, k = 256, 256, 128
        a = torch.randn(m, k, device=dev).bfloat16(); b = torch.randn(k, n, device=dev).bfloat16()
        out = torch.empty((m, n), device=dev, dtype=torch.bfloat16)
        status = torch.zeros(8, dtype=torch.int32, device=dev)
        args = N.OpArgs()
        args.mode, args.in_fmt = N.MODE_LOCAL, N.IN_BF16
        args.M, args.N, args.K = m, n, k
        args.a, args.lda, args.b, args.ldb = a.data_ptr(), k, b.data_ptr(), n
        args.out, args.ldc, args.out_fmt, args.partial_fmt = out.data_ptr(), n, N.FMT_BF16, N.FMT_BF16
        args.rank, args.W = 0, 1
        args.status = status.data_ptr()
        args.limit[N.LIM_OUT] = 100
        try:
            cm.launch(args, dev)
            print(json.dumps({"refused": False}))
        except N.NativeError as e:
            print(json.dumps({"refused": True, "code": e.code, "msg": str(e)}))
    """)
    assert out[-1]["refused"] and out[-1]["code"] == -1 and "smaller than" in out[-1]["msg"]


def test_fused_ops_on_two_gpus_pass_under_the_checked_build(gpu_count):
    if gpu_count < 2:
        pytest.skip("needs 2 GPUs")
    from test_fused_multi_gpu import _run
    cases = _run(2, "checked", {"CATCOC_CHECKED": "1", "CATCOC_TIMEOUT_MS": "3000"}, timeout=600)
    assert len(cases) >= 12


def test_event_ring_gives_a_chrome_trace_with_matched_begin_and_end_records(tmp_path):
    path = str(tmp_path / "trace.json")
    out = _child("""
        import json, torch
        import mm_rs_with_catlass_b200 as catcoc
        from mm_rs_with_catlass_b200.utils.trace import EventTrace
        dev = torch.device("cuda:0")
        a = torch.randn(1024, 512, device=dev).bfloat16()
        b = torch.randn(512, 1024, device=dev).bfloat16()
        with EventTrace(capacity=4096) as tr:
            catcoc.matmul(a, b, tiling=catcoc.TilingConfig(bn=256, cta_pair=1))
        recs = tr.records()
        n = tr.dump_chrome(%r)
        by = {}
        for r in recs:
            by.setdefault((r["cta"], r["role"], r["tile"]), []).append(r["phase"])
        epi = [k for k in by if k[1] == 2]
        print(json.dumps({"events": n, "dropped": tr.dropped, "epilogue_tiles": len(epi),
                          "paired": all(sorted(by[k]) == [0, 1] for k in epi),
                          "ordered": all(x["t_ns"] <= y["t_ns"] for x, y in zip(recs, recs[1:]))}))
    """ % path)
    r = out[-1]
    assert r["epilogue_tiles"] == 32 and r["paired"] and r["ordered"] and r["dropped"] == 0, r   # 8 x 4 tiles
    with open(path) as fh:
        trace = json.load(fh)
    assert len([e for e in trace["traceEvents"] if e.get("ph") in ("B", "E")]) == r["events"]


def test_event_ring_of_double_tiles():
    out = _child("""
        import json, torch
        import mm_rs_with_catlass_b200 as catcoc
        from mm_rs_with_catlass_b200.utils.trace import EventTrace
        dev = torch.device("cuda:0")
        a, b = (torch.randn(1000, 512, device=dev).bfloat16() for _ in range(2))
        for swap in (False, True):
            for cut in (dict(), dict(cut_slices=2, cut_k=256, num_ctas=14)):
                with EventTrace(capacity=4096) as tr:
                    catcoc.matmul(a, b, trans_b=True, tiling=catcoc.TilingConfig(bn=128, cta_pair=2, twice=True, swap=swap, **cut))
                by = {}
                for r in tr.records():
                    by.setdefault((r["cta"], r["role"], r["tile"]), []).append(r["phase"])
                count = lambda role: len([k for k in by if k[1] == role])
                print(json.dumps({"cut": bool(cut), "producers": count(0), "mma": count(1), "epilogues": count(2) + count(5), "dropped": tr.dropped,
                                  "paired": all(sorted(v) == [0, 1] for k, v in by.items() if k[1] != 0)}))
    """)
    # 4 x 8 units of 256 x 128: on 74 pairs 32 single units; on 7 pairs 4 of them are cut in two and the others are 14 double
    # tiles. Producers and epilogues of both CTAs, one issuer a pair.
    assert len(out) == 4
    for r in out:
        items, halves = (14 + 8, 28 + 8) if r["cut"] else (32, 32)
        assert r["paired"] and r["dropped"] == 0, r
        assert (r["mma"], r["producers"], r["epilogues"]) == (items, 2 * items, 2 * halves), r


def test_trace_counters_are_those_of_the_kernel_that_a_plain_call_runs():
    out = _child("""
        import json, torch
        import mm_rs_with_catlass_b200 as catcoc
        from mm_rs_with_catlass_b200.ops import gemm
        dev = torch.device("cuda:0")
        for m, n, k in ((1024, 5120, 6144), (300, 200, 264)):
            a, b = torch.randn(m, k, device=dev).bfloat16(), torch.randn(n, k, device=dev).bfloat16()
            trace, twice = torch.zeros(16, dtype=torch.int64, device=dev), []
            for t in (None, trace):
                gemm._plans.clear()
                catcoc.matmul(a, b, trans_b=True, trace=t)
                twice.append([p[0].tiling.twice for p in gemm._plans.values()])
            print(json.dumps({"twice": twice, "trace": trace.tolist()}))
    """, {"CATCOC_CHECKED": "0"})
    assert [r["twice"] for r in out] == [[[1], [1]], [[0], [0]]], out
    # lifetimes of the CTAs, and the double tile's second half
    assert all(r["trace"][8] > 0 for r in out) and out[0]["trace"][14] > 0 and out[0]["trace"][15] > 0, out
