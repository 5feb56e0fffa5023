"""The latent-attention kernel for few query rows, where it can go wrong: page runs that end inside a sequence, at its end
or hold several; empty sequences at either end of the batch and between others; row counts below, at and above a chunk;
masked rows of the last page; reference maxima that move in every page, or never after the first."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(q_len, heads, lens, dtype, causal=False, gain=None, seed=0, extra_pages=0, stale=False):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops.mla import mla_decode_reference
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    batch, max_pages = len(lens), max(1, (max(lens) + 127) // 128) + extra_pages
    pages = batch * max_pages + 2
    u = lambda *shape: (torch.rand(*shape, device=dev, generator=g) * 2 - 1).to(dtype)
    qn, qr, ckv, kr = u(batch * q_len, heads, 512), u(batch * q_len, heads, 64), u(pages, 128, 512), u(pages, 128, 64)
    table = torch.randperm(pages, device=dev, generator=g)[:batch * max_pages].reshape(batch, max_pages).to(torch.int32)
    if gain is not None:
        # rotary keys that point along the queries, ever longer (or shorter) with the position in the sequence
        qr = qr.abs()
        ramp = torch.linspace(gain[0], gain[1], max_pages, device=dev)
        for b in range(batch):
            kr[table[b].long()] = (kr[table[b].long()].abs().float() * ramp[:, None, None]).to(dtype)
    if stale:
        # slots of the last page that no token was written to yet hold whatever the memory held before (the kernel reads
        # 16 keys at a time, so those up to the next multiple have to be finite)
        for b, n in enumerate(lens):
            page = table[b, (n - 1) // 128]
            first = ((n - 1) % 128 + 16) // 16 * 16
            for i, cache in enumerate((ckv, kr)):
                cache[page, first:] = (float("nan"), float("inf"))[(b + i) % 2]
    kv = torch.tensor(lens, dtype=torch.int32, device=dev)
    out = catcoc.mla_decode(qn, qr, ckv, kr, table, kv, q_len=q_len, causal=causal)
    torch.cuda.synchronize()
    raise_on_status(local_status(dev), "mla_decode")
    gold = mla_decode_reference(qn, qr, ckv, kr, table, kv, q_len=q_len, causal=causal)
    assert torch.isfinite(out.float()).all()
    # as for the general kernel: probabilities and the result are rounded to the operand type, |V| <= 1
    tol = 1.5e-2 if dtype == torch.bfloat16 else 3e-3
    err = (out.float() - gold).abs().max().item()
    assert err < tol, "max |err| %.4g (tolerance %.3g)" % (err, tol)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", [[1], [128], [129], [0, 5, 0], [0, 0, 300], [4096, 0, 17, 2050, 128], [700] * 150, [100] * 140,
                                  [(37 * i) % 900 for i in range(70)], [20000]])
@pytest.mark.parametrize("heads", [16, 5, 32, 17])
def test_runs_of_pages(lens, dtype, heads):
    _case(1, heads, lens, dtype, seed=sum(lens) + heads)


@pytest.mark.parametrize("q_len,heads", [(2, 16), (4, 8), (4, 4), (3, 9)])
@pytest.mark.parametrize("causal", [False, True])
def test_new_tokens_and_the_causal_mask(q_len, heads, causal):
    _case(q_len, heads, [260, 4, 128, 129, 1000, 131], torch.bfloat16, causal=causal, seed=q_len)


@pytest.mark.parametrize("heads", [16, 32])
@pytest.mark.parametrize("lens", [[129, 130, 257, 1, 131, 128, 132, 258], [129, 130, 257, 3] * 20])
def test_chunks_that_see_nothing_of_a_last_page(heads, lens):
    # two and four chunks of rows; the first tokens' chunks see no key of a last page of one to three keys, which is a piece of
    # its own in the short list (a page per CTA) and the start or end of a longer run in the other
    for dtype in (torch.bfloat16, torch.float16):
        _case(4, heads, lens, dtype, causal=True, seed=heads + len(lens))
    _case(3, heads, lens, torch.bfloat16, causal=True, seed=heads)


@pytest.mark.parametrize("gain", [(0.0, 40.0), (40.0, 0.0)])
def test_moving_reference_maximum(gain):
    _case(1, 16, [3000, 900], torch.bfloat16, gain=gain, seed=1)
    _case(1, 32, [2000, 50, 2500], torch.float16, gain=gain, seed=2)


def test_table_wider_than_the_sequences():
    _case(1, 16, [100, 300], torch.bfloat16, seed=3, extra_pages=5)


@pytest.mark.parametrize("heads", [16, 32])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_stale_slots_of_the_last_page_do_not_matter(heads, dtype):
    _case(1, heads, [1, 16, 17, 32, 96, 127, 128, 130, 300, 1000], dtype, seed=heads, stale=True)
    _case(4, heads, [4, 32, 132, 260], dtype, seed=heads + 1, causal=True, stale=True)
