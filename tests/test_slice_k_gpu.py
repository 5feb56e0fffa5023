"""Products over ragged ranges of K in one launch: ranges that end inside a K block, on one and on an MMA boundary, empty
and one-row groups, more groups than one batch of tensor maps holds, output rows and columns that are not whole tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(m, n, sizes, dtype, seed=0, poison=False):
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    from mm_rs_with_catlass_b200.utils.verify import assert_close
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    total = sum(sizes)
    a = torch.randn(total, m, device=dev, generator=g).to(dtype)
    b = torch.randn(total, n, device=dev, generator=g).to(dtype)
    ends, acc = [], 0
    for s in sizes:
        acc += s
        ends.append(acc)
    if poison:                       # an infinity in the row behind the first group must not reach its result
        a[ends[0]] = float("inf")
        b[ends[0]] = float("nan")
    out = catcoc.grouped_matmul_slice_k(a, b, ends)
    torch.cuda.synchronize()
    raise_on_status(local_status(dev), "slice_k")
    begin = 0
    for i, end in enumerate(ends):
        if not (poison and i == 1):
            gold = a[begin:end].float().t() @ b[begin:end].float()
            assert_close(out[i], gold, k=max(1, end - begin), dtype=dtype, what="group %d" % i)
        begin = end


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n", [(256, 256), (128, 64), (512, 1408), (200, 136), (1024, 72)])
def test_ragged_ranges(dtype, m, n):
    _check(m, n, [1, 0, 63, 64, 65, 16, 17, 300, 0, 128, 5], dtype, seed=m + n)


def test_more_groups_than_one_batch_of_maps():
    _check(256, 128, [(7 * i) % 90 for i in range(113)], torch.bfloat16, seed=3)


def test_neighbouring_rows_are_not_read():
    _check(256, 256, [100, 30, 77], torch.bfloat16, seed=4, poison=True)
    _check(136, 256, [100, 30, 77], torch.bfloat16, seed=5, poison=True)


def test_short_and_long_ranges_store_by_different_paths():
    # ranges of up to 256 rows store from registers, longer ones through the staging buffers; rows that do not start on a
    # 32-byte sector (n = 328) never do
    _check(256, 512, [256, 257, 40, 700, 256], torch.bfloat16, seed=6)
    _check(256, 328, [256, 40, 700], torch.float16, seed=7)


@pytest.mark.parametrize("rows", [0, 40])
def test_every_group_empty(rows):
    # a rank of a mixture of experts that received no token in this step: zeros, whether or not rows are there
    import mm_rs_with_catlass_b200 as catcoc
    from mm_rs_with_catlass_b200.ops._common import local_status, raise_on_status
    a, b = (torch.randn(rows, c, device="cuda").bfloat16() for c in (256, 128))
    torch.full((4, 256, 128), float("nan"), device="cuda", dtype=torch.bfloat16)     # what the allocator hands out next
    out = catcoc.grouped_matmul_slice_k(a, b, [0, 0, 0, 0])
    assert tuple(out.shape) == (4, 256, 128) and bool((out == 0).all())
    assert catcoc.grouped_matmul_slice_k(a, b, torch.zeros(3, dtype=torch.int64), out_dtype=torch.float32).abs().sum().item() == 0
    raise_on_status(local_status(a.device), "slice_k")


def test_an_integer_output_is_refused_however_many_groups():
    import mm_rs_with_catlass_b200 as catcoc
    a, b = (torch.randn(96, c, device="cuda").bfloat16() for c in (256, 128))
    for ends in ([96], [40, 96]):
        with pytest.raises(ValueError, match="int32"):
            catcoc.grouped_matmul_slice_k(a, b, ends, out_dtype=torch.int32)


def test_ends_are_whole_numbers():
    import mm_rs_with_catlass_b200 as catcoc
    a, b = (torch.randn(96, c, device="cuda").bfloat16() for c in (256, 128))
    for ends in ([96.0], [40.5, 96.0], torch.tensor([40.5, 96.0])):
        with pytest.raises(TypeError):
            catcoc.grouped_matmul_slice_k(a, b, ends)
    whole = catcoc.grouped_matmul_slice_k(a, b, torch.tensor([40, 96]))
    assert torch.equal(whole, catcoc.grouped_matmul_slice_k(a, b, list(torch.tensor([40, 96], dtype=torch.int32))))
