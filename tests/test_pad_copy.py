"""The padded copy that makes an operand of any pitch and base fit for tensor loads: bytes of the rows, zeros behind them."""
import ctypes as C

import pytest
import torch

from mm_rs_with_catlass_b200 import _native as N

# around one 16-byte chunk; around the 107 chunks from which rows go by stretches of 128, full stretches, a little past them
WIDTHS = (1, 2, 15, 16, 17, 31, 374, 511, 512, 513, 1009, 1696, 1697, 2031, 2033, 2047, 2048, 2049, 3413, 4080, 4095, 4096, 4112)


def _job(rows, width, pitch, offset, extra, g):
    src = torch.randint(1, 256, (offset + rows * pitch + 64,), generator=g, dtype=torch.int32).to(torch.uint8).cuda()
    dst_pitch = -(-width // 16) * 16 + extra
    dst = torch.full((rows + 1, dst_pitch), 99, device="cuda", dtype=torch.uint8)
    want = torch.zeros(rows, dst_pitch, device="cuda", dtype=torch.uint8)
    want[:, :width] = src[offset:offset + rows * pitch].view(rows, pitch)[:, :width]
    return src, dst, want, (dst.data_ptr(), dst_pitch, src.data_ptr() + offset, pitch, rows, width)


def _check(job):
    src, dst, want, a = job
    assert torch.equal(dst[:-1], want) and bool((dst[-1] == 99).all()), a[1:2] + a[3:]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 3, 37])
def test_every_width_and_alignment(rows):
    g, st = torch.Generator().manual_seed(rows), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for width in WIDTHS:
        for pitch, offset, extra in ((width, 0, 0), (width, 1, 0), (width + 1, 2, 16), (width + 6, 7, 0), (width + 3, 8, 32), (width + 16, 13, 0)):
            job = _job(rows, width, pitch, offset, extra, g)
            N.check(N.lib().catcoc_pad2d(*job[3], st))
            _check(job)
    for w0, w1 in ((374, 31), (31, 2040), (512, 1025), (17, 4112), (2049, 2048), (4095, 100)):
        jobs = [_job(rows, w0, w0, 1, 0, g), _job(11, w1, w1 + 5, 3, 16, g)]
        N.check(N.lib().catcoc_pad2d_pair(*jobs[0][3], *jobs[1][3], st))
        _check(jobs[0])
        _check(jobs[1])
