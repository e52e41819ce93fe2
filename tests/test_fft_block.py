"""The FFT path's one-block kernel (csrc/xcorr_fft_block.cu) at every kind of transform length it uses --
each radix as a first, inner and last pass, single passes, odd and even matrix heights -- and on both sides of
the rules that choose it, against double-precision transforms."""
import re

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (rows, cols): lengths 2, 4, 8, 16, 2x3.., 48 = 3*16, 96 = 6*16, 160 = 10*16, 192 = 12*16, 256 = 16*16,
# 320 = 5*8*8, 384 = 3*16*8, 480 = 5*6*16, 512 = 16*8*4; the last two too large for one SM
SIZES = [(1, 1), (1, 7), (2, 3), (3, 2), (5, 24), (24, 5), (17, 33), (48, 40), (40, 48), (90, 75), (75, 90), (100, 20),
         (20, 100), (150, 10), (10, 150), (180, 9), (9, 185), (230, 6), (7, 231), (250, 8), (8, 250), (128, 60), (128, 128), (200, 200)]


def check(xc, mode, rows, cols, nl, nr, launches=None):
    gen = torch.Generator(device="cuda").manual_seed(rows * 1000 + cols)
    left = torch.rand((nl, rows, cols), generator=gen, device="cuda")
    right = torch.rand((nr, rows, cols), generator=gen, device="cuda")
    hints = xc.make_hints(kernel="fft")
    guard, n = 256, int(np.prod(xc.out_shape(mode, rows, cols, nl, nr)))
    whole = torch.full((n + 2 * guard,), -7.25e30, device="cuda")
    out = whole[guard:guard + n]
    out.fill_(float("nan"))
    wsb = xc.workspace_bytes(mode, rows, cols, nl, nr, hints)
    ws = torch.full((wsb + 2 * guard,), 77, dtype=torch.uint8, device="cuda")
    xc.reset_launch_count()
    xc.run_device(mode, left.data_ptr(), right.data_ptr(), out.data_ptr(), rows, cols, nl, nr, hints,
                  ws.data_ptr() + guard, wsb, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert bool((whole[:guard] == -7.25e30).all()) and bool((whole[guard + n:] == -7.25e30).all())
    assert bool((ws[:guard] == 77).all()) and bool((ws[guard + wsb:] == 77).all())
    if launches is not None:
        assert xc.launch_count() == launches
    # the text names what ran: lengths that hold the result, a power of two times at most one 3 and one 5, or cuFFT's
    text = xc.last_launch()
    p, q = (int(v) for v in re.search(r" transform=(\d+)x(\d+) ", text).groups())
    if " route=block " in text:
        assert "product=in-block" in text and ("right-spectra=once" in text) == (xc.launch_count() == 3)
        for length, need in ((p, 2 * rows - 1), (q, 2 * cols - 1)):
            odd = length // (length & -length)
            assert length >= need and length % 2 == 0 and odd in (1, 3, 5, 15)
    else:
        assert " route=cufft " in text and (p, q) == (2 * rows, 2 * cols) and xc.launch_count() == 4
    p = (2 * rows, 2 * cols)
    fl, fr = torch.fft.rfft2(left.double(), s=p), torch.fft.rfft2(right.double(), s=p).conj()
    f = (fl[:, None] * fr[None]).reshape(-1, *fl.shape[1:]) if mode == "n_to_m" else fl.repeat_interleave(nr // nl, 0) * fr
    want = torch.roll(torch.fft.irfft2(f, s=p), (rows - 1, cols - 1), (1, 2))[:, :2 * rows - 1, :2 * cols - 1].reshape(-1)
    # a few units of 2^-24 per pass: the bound the timed cases state for this path
    assert float((out.double() - want).norm() / want.norm()) <= 7e-7
    rms = want.pow(2).mean().sqrt()
    assert float((out.double() - want).abs().max() / torch.maximum(rms, want.abs().max())) <= 3.3e-6
    xc.check_device()


@pytest.mark.parametrize("rows,cols", SIZES)
def test_every_length(xc, rows, cols):
    check(xc, "n_to_mn", rows, cols, 3, 27)


def test_rules(xc):
    check(xc, "one_to_one", 60, 60, 1, 1, launches=2)          # forward transform of the left, pair
    check(xc, "one_to_one", 200, 40, 1, 1, launches=4)         # a few large transforms: spread over the GPU
    check(xc, "one_to_many", 200, 40, 1, 24, launches=2)
    check(xc, "n_to_m", 24, 20, 9, 14, launches=2)             # every pair transforms its right matrix
    check(xc, "n_to_m", 24, 20, 40, 30, launches=3)            # right spectra made once
    check(xc, "n_to_m", 200, 200, 2, 2, launches=4)            # too large for one SM


def test_capture(xc):
    left, right = torch.rand((1, 30, 30), device="cuda"), torch.rand((6, 30, 30), device="cuda")
    hints = xc.make_hints(kernel="fft")
    wsb = xc.workspace_bytes("one_to_many", 30, 30, 1, 6, hints)
    ws, out = torch.empty(wsb, dtype=torch.uint8, device="cuda"), torch.empty((6, 59, 59), device="cuda")

    def call():
        xc.run_device("one_to_many", left.data_ptr(), right.data_ptr(), out.data_ptr(), 30, 30, 1, 6, hints, ws.data_ptr(), wsb,
                      torch.cuda.current_stream().cuda_stream)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
        side.synchronize()
        want = out.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            call()
        out.zero_()
        right.mul_(0.5)
        graph.replay()
        side.synchronize()
    assert torch.equal(out, want * 0.5)
