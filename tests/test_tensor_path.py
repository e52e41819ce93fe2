"""The tensor-core route of the automatic choice (csrc/xcorr_tensor.cu): when it is taken (CPU, from the
plan text), and its results against the CPU oracle at the edges of its tiles (GPU)."""
import os

import numpy as np
import pytest

from conftest import file_to_grouped, grouped_to_file, seeded_inputs

# shapes the planner sends to the tensor cores: one and two Toeplitz rows taken together, one and two
# matrices interleaved, several matrices B, mirrored results, one to four column chunks, odd sizes, tiles of
# x shifts, row slices with partial images, groups that fill no tile
ROUTED = [("n_to_m", 27, 43, 9, 35), ("n_to_m", 32, 32, 32, 64), ("n_to_m", 113, 19, 11, 45), ("n_to_mn", 48, 48, 4, 256),
          ("n_to_mn", 82, 23, 15, 900), ("one_to_one", 225, 132, 1, 1), ("one_to_one", 256, 256, 1, 1), ("n_to_m", 14, 114, 43, 17),
          ("one_to_many", 32, 121, 1, 228), ("one_to_many", 64, 64, 1, 129), ("n_to_mn", 41, 50, 3, 333), ("one_to_many", 128, 128, 1, 8)]


def plan(xc, shape, hints=None):
    return xc.describe_plan(*shape, hints)


@pytest.mark.parametrize("shape", ROUTED)
def test_route_and_what_keeps_to_the_tile_kernel(xc, shape):
    assert plan(xc, shape).startswith("kernel=tensor<")
    # hints that ask for another plan are obeyed; `reproducible` is met as it is (no atomically added sums)
    for hints in (dict(kernel="tile"), dict(overlap_rows=1), dict(schedule=1), dict(class_lanes=32), dict(kernel="overlap_wise")):
        assert "kernel=tensor" not in plan(xc, shape, xc.make_hints(**hints)), hints
    # one plan, the one that runs
    assert plan(xc, shape).count("kernel=") == 1 and plan(xc, shape).endswith("}")
    # the workspace stays what the tile plan asks for
    assert xc.workspace_bytes(*shape) == xc.workspace_bytes(*shape, xc.make_hints(kernel="tile"))


@pytest.mark.parametrize("shape", [("one_to_one", 16, 16, 1, 1), ("one_to_one", 100, 75, 1, 1), ("n_to_m", 32, 32, 8, 8),
                                   ("one_to_many", 16, 16, 1, 1000), ("one_to_many", 4, 600, 1, 300), ("n_to_mn", 87, 43, 61, 61)])
def test_small_calls_and_finer_sums_stay(xc, shape):
    """Too little work, sizes the route does not take, and plans whose many short sums round less."""
    assert "kernel=tensor" not in plan(xc, shape)


# timed at least as fast on the tile kernel (us on one B200, tile kernel / tensor cores): few rows, of which several of a
# warp wrap at once, and shapes whose blocks fill little more than a whole number of waves
TILE_FASTER = [("one_to_many", 8, 158, 1, 411), ("one_to_many", 69, 68, 1, 67), ("n_to_m", 13, 72, 2, 1482), ("n_to_mn", 12, 94, 2, 752),   # 47/54 112/115 169/187 52/60
               ("n_to_mn", 10, 148, 3, 387), ("one_to_many", 8, 85, 1, 781), ("one_to_many", 40, 200, 1, 30), ("n_to_mn", 93, 75, 59, 59)]   # 65/61 38/37 123/169 194/206


@pytest.mark.parametrize("shape", TILE_FASTER)
def test_calls_that_gain_nothing_stay(xc, shape):
    assert plan(xc, shape).startswith("kernel=tile<")


def run(xc, torch, shape, left, right, hints=None, workspace=True):
    mode, rows, cols, nl, nr = shape
    guard = 256
    out_shape = xc.out_shape(mode, rows, cols, nl, nr)
    n = int(np.prod(out_shape))
    dl, dr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    whole = torch.full((n + 2 * guard,), -7.25e30, dtype=torch.float32, device="cuda")
    out = whole[guard:guard + n]
    out.fill_(float("nan"))
    wsb = xc.workspace_bytes(mode, rows, cols, nl, nr, hints) if workspace else 0
    ws = torch.empty(wsb + 16, dtype=torch.uint8, device="cuda")
    xc.run_device(mode, dl.data_ptr(), dr.data_ptr(), out.data_ptr(), rows, cols, nl, nr, hints,
                  ws.data_ptr() if wsb else 0, wsb, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert bool((whole[:guard] == -7.25e30).all()) and bool((whole[guard + n:] == -7.25e30).all())
    return out.reshape(out_shape).cpu().numpy()


def reference(oracle, shape, left, right):
    mode, nl = shape[0], shape[3]
    threads = os.cpu_count() or 1
    if mode == "n_to_mn":
        return file_to_grouped(oracle.run(mode, left, grouped_to_file(right, nl), acc64=True, threads=threads), nl)
    return oracle.run(mode, left, right, acc64=True, threads=threads)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ROUTED)
def test_results_against_the_oracle(xc, oracle, shape):
    """2-norm within 3.5 units of 2^-24: about one for the rounding towards zero inside tensor memory, 0.2
    sqrt(row sums) for the sums in registers (at most 1024 / 4 of them here) and a margin; two runs agree bit for bit."""
    torch = pytest.importorskip("torch")
    mode, rows, cols, nl, nr = shape
    left, right = seeded_inputs(rows, cols, nl, nr, 31 * rows + cols)
    got = run(xc, torch, shape, left, right)
    assert xc.last_launch().startswith("kernel=tensor<"), xc.last_launch()
    assert xc.last_launch() == plan(xc, shape)
    want = reference(oracle, shape, left, right)
    assert not np.isnan(got).any()
    err = np.linalg.norm((got - want).ravel()) / np.linalg.norm(want.ravel())
    assert err <= 3.5 * 2.0 ** -24, (err * 2 ** 24, xc.last_launch())
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    assert np.array_equal(got, run(xc, torch, shape, left, right, xc.make_hints(reproducible=1)))
    xc.check_device()


# all builds: 64, 128 and 256 result columns, one and several column chunks
PRECISION = [("n_to_m", 27, 43, 9, 35), ("n_to_mn", 48, 48, 12, 384), ("n_to_m", 32, 32, 32, 64), ("one_to_many", 64, 64, 1, 512),
             ("one_to_one", 256, 256, 1, 1), ("one_to_many", 96, 96, 1, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uniform", "normal", "sparse"])
@pytest.mark.parametrize("shape", PRECISION)
def test_no_less_precise_than_fmas(xc, shape, kind):
    """Errors against the double-precision kernel, by the number of products of a result (overlaps of 1, 2..3, 4..7, ...
    elements), beside the tile kernel's FMAs: no larger in the 2-norm, over the whole result and in any class of 2000
    results or more (5 % and 0.03 units of 2^-24 for the sample), and without a bias towards zero for small sums: FMAs
    have none, sums of up to 31 products showed 0.11 units, one accumulator for large and small products 0.57 and more."""
    torch = pytest.importorskip("torch")
    mode, rows, cols, nl, nr = shape
    rng = np.random.default_rng(rows * cols + nr)

    def operand(n):
        a = rng.standard_normal((n, rows, cols)) if kind == "normal" else rng.random((n, rows, cols))
        return (a * (rng.random(a.shape) < 0.03) if kind == "sparse" else a).astype(np.float32)

    left, right = operand(nl), operand(nr)
    dl, dr = torch.from_numpy(left).cuda().double(), torch.from_numpy(right).cuda().double()
    want = torch.empty(xc.out_shape(mode, rows, cols, nl, nr), dtype=torch.float64, device="cuda")
    xc.run_device_f64(mode, dl.data_ptr(), dr.data_ptr(), want.data_ptr(), rows, cols, nl, nr, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = want.cpu().numpy()
    count = np.outer(rows - np.abs(np.arange(1 - rows, rows)), cols - np.abs(np.arange(1 - cols, cols)))
    size_class = np.broadcast_to(np.log2(count).astype(int), want.shape).ravel()
    w = want.ravel()

    def per_class(v):
        return np.bincount(size_class, weights=v)

    err, whole, bias = {}, {}, {}
    for name, hints in (("tile", xc.make_hints(kernel="tile")), ("auto", None)):
        e = run(xc, torch, shape, left, right, hints).astype(np.float64).ravel() - w
        assert xc.last_launch().startswith("kernel=tensor<" if name == "auto" else "kernel=tile<"), xc.last_launch()
        whole[name] = np.linalg.norm(e) / np.linalg.norm(w) * 2.0 ** 24
        err[name] = np.sqrt(per_class(e * e) / np.maximum(per_class(w * w), 1e-300)) * 2.0 ** 24
        bias[name] = per_class(e * np.sign(w)) / np.maximum(per_class(np.abs(w)), 1e-300) * 2.0 ** 24
    assert whole["auto"] <= 1.02 * whole["tile"], whole
    for c in range(len(err["auto"])):
        if np.count_nonzero(w[size_class == c]) < 2000:
            continue
        assert err["auto"][c] <= 1.05 * err["tile"][c] + 0.03, (2 ** c, err)
        if c < 5:
            assert abs(bias["auto"][c]) <= 0.3, (2 ** c, bias)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [("n_to_m", 27, 43, 9, 35), ("n_to_mn", 48, 48, 4, 256), ("one_to_one", 225, 132, 1, 1),
                                   ("one_to_one", 256, 256, 1, 1), ("n_to_m", 20, 48, 33, 63)])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30, 1e-30])
def test_operands_outside_the_range_of_the_split(xc, oracle, shape, value):
    """Infinities and NaN meet exactly the products of the definition (the padding's zeros are not multiplied
    with them); very large and very small matrices keep their precision."""
    torch = pytest.importorskip("torch")
    mode, rows, cols, nl, nr = shape
    left, right = seeded_inputs(rows, cols, nl, nr, 9)
    if abs(value) < 1:
        right[nr // 2] *= np.float32(value)                       # a whole matrix far below the others
        left[0] *= np.float32(1e8)
    else:
        right[nr // 2, rows // 3, cols - 1] = value
        left[nl - 1, rows - 1, 0] = 0.0                           # inf * 0 where they meet
    got = run(xc, torch, shape, left, right)
    assert xc.last_launch().startswith("kernel=tensor<"), xc.last_launch()
    with np.errstate(all="ignore"):
        want = reference(oracle, shape, left, right)
    for g, w in zip(got, want):                                   # per result matrix
        finite = np.isfinite(w)
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(g[~finite], w[~finite].astype(np.float32), equal_nan=True)
        if finite.any():
            scale = np.abs(w[finite]).max()
            assert np.abs(g[finite] - w[finite]).max() <= 1e-5 * scale


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [("one_to_many", 64, 64, 1, 512), ("one_to_one", 256, 256, 1, 1), ("n_to_m", 32, 32, 32, 64)])
def test_a_nan_costs_no_more_than_a_few_times_the_tile_kernel(xc, shape):
    """One NaN in the left matrix sends every block that meets it through the definition: timed 3.2, 4.1 and 4.7 times
    the tile kernel (44, 54 and 28 times without reuse of what is read).  Ten times is the line."""
    torch = pytest.importorskip("torch")
    mode, rows, cols, nl, nr = shape
    left, right = seeded_inputs(rows, cols, nl, nr, 8)
    left[:, 0, 0] = np.nan
    dl, dr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    out = torch.empty(xc.out_shape(*shape), dtype=torch.float32, device="cuda")
    times = {}
    for kernel in ("tile", "auto"):
        hints = xc.make_hints(kernel=kernel)
        wsb = xc.workspace_bytes(*shape, hints)
        ws = torch.empty(wsb + 16, dtype=torch.uint8, device="cuda")
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            xc.run_device(mode, dl.data_ptr(), dr.data_ptr(), out.data_ptr(), rows, cols, nl, nr, hints,
                          ws.data_ptr() if wsb else 0, wsb, torch.cuda.current_stream().cuda_stream)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times[kernel] = best
        assert xc.last_launch().startswith("kernel=tensor<" if kernel == "auto" else "kernel=tile<")
    assert times["auto"] <= 10.0 * times["tile"], times


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [("n_to_m", 27, 43, 9, 35), ("n_to_mn", 48, 48, 16, 512), ("one_to_one", 225, 132, 1, 1)])
@pytest.mark.parametrize("kind", ["far below the largest", "small products", "large"])
def test_elements_and_products_at_the_ends_of_the_range(xc, oracle, shape, kind):
    """Results that meet only elements below 2^-110 of matrices whose other elements are ordinary, results of matrices
    whose products come near the smallest normal number, and elements up to 2^49 keep the precision of single-precision
    sums: 0.2 sqrt(n) units of 2^-24 in the 2-norm for n products taken in sequence, and one for the margin."""
    torch = pytest.importorskip("torch")
    mode, rows, cols, nl, nr = shape
    left, right = seeded_inputs(rows, cols, nl, nr, 17)
    left, right = left + np.float32(0.5), right + np.float32(0.5)
    if kind == "far below the largest":
        left[:, rows - 1] *= np.float32(1e-35)                     # met alone by the first row of every right matrix
    elif kind == "small products":
        left, right = left * np.float32(2.0 ** -55), right * np.float32(2.0 ** -59)
    else:
        left, right = left * np.float32(2.0 ** 48), right * np.float32(2.0 ** 48)
    got = run(xc, torch, shape, left, right).astype(np.float64)
    assert xc.last_launch().startswith("kernel=tensor<"), xc.last_launch()
    dl, dr = torch.from_numpy(left).cuda().double(), torch.from_numpy(right).cuda().double()
    want = torch.empty(got.shape, dtype=torch.float64, device="cuda")
    xc.run_device_f64(mode, dl.data_ptr(), dr.data_ptr(), want.data_ptr(), rows, cols, nl, nr, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = want.cpu().numpy()

    def units(g, w, n):
        return np.linalg.norm((g - w).ravel()) / np.linalg.norm(w.ravel()) * 2.0 ** 24 <= 1.0 + 0.2 * n ** 0.5

    assert units(got, want, rows * cols)
    assert units(got[:, -1], want[:, -1], cols)                    # shift rows - 1: one row of products


@pytest.mark.gpu
def test_side_stream_capture_and_missing_workspace(xc, oracle):
    torch = pytest.importorskip("torch")
    shape = ("one_to_one", 225, 132, 1, 1)
    left, right = seeded_inputs(225, 132, 1, 1, 3)
    want = reference(oracle, shape, left, right)
    # without the workspace its partial images live in, the call keeps to a plan that needs none
    got = run(xc, torch, shape, left, right, workspace=False)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    # odd addresses: operands and result 4 bytes into a buffer
    shape = ("n_to_m", 27, 43, 9, 35)
    left, right = seeded_inputs(27, 43, 9, 35, 4)
    want = reference(oracle, shape, left, right)
    n = int(np.prod(xc.out_shape(*shape)))
    dl = torch.from_numpy(np.concatenate([np.zeros(1, np.float32), left.ravel()])).cuda()
    dr = torch.from_numpy(np.concatenate([np.zeros(1, np.float32), right.ravel()])).cuda()
    out = torch.full((n + 1,), float("nan"), dtype=torch.float32, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())

    def call(stream):
        xc.run_device("n_to_m", dl.data_ptr() + 4, dr.data_ptr() + 4, out.data_ptr() + 4, 27, 43, 9, 35, None, 0, 0, stream)

    with torch.cuda.stream(side):
        call(side.cuda_stream)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            call(torch.cuda.current_stream().cuda_stream)
        out.fill_(float("nan"))
        graph.replay()
        side.synchronize()
    assert xc.last_launch().startswith("kernel=tensor<")
    got = out[1:].cpu().numpy().reshape(want.shape)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1, 4])
@pytest.mark.parametrize("shape", [("n_to_m", 20, 48, 33, 63), ("n_to_m", 20, 64, 35, 31), ("one_to_one", 225, 132, 1, 1)])
def test_operands_at_any_alignment(xc, oracle, shape, offset):
    """A rows are staged with 16-byte loads where the operand and its rows allow it: operands 0, 4 and 16 bytes into a
    buffer, odd numbers of matrices interleaved by two (the absent one is staged as zeros)."""
    torch = pytest.importorskip("torch")
    mode, rows, cols, nl, nr = shape
    left, right = seeded_inputs(rows, cols, nl, nr, 6)
    want = reference(oracle, shape, left, right)
    pad = np.full(offset, 1e30, np.float32)
    dl = torch.from_numpy(np.concatenate([pad, left.ravel()])).cuda()
    dr = torch.from_numpy(np.concatenate([pad, right.ravel()])).cuda()
    out = torch.full((int(np.prod(xc.out_shape(*shape))),), float("nan"), dtype=torch.float32, device="cuda")
    wsb = xc.workspace_bytes(*shape)
    ws = torch.empty(wsb + 16, dtype=torch.uint8, device="cuda")
    xc.run_device(mode, dl.data_ptr() + 4 * offset, dr.data_ptr() + 4 * offset, out.data_ptr(), rows, cols, nl, nr, None,
                  ws.data_ptr() if wsb else 0, wsb, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert xc.last_launch().startswith("kernel=tensor<"), xc.last_launch()
    assert np.abs(out.cpu().numpy().reshape(want.shape) - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("polls", [1, 4096])
def test_waits_that_run_out_are_reported(xc, oracle, polls):
    """The waits between the kernel's roles are bounded.  The test hook keeps one arrival from the barrier that says a
    row's products are done, and lowers the limit: at one poll the first wait of any role gives up, at 4096 the
    products of two rows are issued before the warps that wait for them do.  No fault, no hang: the blocks drop their work,
    the check reports them once and beside those of the tile kernel, and the next launch is right."""
    torch = pytest.importorskip("torch")
    lib = xc.lib()
    xc.check_device()
    # several matrices B, one chunk of columns; one pair in row slices, several chunks
    shapes = [("n_to_m", 27, 43, 9, 35), ("one_to_one", 225, 132, 1, 1)]
    inputs = [seeded_inputs(*s[1:], 5) for s in shapes]
    small = seeded_inputs(32, 32, 1, 6, 77)
    for tile_too in (False, True):
        lib.xcorr_debug_stage_wait(polls, 64)
        try:
            for s, (left, right) in zip(shapes, inputs):
                run(xc, torch, s, left, right)
                assert xc.last_launch().startswith("kernel=tensor<")
            if tile_too:
                run(xc, torch, ("one_to_many", 32, 32, 1, 6), *small, xc.make_hints(kernel="tile"))
            assert lib.xcorr_check_device() == 8
            text = lib.xcorr_last_error_string().decode()
            assert "gave up" in text and " 0 block(s) of tensor_kernel" not in text
            assert text.startswith("0 block(s) of tile_kernel") != tile_too
        finally:
            lib.xcorr_debug_stage_wait(0, 0)
        xc.check_device()                                      # both counts were cleared by the report
        for s, (left, right) in zip(shapes, inputs):
            got, want = run(xc, torch, s, left, right), reference(oracle, s, left, right)
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    xc.check_device()
