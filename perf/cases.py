"""The work users have this library do, as timed cases: full 2-D cross-correlation through the
public entry points -- device pointers in single precision (the four input modes), the FFT path,
double precision, and host buffers -- from one 16x16 pair to hundreds of gigaflops.

Values are uniform [0, 1), the distribution of the input generator whose matrices the `cross`
program reads.  Sizes are those of this repository's benchmark, plus odd ones: real templates
and images are rarely multiples of 16.
"""
import importlib.util
import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The binding, loaded by path (its directory name has a hyphen)."""
    name = "jpdc23_artifact_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(ROOT, "jpdc23-artifact_b200", "__init__.py"))
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def _case(name, path, mode, rows, cols, n_left, n_right):
    return {"name": name, "path": path, "mode": mode, "rows": rows, "cols": cols, "n_left": n_left, "n_right": n_right}


def listed():
    return [
        # one small patch against another (tracking a feature from frame to frame): latency of a call
        _case("pair_16", "f32", "one_to_one", 16, 16, 1, 1),
        # one pair of odd size: a cut-out of an image against its reference
        _case("pair_100x75", "f32", "one_to_one", 100, 75, 1, 1),
        # one large pair: the registration of two images, no parallelism over matrices
        _case("pair_256", "f32", "one_to_one", 256, 256, 1, 1),
        # one reference against many deformed images
        _case("many_64", "f32", "one_to_many", 64, 64, 1, 512),
        # every patch against every template
        _case("all_pairs_32", "f32", "n_to_m", 32, 32, 32, 64),
        # every patch of an image against its own group of candidates
        _case("groups_48", "f32", "n_to_mn", 48, 48, 16, 2048),
        # the same with sizes and counts that fit no tile
        _case("all_pairs_27x43", "f32", "n_to_m", 27, 43, 9, 35),
        # large images against one reference: the longest call
        _case("many_256", "f32", "one_to_many", 256, 256, 1, 32),
        # the FFT engine on the benchmark's batch and on an odd size
        _case("fft_many_64", "fft", "one_to_many", 64, 64, 1, 512),
        _case("fft_groups_90x75", "fft", "n_to_mn", 90, 75, 4, 48),
        # double precision
        _case("double_groups_48", "f64", "n_to_mn", 48, 48, 4, 256),
        # the whole computation of the `cross` program: page-locked host buffers in, host result out
        _case("host_all_pairs_32", "host", "n_to_m", 32, 32, 32, 64),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# a drawn case stays below the listed ones in arithmetic (double at half the rate of single) and in bytes
_MAX_FLOPS = {"f32": 2.7e11, "fft": 2.7e11, "f64": 5e10, "host": 1e11}
_MAX_BYTES = 9e7


def draw(rng):
    path = rng.choices(["f32", "fft", "f64", "host"], [7, 2, 2, 1])[0]
    mode = rng.choices(["one_to_one", "one_to_many", "n_to_mn", "n_to_m"], [2, 3, 3, 3])[0]
    while True:
        rows, cols = _log_uniform(rng, 8, 256), _log_uniform(rng, 8, 256)
        n_left = 1 if mode.startswith("one") else _log_uniform(rng, 2, 64)
        n_right = 1 if mode == "one_to_one" else _log_uniform(rng, 2, 2048)
        if mode == "n_to_mn":
            n_right = n_left * max(1, n_right // n_left)
        case = {"path": path, "mode": mode, "rows": rows, "cols": cols, "n_left": n_left, "n_right": n_right}
        if _direct_flops(case) <= _MAX_FLOPS[path] and work(case)["bytes"] <= _MAX_BYTES:
            return case


def _pairs(case):
    return case["n_left"] * case["n_right"] if case["mode"] == "n_to_m" else case["n_right"]


def _direct_flops(case):
    return 2.0 * _pairs(case) * (case["rows"] * case["cols"]) ** 2


def prepare(case, seed):
    xc = _package()
    xc.lib()
    rows, cols, nl, nr, mode, path = (case[k] for k in ("rows", "cols", "n_left", "n_right", "mode", "path"))
    dtype = torch.float64 if path == "f64" else torch.float32
    device = "cpu" if path == "host" else "cuda"
    gen = torch.Generator(device=device).manual_seed(seed)
    state = dict(case)
    state["xc"] = xc
    shape = xc.out_shape(mode, rows, cols, nl, nr)
    if path == "host":
        for key, sh in (("left", (nl, rows, cols)), ("right", (nr, rows, cols)), ("out", shape)):
            state["pinned_" + key] = torch.empty(sh, dtype=dtype, pin_memory=True)
            state[key] = state["pinned_" + key].numpy()
        state["pinned_left"].uniform_(generator=gen)
        state["pinned_right"].uniform_(generator=gen)
        return state
    state["left"] = torch.rand((nl, rows, cols), generator=gen, dtype=dtype, device=device)
    state["right"] = torch.rand((nr, rows, cols), generator=gen, dtype=dtype, device=device)
    state["out"] = torch.empty(shape, dtype=dtype, device=device)
    state["hints"] = xc.make_hints(kernel="fft") if path == "fft" else None
    state["ws_bytes"] = 0 if path == "f64" else xc.workspace_bytes(mode, rows, cols, nl, nr, state["hints"])
    state["ws"] = torch.empty(max(state["ws_bytes"], 256), dtype=torch.uint8, device=device)
    return state


def run(state):
    xc, out = state["xc"], state["out"]
    if state["path"] == "host":
        return xc.run_host(state["mode"], state["left"], state["right"], out=out)
    stream = torch.cuda.current_stream().cuda_stream
    args = (state["mode"], state["left"].data_ptr(), state["right"].data_ptr(), out.data_ptr(),
            state["rows"], state["cols"], state["n_left"], state["n_right"])
    if state["path"] == "f64":
        xc.run_device_f64(*args, stream)
    else:
        xc.run_device(*args, state["hints"], state["ws"].data_ptr() if state["ws_bytes"] else 0, state["ws_bytes"], stream)
    return out


def work(case):
    """Direct paths: rows^2 cols^2 multiply-adds a pair.  FFT path: real transforms (2.5 n log2 n) of
    2*rows x 2*cols points of every input and every result, and the products of the half spectra."""
    h, w, pairs = case["rows"], case["cols"], _pairs(case)
    inputs = case["n_left"] + case["n_right"]
    size = 8 if case["path"] == "f64" else 4
    moved = size * (inputs * h * w + pairs * (2 * h - 1) * (2 * w - 1))
    if case["path"] != "fft":
        return {"bytes": moved, "flops": _direct_flops(case)}
    points = 4 * h * w
    return {"bytes": moved, "flops": 2.5 * points * math.log2(points) * (inputs + pairs) + 6.0 * pairs * 2 * h * (w + 1)}


def tolerance(case):
    """Against the same sums in double: a sum of rows * cols products taken in sequence is off by
    0.185 * sqrt(rows * cols) units of rounding (2-norm; largest single difference 1.06), measured from
    16x16 to 64x64 and 10x235, and less where the rows are summed in parts; the FFT path by 1.7e-7 and
    8.1e-7 at every size; the double path by the same multiple of its own unit.  Four times that, and
    no less than a 16x16 pair would be allowed."""
    if case["path"] == "fft":
        return {"rel": 7e-7, "max": 3.3e-6}
    unit = 2.0 ** -53 if case["path"] == "f64" else 2.0 ** -24
    unit *= math.sqrt(max(256, case["rows"] * case["cols"]))
    return {"rel": 0.75 * unit, "max": 4.3 * unit}
