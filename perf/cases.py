"""Workloads that stand for what programs do with turbofft_b200, for timing two builds against each other.

A case names an entry point, a data type and a shape.  The kinds:

  fft / ifft   the torch-style call on a CUDA tensor (plan taken from the library's cache, output allocated per call)
  plan         a plan and an output buffer the program keeps, executed again and again (the sweep benchmark's form)
  detect       the same with checksums on (thread_bs = the tuned value), the counters read after every call
  correct      the same with one faulty block in a thousand, repaired inside the kernels
  fft2         2-D transform of a stack of images (strided-batch plan along the rows' axis, then the rows)
  host         pinned host buffers in and out through Plan.exec_host
"""
import math

import torch

import turbofft_b200 as tf

_DTYPES = {"c64": (tf.FLOAT2, torch.complex64, 8), "c128": (tf.DOUBLE2, torch.complex128, 16)}


def _case(kind, dtype, logn, batch, name=None, rows=0):
    c = {"kind": kind, "dtype": dtype, "logn": logn, "batch": batch}
    if rows:
        c["log_rows"] = rows
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one frame of a few channels at a time: the latency configuration of the benchmark
        _case("fft", "c64", 10, 16, "c64_2^10_x16"),
        # a handful of medium signals in double precision, back to time or frequency: two launches that fill no GPU
        _case("ifft", "c128", 16, 3, "c128_2^16_x3_ifft"),
        # very many short signals, a count that fits no tile (radar pulses, OFDM symbols)
        _case("plan", "c64", 5, 1000003, "c64_2^5_x1000003"),
        # three points of the sweep logN + log batch = 28 in single precision: one, two and three launches
        _case("plan", "c64", 13, 1 << 15, "c64_2^13_x2^15"),
        _case("plan", "c64", 16, 1 << 12, "c64_2^16_x2^12"),
        # an odd number of long records, transformed back and scaled
        _case("ifft", "c64", 24, 5, "c64_2^24_x5_ifft"),
        # double precision spectra of an odd number of ordinary frames
        _case("fft", "c128", 12, 5001, "c128_2^12_x5001"),
        # the double precision sweep's middle
        _case("plan", "c128", 18, 1 << 9, "c128_2^18_x2^9"),
        # checksums on, nothing goes wrong, the program looks at the counters after every call
        _case("detect", "c64", 12, 1 << 14, "c64_2^12_x2^14_detect"),
        # the fault-tolerance configuration: logN 20, 256 signals, a fault in one block of a thousand, corrected online
        _case("correct", "c64", 20, 1 << 8, "c64_2^20_x2^8_correct"),
        # a stack of images
        _case("fft2", "c64", 10, 48, "c64_2^10x2^10_x48_fft2", rows=10),
        # data that lives on the host: 128 MiB in, 128 MiB out
        _case("host", "c64", 12, 1 << 12, "c64_2^12_x2^12_host"),
    ]


def _spread(rng, low, high):
    """log-uniform whole number, odd ones as likely as not."""
    v = int(round(2.0 ** rng.uniform(low, high)))
    return max(1, v | 1 if rng.random() < 0.5 else v)


def draw(rng):
    kind = rng.choice(["fft", "fft", "ifft", "ifft", "plan", "plan", "plan", "plan", "detect", "correct", "fft2", "host"])
    dtype = "c64" if kind == "host" else rng.choice(["c64", "c64", "c64", "c128"])
    wide = 1 if dtype == "c128" else 0
    if kind == "fft2":
        rows, logn = rng.randint(6, 10), rng.randint(6, 12)
        total = rng.uniform(max(14, rows + logn), 26 - wide)
        return _case(kind, dtype, logn, _spread(rng, 0, total - rows - logn), rows=rows)
    low, high, least, most = {
        "fft": (3, 22, 10, 25), "ifft": (3, 22, 10, 25), "plan": (5, 24, 14, 27), "detect": (7, 22, 16, 26), "correct": (7, 22, 18, 26),
        "host": (8, 18, 16, 25)}[kind]
    logn = rng.randint(low, high)
    total = rng.uniform(max(least, logn), max(most - wide, logn))
    return _case(kind, dtype, logn, _spread(rng, 0, total - logn))


def _uniform(shape, dtype, gen, device):
    """Both components uniform in [-1, 1), the sweep's distribution."""
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    x = torch.rand(*shape, 2, dtype=real, generator=gen, device=device)
    return torch.view_as_complex(x.mul_(2).sub_(1))


def prepare(case, seed):
    code, dtype, _ = _DTYPES[case["dtype"]]
    kind, logn, batch = case["kind"], case["logn"], case["batch"]
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device).manual_seed(seed)
    shape = (batch, 1 << logn) if kind != "fft2" else (batch, 1 << case["log_rows"], 1 << logn)
    x = _uniform(shape, dtype, gen, device)
    state = {"kind": kind, "x": x}
    if kind in ("plan", "detect", "correct", "host"):
        plan = tf.Plan(logn, batch, code, if_ft=int(kind in ("detect", "correct")), if_err=int(kind == "correct"), thread_bs=0, device=device.index)
        if kind in ("detect", "correct"):
            # a fault far above the spectrum's own values, a threshold far above rounding
            plan.set_ft_params(err_inj=50.0 * math.sqrt(1 << logn), err_smoothing=1000.0, err_threshold=1e-5)
        if kind == "correct":
            plan.set_injection(True, period=1000)
        state["plan"] = plan
        if kind == "host":
            state["x"] = torch.empty(shape, dtype=dtype, pin_memory=True).copy_(x)
            state["out"] = torch.empty(shape, dtype=dtype, pin_memory=True)
        else:
            state["out"] = torch.empty_like(x)
    return state


def run(state):
    kind = state["kind"]
    if kind == "fft":
        return tf.fft(state["x"])
    if kind == "ifft":
        return tf.ifft(state["x"])
    if kind == "fft2":
        return tf.fft2(state["x"])
    if kind == "host":
        return state["plan"].exec_host(state["x"], state["out"])
    y = state["plan"](state["x"], state["out"])
    if kind == "detect":
        detected, corrected, _ = state["plan"].ft_status()
        return {"y": y, "detected": detected, "corrected": corrected}
    return y


def work(case):
    """One read of the input, one write of the output, 5 N log2 N operations per signal of N points."""
    logn = case["logn"] + case.get("log_rows", 0)
    n = case["batch"] << logn
    return {"bytes": 2 * n * _DTYPES[case["dtype"]][2], "flops": 5 * n * logn}


def tolerance(case):
    """Two correctly rounded radix orders differ by a few units of the last place per stage."""
    return {"rel": 2e-6} if case["dtype"] == "c64" else {"rel": 5e-15}
