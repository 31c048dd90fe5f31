"""Timed cases: the transforms that programs run through the C ABI.

`listed()` names the workloads (the benchmark's own configurations and the
published shapes), `draw(rng)` gives one more case of the same ranges,
`prepare(case, seed)` makes what a program holds before the call (inputs on
the GPU, the plan with its workspace, the tensor descriptors), `run(state)`
executes once and returns the outputs, `work(case)` counts the bytes and
flops a pass cannot do without, and `exact(case, seed)` is the same result
in 64 bits.
"""
from __future__ import annotations

import math

import torch

from sip_b200 import _lib as L
from sip_b200.fft import FftHandle, check, create_acl_tensor

# The legacy default stream, which torch's default stream is; the C ABI
# rejects a null stream.
LEGACY_STREAM = 1


# ------------------------------------------------------------------ cases
def listed():
    return [
        # The smallest call: one plain forward transform of 256 rows, a few
        # microseconds, where latency and the launch count.
        {"name": "c2c_4096x256", "kind": "c2c", "dims": "4096", "batch": 256, "forward": True},
        # Rows that fill one tile, the largest published power of two.
        {"name": "c2c_8192x8192", "kind": "c2c", "dims": "8192", "batch": 8192, "forward": True},
        # Rows of a length that is no power of two (2^8 3 5), inverse: a
        # kernel compiled at run time, as for most lengths users have.
        {"name": "c2c_inv_3840x8192", "kind": "c2c", "dims": "3840", "batch": 8192, "forward": False},
        # The benchmark's real round trips, R2C then C2R, 1 GiB of samples
        # each: short even rows, odd rows (3^7), longer even rows, and rows
        # far above one tile.
        {"name": "real_1000", "kind": "real", "dims": "1000", "batch": 268435, "forward": True},
        {"name": "real_2187", "kind": "real", "dims": "2187", "batch": 122741, "forward": True},
        {"name": "real_6000", "kind": "real", "dims": "6000", "batch": 44739, "forward": True},
        {"name": "real_1048576", "kind": "real", "dims": "1048576", "batch": 256, "forward": True},
        # Images: a batch of 2-D transforms.
        {"name": "c2c_2048x2048_b8", "kind": "c2c", "dims": "2048x2048", "batch": 8, "forward": True},
        # A volume: one 3-D transform, inverse.
        {"name": "c2c_inv_256x256x256", "kind": "c2c", "dims": "256x256x256", "batch": 1, "forward": False},
        # Long complex rows, the largest listed data: two passes.
        {"name": "c2c_65536x4096", "kind": "c2c", "dims": "65536", "batch": 4096, "forward": True},
        # Radar pulse compression (FFT, matched filter, inverse FFT) of rows
        # above one tile, a typical large serving request.
        {"name": "pulse_65536x256", "kind": "pulse", "dims": "65536", "batch": 256, "forward": True},
        # A published length with a large prime factor (2^5 211), inverse.
        {"name": "c2c_inv_6752x8192", "kind": "c2c", "dims": "6752", "batch": 8192, "forward": False},
    ]


def _smooth(lo: int, hi: int, odd: bool = False) -> list[int]:
    """The 2,3,5,7-smooth lengths of [lo, hi] (odd ones only with `odd`)."""
    out = []
    for p7 in (1, 7, 49):
        n5 = p7
        while n5 <= hi:
            n3 = n5
            while n3 <= hi:
                n2 = n3
                while n2 <= hi:
                    if n2 >= lo:
                        out.append(n2)
                    n2 *= 2
                    if odd:
                        break
                n3 *= 3
            n5 *= 5
    return sorted(out)


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _length(rng, lo: int, hi: int, odd: bool = False) -> int:
    """A smooth length near a log-uniform target."""
    pool = _smooth(lo, hi, odd)
    target = _log_uniform(rng, lo, hi)
    pool.sort(key=lambda n: abs(math.log(n / target)))
    return rng.choice(pool[:4])


def _batch(rng, n: int, lo: int, hi: int, most: int | None = None) -> int:
    """A batch that makes lo..hi values in all, log-uniform."""
    b = max(1, round(_log_uniform(rng, max(lo, n), max(hi, n)) / n))
    return b if most is None else min(b, most)


def draw(rng):
    kind = rng.choice(["rows", "rows", "large", "real", "real", "real_odd", "2d", "3d", "pulse", "prime"])
    forward = rng.random() < 0.5
    if kind == "rows":  # one tile: powers of two and mixed lengths alike
        n = 2 ** rng.randint(8, 13) if rng.random() < 0.4 else _length(rng, 256, 8192)
        return {"kind": "c2c", "dims": str(n), "batch": _batch(rng, n, 2 ** 20, 2 ** 26), "forward": forward}
    if kind == "large":
        n = 2 ** rng.randint(15, 20) if rng.random() < 0.4 else _length(rng, 20000, 2 ** 20)
        return {"kind": "c2c", "dims": str(n), "batch": _batch(rng, n, 2 ** 21, 2 ** 26), "forward": forward}
    if kind == "real":
        n = _length(rng, 500, 2 ** 20)
        n *= 1 + n % 2
        hi = 2 ** 27 if n <= 16384 else 2 ** 26
        return {"kind": "real", "dims": str(n), "batch": _batch(rng, n, 2 ** 21, hi), "forward": True}
    if kind == "real_odd":
        n = _length(rng, 500, 16000, odd=True)
        return {"kind": "real", "dims": str(n), "batch": _batch(rng, n, 2 ** 21, 2 ** 27), "forward": True}
    if kind == "2d":
        x, y = (2 ** rng.randint(8, 11) if rng.random() < 0.4 else _length(rng, 256, 2048) for _ in range(2))
        return {"kind": "c2c", "dims": f"{x}x{y}", "batch": _batch(rng, x * y, 2 ** 20, 2 ** 25),
                "forward": forward}
    if kind == "3d":
        x, y, z = (2 ** rng.randint(6, 8) if rng.random() < 0.4 else _length(rng, 64, 256) for _ in range(3))
        return {"kind": "c2c", "dims": f"{x}x{y}x{z}", "batch": _batch(rng, x * y * z, 2 ** 20, 2 ** 24),
                "forward": forward}
    if kind == "pulse":
        n = _length(rng, 2048, 2 ** 18)
        return {"kind": "pulse", "dims": str(n), "batch": _batch(rng, n, 2 ** 20, 2 ** 24, 512), "forward": True}
    # a prime factor above 31
    p = rng.choice([37, 41, 53, 67, 97, 131, 167, 211, 251])
    n = p * max(2, round(_log_uniform(rng, 1000, 6752) / p))
    return {"kind": "c2c", "dims": str(n), "batch": _batch(rng, n, 2 ** 20, 2 ** 25), "forward": forward}


def _dims(case) -> list[int]:
    return [int(d) for d in case["dims"].split("x")]


# ----------------------------------------------------------------- inputs
def _input(case, seed: int) -> torch.Tensor:
    """C2C: i.i.d. N(0, 1); real: U[-1, 1]; pulse: delayed chirp + noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    dims, batch = _dims(case), case["batch"]
    if case["kind"] == "real":
        return torch.rand((batch, dims[0]), generator=g, device="cuda").mul_(2).sub_(1)
    x = torch.randn((batch, *dims), generator=g, device="cuda", dtype=torch.complex64)
    x.mul_(math.sqrt(2.0))
    if case["kind"] == "pulse":
        x.mul_(0.1)
        pulse = _chirp(dims[0]).to(torch.complex64)
        x[:, dims[0] // 3: dims[0] // 3 + pulse.numel()] += pulse
    return x


def _chirp(n: int) -> torch.Tensor:
    """The transmitted pulse: a linear chirp of n / 4 samples."""
    t = torch.arange(n // 4, device="cuda", dtype=torch.float64)
    return torch.polar(torch.ones_like(t), math.pi * t * t / max(1, n // 4))


def _filter(n: int) -> torch.Tensor:
    """The pulse's spectrum, as a program stores it."""
    return torch.fft.fft(_chirp(n), n=n).to(torch.complex64)


class _Plan:
    """One planned handle with its workspace, on torch's default stream."""

    def __init__(self, make):
        self.h = make()
        # A length whose kernels are compiled at run time is planned again
        # once they are there, as a program that starts up does.
        check(L.lib().sipFftJitWait(600000), "sipFftJitWait")
        self.h.destroy()
        self.h = make()
        self.h.bind_workspace()
        check(self.h.set_stream(LEGACY_STREAM), "asdFftSetStream")


def _planned(dims, fft_type, forward, batch) -> _Plan:
    direction = L.ASCEND_FFT_FORWARD if forward else L.ASCEND_FFT_INVERSE

    def make():
        h = FftHandle()
        if len(dims) == 1:
            rc = h.make_plan_1d(dims[0], fft_type, direction, batch)
        elif len(dims) == 2:
            rc = h.make_plan_2d(dims[0], dims[1], fft_type, direction, batch)
        else:
            rc = h.make_plan_3d(dims[0], dims[1], dims[2], fft_type, direction, batch)
        check(rc, "asdFftMakePlan")
        return h

    return _Plan(make)


class _State:
    """The execs of one pass in order, (function, plan, input, output), and
    the tensors a pass returns."""

    def __init__(self):
        self.execs = []
        self.outputs = []
        self.keep = []

    def tensor(self, t):
        d = create_acl_tensor(t)
        self.keep.append((t, d))
        return d

    def __del__(self):
        for _, d in self.keep:
            L.lib().aclDestroyTensor(d)


def prepare(case, seed):
    s = _State()
    lib = L.lib()
    dims, batch = _dims(case), case["batch"]
    x = _input(case, seed)
    if case["kind"] == "real":
        n = dims[0]
        spec = torch.empty((batch, n // 2 + 1), dtype=torch.complex64, device="cuda")
        back = torch.empty_like(x)
        r2c = _planned(dims, L.ASCEND_FFT_R2C, True, batch)
        c2r = _planned(dims, L.ASCEND_FFT_C2R, False, batch)
        dx, dspec, dback = s.tensor(x), s.tensor(spec), s.tensor(back)
        s.execs = [(lib.asdFftExecR2C, r2c, dx, dspec), (lib.asdFftExecC2R, c2r, dspec, dback)]
        s.outputs = [spec, back]
        return s
    y = torch.empty_like(x)
    if case["kind"] == "pulse":
        filt = _filter(dims[0])
        s.keep.append((filt, None))

        def make():
            h = FftHandle()
            check(h.make_plan_pulse_1d(dims[0], batch, filt.data_ptr(),
                                       L.SIP_FFT_PULSE_CONJ_FILTER | L.SIP_FFT_PULSE_SCALE), "sipFftMakePlanPulse1D")
            return h

        plan = _Plan(make)
    else:
        plan = _planned(dims, L.ASCEND_FFT_C2C, case["forward"], batch)
    s.execs = [(lib.asdFftExecC2C, plan, s.tensor(x), s.tensor(y))]
    s.outputs = [y]
    return s


def run(state):
    for fn, plan, a, b in state.execs:
        check(fn(plan.h.h, a, b), "exec")
    return state.outputs


# ------------------------------------------------------------ what it costs
def work(case):
    dims, batch = _dims(case), case["batch"]
    n = math.prod(dims)
    if case["kind"] == "real":  # two calls: each reads its input and writes its output once
        return {"bytes": 2.0 * batch * (4 * n + 8 * (n // 2 + 1)), "flops": 2 * 2.5 * n * math.log2(n) * batch}
    flops = 5.0 * n * math.log2(n) * batch
    if case["kind"] == "pulse":  # two transforms and the filter product; the filter is read once
        return {"bytes": 16.0 * n * batch + 8.0 * n, "flops": 2 * flops + 6.0 * n * batch}
    return {"bytes": 16.0 * n * batch, "flops": flops}


def exact(case, seed):
    dims = _dims(case)
    x = _input(case, seed)
    if case["kind"] == "real":
        spec = torch.fft.rfft(x.double(), dim=-1)
        return [spec, torch.fft.irfft(spec, n=dims[0], dim=-1, norm="forward")]
    x = x.to(torch.complex128)
    if case["kind"] == "pulse":
        spec = torch.fft.fft(x, dim=-1)
        spec.mul_(_filter(dims[0]).to(torch.complex128).conj())
        return [torch.fft.ifft(spec, dim=-1)]
    axes = tuple(range(1, x.dim()))
    if case["forward"]:
        return [torch.fft.fftn(x, dim=axes)]
    return [torch.fft.ifftn(x, dim=axes, norm="forward")]
