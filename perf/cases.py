"""Workloads the library's speed is judged by: the public entry points over the sizes users bring.

``listed()`` names the workloads, ``draw(rng)`` gives another one of the same ranges,
``prepare`` builds what a program holds before the call (device arrays, plan, convolver, filter
states), ``run`` is one pass through the public API.  Signals are synthetic: uniform or Gaussian
noise, impulse responses Gaussian noise under an exponential decay (-60 dB after 1.5 s at 48 kHz).

Kinds
  frame       one frame on the host: ``FFT.forward``, ``FFT.magnitude`` and ``FFT.inverse`` on arrays
              (an analyser or a plug-in that looks at one block at a time: launches and copies)
  clip        ``FFT.stft`` and ``FFT.istft`` of one recording in host memory, the reference's full
              split spectra crossing to the host and back
  stft        batched STFT (half spectrum, optionally magnitude) and iSTFT on device tensors
  fft         batches of plain real transforms, forward and inverse, on device arrays
  stream      one block of the partitioned convolution for every channel, delay line full
  whole       partitioned convolution of whole recordings, device arrays
  oneshot     the ``.fft`` convolution mode, device arrays
  eq          biquad cascades over recordings, device arrays
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from metalaudio_b200 import AudioDevice, BiquadFilter, FFT, Tensor, WindowType
from metalaudio_b200 import _lib as L

SAMPLE_RATE = 48000.0


def listed():
    return [
        # one 2048-point frame of an analyser, host arrays: the smallest call
        {"name": "frame_2048", "kind": "frame", "n": 2048},
        # ten seconds at 44.1 kHz through the reference's stft / istft arrays
        {"name": "clip_10s", "kind": "clip", "n": 2048, "hop": 512, "length": 441000},
        # the eight channels of four separated stereo stems, one 7.8 s segment
        {"name": "stft_stems", "kind": "stft", "n": 4096, "hop": 1024, "signals": 8, "length": 343980, "magnitude": True},
        # a speech corpus batch: 32 ms windows every 10 ms at 16 kHz, hop not a divisor of the window
        {"name": "stft_speech", "kind": "stft", "n": 512, "hop": 160, "signals": 512, "length": 163123, "magnitude": False},
        # the batched analysis-synthesis configuration: complex and magnitude out, signals back
        {"name": "stft_batch", "kind": "stft", "n": 4096, "hop": 1024, "signals": 256, "length": 1 << 20, "magnitude": True},
        # the large-transform configuration, forward and inverse
        {"name": "fft_65536", "kind": "fft", "n": 65536, "batch": 4096},
        # a stereo reverb insert, 3 s response per ear, 128-sample blocks: latency of one block
        {"name": "stream_stereo", "kind": "stream", "channels": 2, "block": 128, "taps": 143777, "irs": 2},
        # the shared-response streaming configuration, one block of all 512 channels
        {"name": "stream_shared", "kind": "stream", "channels": 512, "block": 256, "taps": 131072, "irs": 1},
        # low latency with one response per channel pair (a quarter of the configuration's channels and taps)
        {"name": "stream_pairs", "kind": "stream", "channels": 256, "block": 64, "taps": 65536, "irs": 128},
        # the same 512 channels convolved as whole recordings
        {"name": "whole_shared", "kind": "whole", "channels": 512, "block": 256, "taps": 131072, "irs": 1, "length": 1 << 20},
        # one-shot convolution of a set of 10 s recordings with a 1.5 s response
        {"name": "oneshot_10s", "kind": "oneshot", "signals": 64, "length": 441000, "taps": 66150},
        # four-band equaliser over the tracks of a mixing session, 10 s
        {"name": "eq_tracks", "kind": "eq", "channels": 24, "sections": 4, "length": 480000},
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["frame", "clip", "stft", "stft", "fft", "stream", "stream", "whole", "oneshot", "eq"])
    if kind == "frame":
        return {"kind": kind, "n": 1 << rng.randint(8, 13)}
    if kind == "clip":
        n = 1 << rng.randint(9, 12)
        return {"kind": kind, "n": n, "hop": rng.choice([n // 4, n // 2, n // 4 + 3]), "length": _spread(rng, 20000, 441000)}
    if kind == "stft":
        n = 1 << rng.randint(8, 13)
        length = _spread(rng, 4 * n, 1 << 20)
        return {"kind": kind, "n": n, "hop": rng.choice([n // 4, n // 4, n // 2, 5 * n // 16]), "length": length,
                "signals": _spread(rng, 1, min(2048, (1 << 27) // length)), "magnitude": rng.random() < 0.5}
    if kind == "fft":
        n = 1 << rng.randint(8, 20)
        return {"kind": kind, "n": n, "batch": _spread(rng, 1, (1 << 27) // n)}
    if kind == "stream":
        block = 1 << rng.randint(6, 9)
        taps = _spread(rng, 4 * block, 131072)
        channels = _spread(rng, 1, min(512, (1 << 26) // taps))
        return {"kind": kind, "channels": channels, "block": block, "taps": taps, "irs": rng.choice([1, (channels + 1) // 2])}
    if kind == "whole":
        taps = _spread(rng, 1000, 131072)
        length = _spread(rng, 20000, 1 << 20)
        channels = _spread(rng, 1, min(256, (1 << 28) // length))
        irs = rng.choice([1, min(channels, 32)])
        return {"kind": kind, "channels": channels, "block": 1 << rng.randint(6, 9), "taps": taps, "irs": irs, "length": length}
    if kind == "oneshot":
        taps = _spread(rng, 500, 131072)
        length = _spread(rng, 2000, 900000)
        return {"kind": kind, "signals": _spread(rng, 1, min(512, (1 << 26) // (length + taps))), "length": length, "taps": taps}
    length = _spread(rng, 4096, 1 << 20)
    return {"kind": kind, "channels": _spread(rng, 1, min(512, (1 << 26) // length)), "sections": rng.randint(1, 8), "length": length}


# --------------------------------------------------------------------------- device state

@functools.lru_cache(maxsize=None)
def _device() -> AudioDevice:
    return AudioDevice(0)


class _Handle:
    """An object of the C API, destroyed with its owner and before the device it lives on."""

    def __init__(self, create, destroy, *args):
        self.lib = L.load()
        self.device = _device()
        self._destroy = getattr(self.lib, destroy)
        self.h = ctypes.c_void_p()
        _ok(getattr(self.lib, create)(*args, ctypes.byref(self.h)))

    def __del__(self):
        if getattr(self, "h", None):
            self._destroy(self.h)


class _DeviceArray:
    """Lets torch look at a Tensor's memory, which lives as long as torch's view of it."""

    def __init__(self, tensor: Tensor):
        self.owner = tensor
        self.__cuda_array_interface__ = {"shape": tensor.shape, "typestr": "<f4", "data": (tensor.pointer, False),
                                         "version": 3, "strides": None}


def _ok(status):
    if status != L.MA_OK:
        raise RuntimeError(L.load().ma_status_string(status).decode())


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _uniform(shape, gen):
    return torch.rand(shape, device="cuda", generator=gen) * 2.0 - 1.0


def _gauss(shape, gen, sigma):
    return torch.randn(shape, device="cuda", generator=gen) * sigma


def _responses(n_irs, taps, gen):
    """Decaying noise of unit energy, as the host array a program loads its responses into."""
    decay = torch.exp(torch.arange(taps, device="cuda", dtype=torch.float64) * (-math.log(1000.0) / (1.5 * SAMPLE_RATE)))
    h = torch.randn((n_irs, taps), device="cuda", generator=gen) * decay.float()
    return (h / h.double().square().sum(1, keepdim=True).sqrt().float()).cpu().numpy()


def _ramp(channels, irs):
    """channel -> response: neighbouring channels share, as evenly as it goes."""
    return (np.arange(channels, dtype=np.int64) * irs // channels).astype(np.int32)


def _hann(n):
    k = np.arange(n, dtype=np.float64)
    return (0.5 * (1.0 - np.cos(2.0 * np.pi * k / n))).astype(np.float32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dev = _device()
    kind = case["kind"]
    s = {"case": case}
    if kind == "frame":
        n = case["n"]
        s["x"] = np.random.default_rng(seed).standard_normal(n).astype(np.float32)
        s["fwd"] = FFT(dev, FFT.Config(size=n, windowType=WindowType.none))
        s["inv"] = FFT(dev, FFT.Config(size=n, inverse=True, windowType=WindowType.none))
        for name, count in (("re", n), ("im", n), ("mag", n // 2 + 1), ("back", n)):
            s[name] = np.zeros(count, np.float32)
    elif kind == "clip":
        s["x"] = np.random.default_rng(seed).uniform(-1.0, 1.0, case["length"]).astype(np.float32)
        s["fft"] = FFT(dev, FFT.Config(size=case["n"], hopSize=case["hop"]))
    elif kind == "stft":
        n, signals = case["n"], case["signals"]
        s["fft"] = FFT(dev, FFT.Config(size=n, hopSize=case["hop"]), window=_hann(n))
        frames = s["fft"].frameCount(case["length"])
        shapes = {"x": (signals, case["length"]), "spec": (signals, frames, n // 2 + 1, 2),
                  "out": (signals, (frames - 1) * case["hop"] + n)}
        if case["magnitude"]:
            shapes["mag"] = (signals, frames, n // 2 + 1)
        for name, shape in shapes.items():
            s[name] = Tensor(dev, shape)
            s["t_" + name] = torch.as_tensor(_DeviceArray(s[name]), device="cuda")
        s["t_x"].uniform_(-1.0, 1.0, generator=gen)
    elif kind == "fft":
        n, batch = case["n"], case["batch"]
        s["plan"] = _Handle("ma_fft_plan_create", "ma_fft_plan_destroy", dev.handle, n, None, n)
        s["x"] = _gauss((batch, n), gen, 1.0)
        s["spec"] = torch.empty((batch, n // 2 + 1, 2), device="cuda")
        s["back"] = torch.empty((batch, n), device="cuda")
    elif kind in ("stream", "whole"):
        channels, block, taps = case["channels"], case["block"], case["taps"]
        pc = s["pc"] = _Handle("ma_pconv_create", "ma_pconv_destroy", dev.handle, block, channels)
        irs = _responses(case["irs"], taps, gen)
        cmap = _ramp(channels, case["irs"])
        _ok(pc.lib.ma_pconv_set_kernels(pc.h, irs.ctypes.data_as(ctypes.c_void_p), taps, case["irs"],
                                        cmap.ctypes.data_as(ctypes.c_void_p)))
        if kind == "whole":
            _ok(pc.lib.ma_pconv_reserve(pc.h, case["length"]))
            s["x"] = _gauss((channels, case["length"]), gen, 0.1)
            s["out"] = torch.empty((channels, case["length"] + taps - 1), device="cuda")
        else:
            # a stream that has been running: every partition of the delay line holds a block
            past = -(-taps // block)
            s["x"] = _gauss((channels, block), gen, 0.1)
            s["out"] = torch.empty((channels, block), device="cuda")
            history = _gauss((channels, past * block), gen, 0.1)
            torch.cuda.synchronize()
            for b in range(past):
                _ok(pc.lib.ma_pconv_step_dev(pc.h, ctypes.c_void_p(history.data_ptr() + 4 * b * block), past * block,
                                             _p(s["out"]), block))
            dev.synchronize(30.0)
    elif kind == "oneshot":
        signals, length, taps = case["signals"], case["length"], case["taps"]
        h = _responses(1, taps, gen)[0]
        fc = s["fc"] = _Handle("ma_fftconv_create", "ma_fftconv_destroy", dev.handle,
                               h.ctypes.data_as(ctypes.c_void_p), taps, length, signals)
        size = ctypes.c_int64(0)
        _ok(fc.lib.ma_fftconv_fft_size(fc.h, ctypes.byref(size)))
        s["x"] = _gauss((signals, length), gen, 0.1)
        s["out"] = torch.empty((signals, size.value), device="cuda")
    else:
        channels, sections = case["channels"], case["sections"]
        bq = s["bq"] = _Handle("ma_biquad_create", "ma_biquad_destroy", dev.handle, channels, sections)
        coeffs = np.stack([BiquadFilter.design(BiquadFilter.FilterType.peaking(3.0 if k % 2 else -4.0), 80.0 * 2.0 ** k,
                                               SAMPLE_RATE, 1.0).asArray() for k in range(sections)])
        _ok(bq.lib.ma_biquad_set_coefficients(bq.h, coeffs.ctypes.data_as(ctypes.c_void_p), 1, None))
        s["x"] = _gauss((channels, case["length"]), gen, 0.1)
        s["out"] = torch.empty_like(s["x"])
    torch.cuda.synchronize()   # the library runs on its own stream
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        s["fwd"].forward(s["x"], s["re"], s["im"])
        s["fwd"].magnitude(s["re"], s["im"], s["mag"])
        s["inv"].inverse(s["re"], s["im"], s["back"])
        return [s["re"], s["im"], s["mag"], s["back"]]
    if kind == "clip":
        spectra = s["fft"].stft(s["x"])
        return [spectra.real, spectra.imag, s["fft"].istft(spectra)]
    if kind == "stft":
        s["fft"].stftTensor(s["x"], s["spec"], s.get("mag"))
        s["fft"].istftTensor(s["spec"], s["out"])
        return [s["t_spec"], s["t_out"]] + ([s["t_mag"]] if case["magnitude"] else [])
    if kind == "fft":
        plan, batch = s["plan"], case["batch"]
        _ok(plan.lib.ma_fft_forward_dev(plan.h, _p(s["x"]), _p(s["spec"]), None, None, 0, 1.0, batch, L.LAYOUT_HALF_INTERLEAVED))
        _ok(plan.lib.ma_fft_inverse_dev(plan.h, _p(s["spec"]), None, _p(s["back"]), batch, L.LAYOUT_HALF_INTERLEAVED))
        return [s["spec"], s["back"]]
    if kind == "stream":
        pc = s["pc"]
        _ok(pc.lib.ma_pconv_step_dev(pc.h, _p(s["x"]), case["block"], _p(s["out"]), case["block"]))
        return s["out"]
    if kind == "whole":
        pc = s["pc"]
        _ok(pc.lib.ma_pconv_process_dev(pc.h, _p(s["x"]), case["length"], case["length"], _p(s["out"]), s["out"].shape[1]))
        return s["out"]
    if kind == "oneshot":
        fc = s["fc"]
        _ok(fc.lib.ma_fftconv_process_dev(fc.h, _p(s["x"]), case["length"], case["length"], case["signals"], _p(s["out"])))
        return s["out"]
    bq = s["bq"]
    _ok(bq.lib.ma_biquad_process_dev(bq.h, _p(s["x"]), case["length"], _p(s["out"]), case["length"], case["length"]))
    return s["out"]


def work(case):
    """Bytes and operations of one pass that no implementation avoids: inputs read once, outputs
    written once (the delay line is an input of a streaming step), real transforms at 2.5 N log2 N."""
    kind = case["kind"]
    if kind == "frame":
        n = case["n"]
        return {"bytes": 4.0 * (n + 2 * n + (n // 2 + 1) + n), "flops": 2 * 2.5 * n * math.log2(n)}
    if kind in ("clip", "stft"):
        n, hop = case["n"], case["hop"]
        signals = case.get("signals", 1)
        frames = signals * ((case["length"] - n) // hop + 1)
        per_frame = 8.0 * n if kind == "clip" else 8.0 * (n // 2 + 1)
        moved = 2 * frames * per_frame + 4.0 * signals * case["length"] + 4.0 * frames * hop   # spectra out and in, signals in and out
        if case.get("magnitude"):
            moved += 4.0 * frames * (n // 2 + 1)
        return {"bytes": moved, "flops": 2 * frames * 2.5 * n * math.log2(n)}
    if kind == "fft":
        n, batch = case["n"], case["batch"]
        return {"bytes": 2.0 * batch * (4 * n + 8 * (n // 2 + 1)), "flops": 2 * batch * 2.5 * n * math.log2(n)}
    if kind == "stream":
        c, b = case["channels"], case["block"]
        p = -(-case["taps"] // b)
        return {"bytes": 8.0 * c * b + 8.0 * b * (c * p + c + case["irs"] * p), "flops": 8.0 * c * p * b + 10.0 * c * b * math.log2(2 * b)}
    if kind == "whole":
        c, length, taps = case["channels"], case["length"], case["taps"]
        full = length + taps - 1
        return {"bytes": 4.0 * (c * (length + full) + case["irs"] * taps), "flops": c * full * 5.0 * math.log2(full)}
    if kind == "oneshot":
        n = 2
        while n < case["length"] + case["taps"] - 1:
            n *= 2
        return {"bytes": 4.0 * case["signals"] * (case["length"] + n), "flops": case["signals"] * 5.0 * n * math.log2(n)}
    return {"bytes": 8.0 * case["channels"] * case["length"], "flops": 9.0 * case["channels"] * case["length"] * case["sections"]}


def tolerance(case):
    """About four times the largest error measured against the same computation in float64."""
    kind = case["kind"]
    if kind in ("clip", "stft"):
        # The spectra are good to 3e-7.  The first and last samples of a reconstruction are divided by
        # the square of a Hann window that starts at zero, which amplifies their rounding by 1/w: a
        # fixed error energy per signal, whose share falls with its length.
        return {"rel": 1e-6 + 0.026 * min(1.0, case["n"] / 4096) / math.sqrt(case["length"]), "max": 0.017}
    return {"rel": {"frame": 1.3e-6, "fft": 1.5e-6, "stream": 1.5e-6, "whole": 3.2e-6, "oneshot": 1.5e-6, "eq": 2e-7}[kind]}
