"""The pipelined host forms (ma_stft_host, ma_istft_host, ma_pconv_process_host) on PINNED host arrays:
chunks travel on three streams through two workspace lanes.  A small workspace forces several chunks,
so every lane is reused; results must equal the pageable path's bit for bit (same kernels, same
chunk-independent arithmetic) and agree with the float64 oracle."""
import ctypes

import numpy as np
import pytest

from oracle import float64 as o64

pytestmark = pytest.mark.gpu
TOL = 1e-5


class Pinned:
    """float32 numpy views of page-locked host memory from ma_host_alloc."""

    def __init__(self, lib, dev):
        self.lib, self.dev, self.ptrs = lib, dev, []

    def array(self, shape):
        n = int(np.prod(shape))
        p = ctypes.c_void_p()
        assert self.lib.ma_host_alloc(self.dev.handle, 4 * max(n, 1), ctypes.byref(p)) == 0
        self.ptrs.append(p)
        a = np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_float)), shape=(max(n, 1),))[:n]
        return a.reshape(shape)

    def close(self):
        for p in self.ptrs:
            assert self.lib.ma_host_free(self.dev.handle, p) == 0
        self.ptrs = []


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.fixture()
def small_device(lib):
    """A context of its own whose workspace lanes hold only a few rows."""
    from metalaudio_b200 import AudioDevice
    dev = AudioDevice()
    yield dev
    dev.close()


def test_convolution_host_pinned_groups(lib, small_device):
    """12 channels with per-pair impulse responses (groups of two stay together), strided host rows,
    workspace of 2 x 200 KB: three chunks of two groups.  Two consecutive calls."""
    from metalaudio_b200 import Convolution
    dev = small_device
    assert lib.ma_context_reserve_workspace(dev.handle, 400 << 10) == 0
    block, taps, length, channels = 64, 300, 5000, 12
    full = length + taps - 1
    rng = np.random.default_rng(12)
    irs = (rng.standard_normal((channels // 2, taps)) * np.exp(-np.arange(taps) / 80.0)).astype(np.float32)
    cmap = [c // 2 for c in range(channels)]
    pin = Pinned(lib, dev)
    try:
        in_stride, out_stride = length + 24, full + 40
        x = pin.array((channels, in_stride))
        y = pin.array((channels, out_stride))
        for call in range(2):
            x[:] = rng.standard_normal(x.shape).astype(np.float32)
            y[:] = -7.0
            c_pin = Convolution(dev, Convolution.Mode.partitioned(blockSize=block), channels=channels)
            c_pin.setKernel(irs, channelToKernel=cmap)
            c_page = Convolution(dev, Convolution.Mode.partitioned(blockSize=block), channels=channels)
            c_page.setKernel(irs, channelToKernel=cmap)
            for _ in range(call + 1):  # the second round checks a call that follows another on the same object
                assert lib.ma_pconv_process_host(c_pin._h, ptr(x), length, in_stride, ptr(y), out_stride) == 0
                ref_page = c_page.process(np.ascontiguousarray(x[:, :length]))
            assert np.array_equal(y[:, :full], ref_page)
            assert np.all(y[:, full:] == -7.0)  # nothing written beyond a row's L+K-1 samples
            for c in (0, 5, 11):
                assert o64.rel_rms(y[c, :full], o64.convolve_full(x[c, :length], irs[cmap[c]])) <= TOL
    finally:
        pin.close()


def test_stft_istft_host_pinned_chunks(lib, small_device):
    """9 signals of 30000 samples, N = 1024, hop 256, workspace of 2 x 1.5 MB: the signals go through in
    chunks of two.  Spectra, magnitudes and the reconstruction equal the pageable path's."""
    from metalaudio_b200 import FFT, WindowType
    from metalaudio_b200 import _lib as L
    dev = small_device
    assert lib.ma_context_reserve_workspace(dev.handle, 3 << 20) == 0
    n, hop, signals, length = 1024, 256, 9, 30000
    f = FFT(dev, FFT.Config(size=n, windowType=WindowType.hann, hopSize=hop))
    frames = f.frameCount(length)
    kh = n // 2 + 1
    out_len = (frames - 1) * hop + n
    rng = np.random.default_rng(9)
    pin = Pinned(lib, dev)
    try:
        x = pin.array((signals, length))
        spec = pin.array((signals, frames, kh, 2))
        mag = pin.array((signals, frames, kh))
        y = pin.array((signals, out_len))
        x[:] = rng.standard_normal(x.shape).astype(np.float32)
        assert lib.ma_stft_host(f._h, ptr(x), length, length, signals, ptr(spec), None, ptr(mag), L.MAG_MAGNITUDE, 1.0,
                                L.LAYOUT_HALF_INTERLEAVED) == 0
        spec_page, mag_page = f.stftBatch(np.array(x), magnitude=True)
        assert np.array_equal(spec.view(np.complex64).reshape(signals, frames, kh), spec_page)
        assert np.array_equal(mag, mag_page)
        from metalaudio_b200.dsp import validatedWindowFloor
        assert lib.ma_istft_host(f._h, ptr(spec), None, frames, signals, ptr(y), out_len, validatedWindowFloor(),
                                 L.LAYOUT_HALF_INTERLEAVED) == 0
        assert np.array_equal(y, f.istftBatch(spec_page))
        inner = slice(n, length - n)
        assert o64.rel_rms(y[:, inner], x[:, inner]) <= TOL
    finally:
        pin.close()


@pytest.mark.parametrize("n,batch", [(4096, 700), (65536, 40)])
def test_plain_transforms_host_pinned_chunks(lib, small_device, n, batch):
    """Batches above the pipeline threshold between pinned arrays, workspace of 2 x 4 MB: forward (with
    magnitudes) and inverse run in several chunks and equal the pageable path's results."""
    from metalaudio_b200 import FFT, WindowType
    from metalaudio_b200 import _lib as L
    dev = small_device
    assert lib.ma_context_reserve_workspace(dev.handle, 8 << 20) == 0
    f = FFT(dev, FFT.Config(size=n, windowType=WindowType.none))
    kh = n // 2 + 1
    rng = np.random.default_rng(n + batch)
    pin = Pinned(lib, dev)
    try:
        x = pin.array((batch, n))
        spec = pin.array((batch, kh, 2))
        mag = pin.array((batch, kh))
        y = pin.array((batch, n))
        x[:] = rng.standard_normal(x.shape).astype(np.float32)
        assert lib.ma_fft_forward_host(f._h, ptr(x), ptr(spec), None, ptr(mag), L.MAG_MAGNITUDE, 1.0, batch,
                                       L.LAYOUT_HALF_INTERLEAVED) == 0
        xs = np.array(x)
        spec_page = np.zeros((batch, kh, 2), np.float32)
        mag_page = np.zeros((batch, kh), np.float32)
        assert lib.ma_fft_forward_host(f._h, ptr(xs), ptr(spec_page), None, ptr(mag_page), L.MAG_MAGNITUDE, 1.0, batch,
                                       L.LAYOUT_HALF_INTERLEAVED) == 0
        assert np.array_equal(spec, spec_page) and np.array_equal(mag, mag_page)
        pick = [0, batch // 2, batch - 1]
        assert o64.rel_rms(spec[pick, :, 0] + 1j * spec[pick, :, 1], o64.rfft(xs[pick])) <= TOL
        assert lib.ma_fft_inverse_host(f._h, ptr(spec), None, ptr(y), batch, L.LAYOUT_HALF_INTERLEAVED) == 0
        y_page = np.zeros((batch, n), np.float32)
        assert lib.ma_fft_inverse_host(f._h, ptr(spec_page), None, ptr(y_page), batch, L.LAYOUT_HALF_INTERLEAVED) == 0
        assert np.array_equal(y, y_page)
        assert o64.rel_rms(y, xs) <= TOL
    finally:
        pin.close()


@pytest.mark.parametrize("kind,pinned", [("frame", (True, True)), ("frame", (True, False)), ("frame", (False, False)),
                                         ("stft", (True, True)), ("stft", (True, False)), ("stft", (False, False))])
def test_two_threads_with_an_object_each_on_one_context(lib, small_device, kind, pinned):
    """Two threads, each with its own FFT object and arrays on ONE context: single frames (small calls through
    the staging buffer) and STFTs of several MiB (threaded copies, workspace lanes).  Both must get what a single
    thread gets, bit for bit."""
    import threading

    from metalaudio_b200 import FFT, WindowType
    from metalaudio_b200 import _lib as L
    dev = small_device
    assert lib.ma_context_reserve_workspace(dev.handle, 8 << 20) == 0
    n, rounds = (2048, 300) if kind == "frame" else (1024, 8)
    signals, length, hop = 6, 200000, 256
    pin = Pinned(lib, dev)
    try:
        calls, results = [], []
        for k in range(2):
            f = FFT(dev, FFT.Config(size=n, windowType=WindowType.none, hopSize=hop))
            array = pin.array if pinned[k] else lambda shape: np.zeros(shape, np.float32)
            rng = np.random.default_rng(70 + k)
            if kind == "frame":
                x, re, im, back = (array((n,)) for _ in range(4))
                mag = array((n // 2 + 1,))
                frames = rng.standard_normal((rounds, n)).astype(np.float32)

                def call(i, f=f, x=x, re=re, im=im, back=back, mag=mag, frames=frames):
                    x[:] = frames[i]
                    assert lib.ma_fft_forward_host(f._h, ptr(x), ptr(re), ptr(im), None, 0, 1.0, 1, L.LAYOUT_FULL_SPLIT) == 0
                    assert lib.ma_fft_magnitude_host(f._h, ptr(re), ptr(im), ptr(mag), 1, L.MAG_MAGNITUDE, 1.0) == 0
                    assert lib.ma_fft_inverse_host(f._h, ptr(re), ptr(im), ptr(back), 1, L.LAYOUT_FULL_SPLIT) == 0
                    return [a.copy() for a in (re, im, mag, back)]
            else:
                x = array((signals, length))
                spec = array((signals, f.frameCount(length), n // 2 + 1, 2))
                base = rng.standard_normal(x.shape).astype(np.float32)

                def call(i, f=f, x=x, spec=spec, base=base):
                    x[:] = base * np.float32(i + 1)
                    assert lib.ma_stft_host(f._h, ptr(x), length, length, signals, ptr(spec), None, None, 0, 1.0,
                                            L.LAYOUT_HALF_INTERLEAVED) == 0
                    return [spec.copy()]
            calls.append(call)
            results.append([call(i) for i in range(rounds)])
        got, failed = [[], []], []

        def work(k):
            try:
                got[k] = [calls[k](i) for i in range(rounds)]
            except AssertionError as e:
                failed.append(e)
        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(120)
        assert not failed
        for k in range(2):
            assert len(got[k]) == rounds
            for a, b in zip(got[k], results[k]):
                assert all(np.array_equal(p, q) for p, q in zip(a, b))
    finally:
        pin.close()


@pytest.mark.parametrize("n,batch", [(2048, 12), (2048, 13), (16384, 1), (16384, 2)])
@pytest.mark.parametrize("pinned", [True, False])
def test_small_calls_around_their_threshold(lib, small_device, n, batch, pinned):
    """Plain transforms just below and above the 256 KiB that go through the staging buffer as one transfer each
    way, in place as well (the input array is the output array of the inverse)."""
    from metalaudio_b200 import FFT, WindowType
    from metalaudio_b200 import _lib as L
    dev = small_device
    f = FFT(dev, FFT.Config(size=n, windowType=WindowType.none))
    kh = n // 2 + 1
    pin = Pinned(lib, dev)
    try:
        array = pin.array if pinned else lambda shape: np.zeros(shape, np.float32)
        x, spec, mag = array((batch, n)), array((batch, kh, 2)), array((batch, kh))
        x[:] = np.random.default_rng(n + batch).standard_normal(x.shape)
        keep = np.array(x)
        assert lib.ma_fft_forward_host(f._h, ptr(x), ptr(spec), None, ptr(mag), L.MAG_MAGNITUDE, 1.0, batch,
                                       L.LAYOUT_HALF_INTERLEAVED) == 0
        ref = o64.rfft(keep)
        assert o64.rel_rms(spec[..., 0] + 1j * spec[..., 1], ref) <= TOL
        assert o64.rel_rms(mag, np.abs(ref)) <= TOL
        assert lib.ma_fft_inverse_host(f._h, ptr(spec), None, ptr(spec), batch, L.LAYOUT_HALF_INTERLEAVED) == 0
        assert o64.rel_rms(spec.reshape(-1)[:batch * n].reshape(batch, n), keep) <= TOL
    finally:
        pin.close()


@pytest.mark.parametrize("nbytes", [(2 << 20) - 4, 2 << 20, (2 << 20) + 4, (64 << 20) - 4, (64 << 20) + 8, 130 << 20])
def test_pageable_copies_around_the_threaded_threshold(lib, small_device, nbytes):
    """ma_memcpy_h2d / _d2h of pageable arrays from one thread's double buffering to four threads' pieces, and across
    several fillings of the 64 MiB staging buffer; bytes past either end stay."""
    dev = small_device
    count = nbytes // 4
    x = np.random.default_rng(nbytes).integers(-2**31, 2**31, count + 2, dtype=np.int64).astype(np.int32)
    y = np.full(count + 2, 77, np.int32)
    d = ctypes.c_void_p()
    assert lib.ma_buffer_alloc(dev.handle, nbytes + 8, ctypes.byref(d)) == 0
    try:
        assert lib.ma_buffer_zero(dev.handle, d, nbytes + 8) == 0
        assert lib.ma_memcpy_h2d(dev.handle, ctypes.c_void_p(d.value + 4), ctypes.c_void_p(x.ctypes.data + 4), nbytes - 4) == 0
        assert lib.ma_memcpy_d2h(dev.handle, ctypes.c_void_p(y.ctypes.data), d, nbytes + 4) == 0
        assert y[0] == 0 and np.array_equal(y[1:count], x[1:count]) and y[count] == 0 and y[count + 1] == 77
    finally:
        assert lib.ma_buffer_free(dev.handle, d) == 0
