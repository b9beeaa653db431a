"""GPU parity of STFT / iSTFT against the float64 oracle and the float32 port."""
import numpy as np
import pytest

from oracle import float64 as o64
from oracle import reference_path as rp
from oracle import configs

pytestmark = pytest.mark.gpu
TOL = 1e-5


def interior(frames, n, hop, win, frac=1e-2):
    """Samples whose window sum is not vanishing: near the ends a symmetric window leaves
    sum(w^2) ~ 1e-8, where float32 rounding is amplified by 1/sum(w^2) in any implementation."""
    ws = rp.window_sum(frames, n, hop, win, 0.0)
    return ws >= frac * ws.max()


CASES = [(256, 64, 4000, "hann"), (512, 100, 5000, "hamming"), (64, 7, 700, "blackman"),
         (1024, 1024, 8192, "none"), (2048, 512, 40000, "hann"), (4096, 1024, 70000, "hann"),
         (8192, 2048, 70000, "hann"), (8, 2, 50, "hann"), (4, 1, 21, "hann"), (2, 1, 9, "none"),
         (256, 255, 3001, "hann"),
         # above 8192 points: the two-pass transforms with the window in the loader and a separate overlap-add
         (16384, 4096, 100000, "hann"), (32768, 8192, 140000, "hamming"), (65536, 65536, 200000, "none"),
         (16384, 1000, 60001, "blackman")]


@pytest.mark.parametrize("n,hop,length,kind", CASES)
def test_stft_istft_parity(device, n, hop, length, kind):
    from metalaudio_b200 import FFT, WindowType
    rng = np.random.default_rng(n * 7 + hop)
    x = rng.uniform(-1, 1, length).astype(np.float32)
    fft = FFT(device, FFT.Config(size=n, windowType=WindowType(kind), hopSize=hop))
    res = fft.stft(x)
    w = rp.window(kind, n)
    frames = (length - n) // hop + 1
    assert res.frameCount == frames and res.binCount == n
    ref = o64.stft(x, n, hop, w)
    full_ref = o64.fft_forward(x[np.arange(frames)[:, None] * hop + np.arange(n)[None, :]].astype(np.float64) * w)
    assert o64.rel_rms(res.real + 1j * res.imag, full_ref) <= TOL
    pre, pim = rp.stft(x, n, hop, w)
    assert o64.rel_rms(res.real + 1j * res.imag, pre + 1j * pim) <= TOL
    y = fft.istft(res)
    assert y.shape == ((frames - 1) * hop + n,)
    floor = float(rp.window_floor())
    yref = o64.istft(ref, n, hop, w, floor)
    m = interior(frames, n, hop, w)
    assert o64.rel_rms(y[m], yref[m]) <= TOL
    yport = rp.istft(pre, pim, n, hop, w)
    assert o64.rel_rms(y[m], yport[m]) <= TOL
    # the ends are bounded by the amplification 1/sum(w^2) of float32 rounding
    assert np.isfinite(y).all()
    ws = np.maximum(rp.window_sum(frames, n, hop, w, floor), floor)
    assert np.all(np.abs(y - yref) <= 1e-5 * np.sqrt(n) / np.sqrt(ws) + 1e-5)


# The batched half-spectrum calls have kernels of their own by hop: a quarter and a half of the frame (register
# rings), other multiples of the threads' span that divide the frame or not (thread-private ring), the rest, and short
# frames side by side in a CTA; lengths are odd where signals then start on odd samples.
BATCHED = [(8192, 4096, 40001, 5), (8192, 2048, 40960, 3), (8192, 2560, 50003, 2), (8192, 1024, 30000, 2), (8192, 8192, 60000, 2),
           (4096, 2048, 30001, 7), (4096, 1280, 30000, 3), (4096, 512, 20001, 2), (4096, 3072, 40000, 2), (4096, 1365, 20000, 2),
           (2048, 1024, 9001, 3), (2048, 640, 9000, 4), (1024, 512, 5000, 9), (1024, 320, 5001, 4), (512, 256, 4000, 5),
           (512, 160, 4001, 20), (256, 128, 3000, 4), (256, 80, 2999, 33), (256, 64, 3000, 3), (64, 32, 700, 40), (64, 20, 701, 3),
           (4096, 2048, 4096, 3), (8192, 4096, 12288, 1), (1024, 320, 1024, 2)]


@pytest.mark.parametrize("n,hop,length,signals", BATCHED)
def test_batched_half_spectra(device, n, hop, length, signals):
    """stftBatch with and without magnitudes and istftBatch, interleaved half spectra, against float64: the interior, the
    ends (rounding amplified by 1/sum(w^2)), and runs that repeat bit for bit."""
    from metalaudio_b200 import FFT
    x = np.random.default_rng(n + 3 * hop).uniform(-1, 1, (signals, length)).astype(np.float32)
    w = rp.periodic_hann(n)
    fft = FFT(device, FFT.Config(size=n, hopSize=hop), window=w)
    ref = o64.stft(x, n, hop, w)
    spec, mag = fft.stftBatch(x, magnitude=True)
    assert o64.rel_rms(spec, ref) <= 1e-6
    assert o64.rel_rms(mag, np.abs(ref)) <= 1e-6
    assert o64.rel_rms(fft.stftBatch(x), ref) <= 1e-6
    y = fft.istftBatch(spec)
    frames = ref.shape[1]
    floor = float(rp.window_floor())
    yref = o64.istft(ref, n, hop, w, floor)
    assert y.shape == yref.shape
    m = interior(frames, n, hop, w)
    # 1e-6 for sums of unit weight; where hops are wide the window sum dips to 1e-2 of its maximum, which divides the error
    assert o64.rel_rms(y[:, m], yref[:, m]) <= TOL
    ws = np.maximum(rp.window_sum(frames, n, hop, w, floor), floor)
    assert np.all(np.abs(y - yref) <= 1e-5 * np.sqrt(n) / np.sqrt(ws) + 1e-5)
    assert np.array_equal(fft.istftBatch(spec), y)


def test_stft_input_too_short(device):
    from metalaudio_b200 import FFT, FFTError
    fft = FFT(device, FFT.Config(size=256))
    with pytest.raises(FFTError) as e:
        fft.stft(np.zeros(100, np.float32))
    assert e.value.case == "inputTooShort" and e.value.inputSize == 100 and e.value.requiredSize == 256


def test_istft_empty(device):
    from metalaudio_b200 import FFT, STFTResult
    fft = FFT(device, FFT.Config(size=256))
    assert fft.istft(STFTResult(np.zeros((0, 256), np.float32), np.zeros((0, 256), np.float32))).size == 0


def test_config2_scaled_periodic_and_symmetric(device):
    """Benchmark configuration 2 at reduced signal count/length, with both window readings
    (periodic Hann as the configuration words it, symmetric as the reference computes it):
    half-spectrum complex + magnitude out, overlap-add reconstruction."""
    from metalaudio_b200 import FFT, WindowType
    n, hop = 4096, 1024
    x = configs.c2_signals(n_signals=6, length=1 << 16)
    for w in (rp.periodic_hann(n), rp.window("hann", n)):
        fft = FFT(device, FFT.Config(size=n, windowType=WindowType.hann, hopSize=hop), window=w)
        spec, mag = fft.stftBatch(x, magnitude=True)
        ref = o64.stft(x, n, hop, w)
        assert o64.rel_rms(spec, ref) <= TOL
        assert o64.rel_rms(mag, np.abs(ref)) <= TOL
        y = fft.istftBatch(spec)
        frames = spec.shape[1]
        m = interior(frames, n, hop, w)
        yref = o64.istft(ref, n, hop, w, float(rp.window_floor()))
        assert o64.rel_rms(y[:, m], yref[:, m]) <= TOL
        # COLA reconstruction of the input itself on the interior
        assert o64.rel_rms(y[:, m], x[:, :y.shape[1]][:, m]) <= TOL


def test_stft_bit_stable(device):
    from metalaudio_b200 import FFT
    fft = FFT(device, FFT.Config(size=512, hopSize=128))
    x = np.random.default_rng(1).uniform(-1, 1, 9000).astype(np.float32)
    a = fft.istft(fft.stft(x))
    b = fft.istft(fft.stft(x))
    assert np.array_equal(a, b)


def test_large_frames_many_signals_half_layout(device):
    """More frames than one scratch chunk holds (16384-point frames: 3027 per chunk) over two signals,
    half-spectrum layout with magnitudes, through the batched API."""
    from metalaudio_b200 import FFT, WindowType
    n, hop, length = 16384, 2048, 2048 * 3100 + 16384
    rng = np.random.default_rng(12)
    x = rng.uniform(-1, 1, (2, length)).astype(np.float32)
    fft = FFT(device, FFT.Config(size=n, windowType=WindowType.hann, hopSize=hop))
    spec, mag = fft.stftBatch(x, magnitude=True)
    frames = (length - n) // hop + 1
    assert spec.shape == (2, frames, n // 2 + 1) and frames > 3027
    w = rp.window("hann", n)
    pick = [0, 1, 3026, 3027, 3028, frames - 1]
    for s_ in range(2):
        fr = x[s_][np.array(pick)[:, None] * hop + np.arange(n)[None, :]].astype(np.float64) * w
        ref = np.fft.rfft(fr, axis=-1)
        assert o64.rel_rms(spec[s_, pick], ref) <= TOL
        assert o64.rel_rms(mag[s_, pick], np.abs(ref)) <= TOL
    y = fft.istftBatch(spec)
    m = interior(frames, n, hop, w)
    assert o64.rel_rms(y[:, m], x[:, :y.shape[1]][:, m]) <= TOL


def _istft_dev(lib, fft, spec, out, floor):
    import ctypes
    frames = spec.shape[1]
    assert lib.ma_istft_dev(fft._h, ctypes.c_void_p(spec.pointer), None, frames, spec.shape[0], ctypes.c_void_p(out.pointer),
                            out.shape[1], floor, 0) == 0


@pytest.mark.parametrize("n,hop,frames", [(4096, 1024, 12), (1024, 16, 200), (512, 160, 30), (4096, 1280, 9), (256, 256, 3)])
def test_istft_floor_changes_on_one_plan(lib, device, n, hop, frames):
    """The window sums are tabulated per plan and floor: a plan whose floor changes from call to call gives what the
    definition gives, at the ends of the signal too (Hann, floor up to 0.1: the outermost samples are divided by it)."""
    from metalaudio_b200 import FFT, Tensor
    w = rp.periodic_hann(n)
    fft = FFT(device, FFT.Config(size=n, hopSize=hop), window=w)
    rng = np.random.default_rng(n + hop)
    spec64 = rng.standard_normal((2, frames, n // 2 + 1)) + 1j * rng.standard_normal((2, frames, n // 2 + 1))
    spec64[..., 0] = spec64[..., 0].real
    spec64[..., -1] = spec64[..., -1].real
    half = np.stack([spec64.real, spec64.imag], -1).astype(np.float32)
    spec, out = Tensor(device, half.shape), Tensor(device, (2, (frames - 1) * hop + n))
    spec.copy(half)
    for floor in (0.1, 1e-3, 0.1):
        _istft_dev(lib, fft, spec, out, floor)
        device.synchronize()
        ref = o64.istft(half[..., 0].astype(np.float64) + 1j * half[..., 1], n, hop, w, floor)
        assert o64.rel_rms(out.toArray(), ref) <= TOL
    fft.close()


def test_first_istft_of_a_plan_with_many_overlaps(lib, device):
    """A plan's first iSTFT builds the window sums of both ends, 2N positions of up to N/hop frames each.  At 8192
    points and a hop of 1 that is 6.7e7 terms: 235 ms as a host loop, below a millisecond as a kernel."""
    import time

    from metalaudio_b200 import FFT, Tensor
    n, hop, frames = 8192, 1, 8
    spec, out = Tensor(device, (1, frames, n // 2 + 1, 2)), Tensor(device, (1, (frames - 1) * hop + n))
    spec.copy(np.zeros(spec.shape, np.float32))
    took = []
    for _ in range(3):   # a fresh plan each time; the first one also loads the kernels
        fft = FFT(device, FFT.Config(size=n, hopSize=hop), window=rp.periodic_hann(n))
        device.synchronize()
        t = time.perf_counter()
        _istft_dev(lib, fft, spec, out, 1e-3)
        device.synchronize()
        took.append(time.perf_counter() - t)
        fft.close()
    assert min(took[1:]) < 0.06
