"""GPU parity of the multichannel biquad cascades against the float32 recurrence port and its
float64 evaluation (Sources/MetalDSP/Filters.swift:515-537; Shaders/DSP.metal:709-744), plus the
behavioural cases of Tests/MetalDSPTests/FilterTests.swift that reach the sample path."""
import ctypes

import numpy as np
import pytest

from oracle import float64 as o64
from oracle import reference_path as rp

pytestmark = pytest.mark.gpu
TOL = 1e-5

KINDS = [("lowpass", 0.0), ("highpass", 0.0), ("bandpass", 0.0), ("notch", 0.0), ("allpass", 0.0),
         ("peaking", 6.0), ("lowshelf", -9.0), ("highshelf", 4.5)]


def ftype(kind, gain):
    from metalaudio_b200 import BiquadFilter
    T = BiquadFilter.FilterType
    return getattr(T, kind)(gain) if kind in ("peaking", "lowshelf", "highshelf") else getattr(T, kind)


@pytest.mark.parametrize("kind,gain", KINDS)
@pytest.mark.parametrize("length", [1, 31, 1000, 8192, 8193, 50000])
def test_single_channel_matches_port_and_float64(device, kind, gain, length):
    from metalaudio_b200 import BiquadFilter
    rng = np.random.default_rng(length + len(kind))
    x = rng.standard_normal(length).astype(np.float32)
    f = BiquadFilter(device)
    f.configure(ftype(kind, gain), 1500.0, 44100.0, 0.9)
    c = rp.biquad_coefficients(kind, 1500.0, 44100.0, 0.9, gain)
    assert np.array_equal(f.currentCoefficients.asArray(), c)
    y = f.process(x)
    y64, z64 = rp.biquad_process(x, c, dtype=np.float64)
    y32, _ = rp.biquad_process(x, c)
    scale = max(float(np.sqrt(np.mean(y64 ** 2))), 1e-30)
    assert float(np.sqrt(np.mean((y - y64) ** 2))) / scale < TOL
    assert float(np.sqrt(np.mean((y - y32) ** 2))) / scale < TOL
    assert np.max(np.abs(f.delays[0] - z64)) < 1e-4 * max(1.0, float(np.max(np.abs(z64))))


def test_state_carries_across_calls_and_reset(device):
    """Streaming in uneven pieces equals one call; reset() restores the initial state
    (testFilterReset, testBatchVsSingleSampleConsistency)."""
    from metalaudio_b200 import BiquadFilter
    rng = np.random.default_rng(3)
    x = rng.standard_normal(30000).astype(np.float32)
    f = BiquadFilter(device)
    f.configure(BiquadFilter.FilterType.lowpass, 800.0, 48000.0, 4.0)
    whole = f.process(x)
    f.reset()
    parts = np.concatenate([f.process(x[a:b]) for a, b in [(0, 1), (1, 100), (100, 8292), (8292, 8293), (8293, 30000)]])
    assert o64.rel_rms(parts, whole) < TOL     # same arithmetic up to where the block boundaries fall
    f.reset()
    assert np.allclose(f.process(x[:500]), whole[:500], atol=1e-6)
    f.reset()
    singles = np.array([f.process(sample=float(v)) for v in x[:40]], np.float32)
    assert np.allclose(singles, whole[:40], atol=1e-6)
    assert f.process(np.zeros(0, np.float32)).size == 0


def test_high_q_long_signal_stays_accurate(device):
    """testHighQFilter / testLongTermStability: poles close to the unit circle, a million samples."""
    from metalaudio_b200 import BiquadFilter
    rng = np.random.default_rng(9)
    x = (0.1 * rng.standard_normal(1 << 20)).astype(np.float32)
    f = BiquadFilter(device)
    f.configure(BiquadFilter.FilterType.bandpass, 440.0, 48000.0, 30.0)
    y = f.process(x)
    c = rp.biquad_coefficients("bandpass", 440.0, 48000.0, 30.0)
    y64, _ = rp.biquad_process(x, c, dtype=np.float64)
    assert np.all(np.isfinite(y))
    # at Q = 30 the float32 recurrence itself sits at 1.6e-5 of the float64 result (rounding noise
    # is amplified by the resonance); the GPU path must be no worse than that serial float32 port
    y32, _ = rp.biquad_process(x, c)
    assert o64.rel_rms(y, y64) < max(TOL, 1.25 * o64.rel_rms(y32, y64))
    assert f.isStable


def test_many_channels_per_channel_coefficients_device_pointers(device, lib):
    """The C ABI on device memory: 70 channels, 5 coefficient sets, 3 cascaded sections, strided rows."""
    import torch
    rng = np.random.default_rng(4)
    C, S, L, stride = 70, 3, 20011, 20480
    sets = np.stack([np.stack([rp.biquad_coefficients(k, fr, 48000.0, q, g) for (k, g), fr, q in
                               zip([KINDS[(i + j) % 8] for j in range(S)], (300.0 + 700 * i, 2500.0, 9000.0), (0.7, 2.0, 1.2))])
                     for i in range(5)])                       # (5, S, 5)
    cmap = (np.arange(C) % 5).astype(np.int32)
    x = rng.standard_normal((C, stride)).astype(np.float32)
    h = ctypes.c_void_p()
    assert lib.ma_biquad_create(device.handle, C, S, ctypes.byref(h)) == 0
    assert lib.ma_biquad_set_coefficients(h, sets.ctypes.data, 5, cmap.ctypes.data) == 0
    dx = torch.from_numpy(x).cuda()
    dy = torch.zeros((C, stride), device="cuda")
    torch.cuda.synchronize()
    half = 9000
    for a, b in [(0, half), (half, L)]:           # two calls: the states carry over per channel and section
        assert lib.ma_biquad_process_dev(h, ctypes.c_void_p(dx.data_ptr() + 4 * a), stride,
                                         ctypes.c_void_p(dy.data_ptr() + 4 * a), stride, b - a) == 0
    device.synchronize(10)
    y = dy.cpu().numpy()
    assert np.all(y[:, L:] == 0)
    state = np.empty((C, S, 2), np.float32)
    assert lib.ma_biquad_get_state(h, state.ctypes.data) == 0
    for c in (0, 1, 33, C - 1):
        ref = x[c, :L].astype(np.float64)
        for s in range(S):
            ref, z = rp.biquad_process(ref, sets[cmap[c], s], dtype=np.float64)
            assert np.max(np.abs(state[c, s] - z)) < 1e-4 * max(1.0, float(np.max(np.abs(z))))
        assert o64.rel_rms(y[c, :L], ref) < TOL
    assert lib.ma_biquad_reset(h) == 0
    device.synchronize(10)
    assert lib.ma_biquad_get_state(h, state.ctypes.data) == 0 and np.all(state == 0)
    assert lib.ma_biquad_destroy(h) == 0


def test_filter_bank_series_and_parallel(device):
    """FilterBank (testFilterBankProcessing, ...SetBandGain, ...SeriesVsParallelDifference)."""
    from metalaudio_b200 import FilterBank, FilterError
    rng = np.random.default_rng(8)
    x = rng.standard_normal(12000).astype(np.float32)
    bank = FilterBank(device, bandCount=5)
    bank.configureAsEQ(100.0, 10000.0, 44100.0)
    flat = bank.processSeries(x)
    assert o64.rel_rms(flat, x) < 1e-5                     # 0 dB peaking bands are identities
    freqs = [100.0 * (100.0 ** (i / 4)) for i in range(5)]
    gains = [6.0, -3.0, 0.0, 4.0, -8.0]
    for i, (fr, g) in enumerate(zip(freqs, gains)):
        bank.setBandGain(i, g, fr, 44100.0)
    bank.reset()
    series = bank.processSeries(x)
    bank.reset()
    parallel = bank.processParallel(x)
    cs = [rp.biquad_coefficients("peaking", fr, 44100.0, 1.414, g) for fr, g in zip(freqs, gains)]
    ref = x.astype(np.float64)
    for c in cs:
        ref, _ = rp.biquad_process(ref, c, dtype=np.float64)
    assert o64.rel_rms(series, ref) < TOL
    refp = sum(rp.biquad_process(x, c, dtype=np.float64)[0] for c in cs) / 5.0
    assert o64.rel_rms(parallel, refp) < TOL
    assert o64.rel_rms(series, parallel) > 1e-2
    with pytest.raises(FilterError) as e:
        bank.setBandGain(5, 1.0, 1000.0, 44100.0)
    assert e.value.name == "band"
    with pytest.raises(FilterError):
        FilterBank(device, bandCount=1).configureAsEQ(100.0, 1000.0, 44100.0)


def test_filter_bank_state_carries_between_series_and_parallel(device):
    """The reference runs processSeries and processParallel over the same per-band filters, so a
    band's state survives a switch between the two.  Mirrored by handing the state across: a
    parallel call after a series call continues every band from the state the series call left."""
    from metalaudio_b200 import FilterBank, FilterError
    rng = np.random.default_rng(12)
    bands, n = 4, 3000
    bank = FilterBank(device, bandCount=bands)
    bank.configureAsEQ(100.0, 8000.0, 44100.0)
    for b in range(bands):
        bank.setBandGain(b, 6.0 - 3.0 * b, 200.0 * (b + 1), 44100.0)
    coeffs = np.stack([c.asArray() for c in bank._coeffs])
    x1 = rng.standard_normal(n).astype(np.float32)
    x2 = rng.standard_normal(n).astype(np.float32)
    y1 = bank.processSeries(x1)
    y2 = bank.processParallel(x2)
    # oracle: the cascade on x1 leaves per-band states; each band then filters x2 from its own state
    cur, states = x1.astype(np.float64), []
    for b in range(bands):
        cur, st = rp.biquad_process(cur, coeffs[b], dtype=np.float64)
        states.append(st)
    assert o64.rel_rms(y1, cur) <= TOL
    mix = np.zeros(n)
    for b in range(bands):
        yb, _ = rp.biquad_process(x2.astype(np.float64), coeffs[b], state=states[b], dtype=np.float64)
        mix += yb
    assert o64.rel_rms(y2, mix / bands) <= TOL
    with pytest.raises(FilterError) as e:
        FilterBank(device, bandCount=33)
    assert e.value.name == "bandCount"
    bank.close()


@pytest.mark.parametrize("channels,sections", [(1, 1), (3, 2), (24, 4), (98, 3), (2, 8), (5, 9)])
@pytest.mark.parametrize("tiles,extra", [(3, 0), (4, 1), (5, -1), (70, 5)])
def test_time_splits_match_float64(device, lib, channels, sections, tiles, extra):
    """Few channels: the time axis is cut into chunks that run on CTAs of their own (up to eight sections).
    Edges of tiles and chunks, several coefficient sets, the state in front of and behind the call, in
    place and into other rows.  A tile is 8192 samples, 4096 from three sections up."""
    from metalaudio_b200 import Tensor
    length = tiles * (4096 if sections >= 3 else 8192) + extra
    if channels > 30 and tiles > 10:
        channels = 30
    rng = np.random.default_rng(100 * channels + sections + tiles)
    kinds = [("lowpass", 0.0), ("peaking", 6.0), ("highpass", 0.0), ("lowshelf", -9.0)]
    sets = min(channels, 3)
    coef = np.stack([[rp.biquad_coefficients(kinds[(k + s) % 4][0], 60.0 * 2.0 ** ((k + s) % 8), 48000.0, 0.9, kinds[(k + s) % 4][1])
                      for s in range(sections)] for k in range(sets)]).astype(np.float32)
    of_channel = (np.arange(channels) % sets).astype(np.int32)
    x = rng.standard_normal((channels, length)).astype(np.float32)
    z0 = (0.01 * rng.standard_normal((channels, sections, 2))).astype(np.float32)
    h = ctypes.c_void_p()
    vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.ma_biquad_create(device.handle, channels, sections, ctypes.byref(h)) == 0
    try:
        assert lib.ma_biquad_set_coefficients(h, vp(coef), sets, vp(of_channel)) == 0
        ref = np.empty((channels, length))
        zref = np.empty((channels, sections, 2))
        for c in range(channels):
            y = x[c].astype(np.float64)
            for s in range(sections):
                y, zref[c, s] = rp.biquad_process(y, coef[of_channel[c], s], z0[c, s].astype(np.float64), dtype=np.float64)
            ref[c] = y
        tin = Tensor(device, x.shape)
        for in_place in (False, True):
            tin.copy(x)
            tout = tin if in_place else Tensor(device, x.shape)
            assert lib.ma_biquad_set_state(h, vp(z0)) == 0
            assert lib.ma_biquad_process_dev(h, ctypes.c_void_p(tin.pointer), length, ctypes.c_void_p(tout.pointer), length, length) == 0
            device.synchronize()
            assert max(o64.rel_rms(a, b) for a, b in zip(tout.toArray(), ref)) <= TOL
            z = np.empty_like(z0)
            assert lib.ma_biquad_get_state(h, vp(z)) == 0
            assert np.max(np.abs(z - zref)) <= 1e-4 * max(1.0, float(np.max(np.abs(zref))))
    finally:
        lib.ma_biquad_destroy(h)


def test_coefficients_that_cannot_be_stored(device, lib):
    """ma_biquad_set_coefficients without the memory for one of its arrays: a channel map that cannot be had leaves the
    old coefficients of every channel in force; the tables of the time splits are only for speed, without them the call
    succeeds and the cascade runs unsplit."""
    from metalaudio_b200 import Tensor
    from metalaudio_b200 import _lib as L
    channels, length = 3, 70 * 8192
    x = np.random.default_rng(9).standard_normal((channels, length)).astype(np.float32)
    designs = [rp.biquad_coefficients("peaking", f, 48000.0, 1.0, 6.0) for f in (100.0, 1000.0, 5000.0, 9000.0)]
    old = np.array(designs[:2], np.float32)[:, None, :]
    new = np.array(designs[2:], np.float32)[:, None, :]
    old_map, new_map = np.array([0, 1, 0], np.int32), np.array([1, 0, 1], np.int32)
    vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    h = ctypes.c_void_p()
    assert lib.ma_biquad_create(device.handle, channels, 1, ctypes.byref(h)) == 0
    tin, tout = Tensor(device, x.shape), Tensor(device, x.shape)
    tin.copy(x)

    def run(coefs, of_channel):
        before = lib.ma_kernel_launch_count()
        assert lib.ma_biquad_reset(h) == 0
        assert lib.ma_biquad_process_dev(h, ctypes.c_void_p(tin.pointer), length, ctypes.c_void_p(tout.pointer), length, length) == 0
        device.synchronize()
        for c in range(channels):
            ref, _ = rp.biquad_process(x[c].astype(np.float64), coefs[of_channel[c], 0], dtype=np.float64)
            assert o64.rel_rms(tout.toArray()[c], ref) <= TOL
        return lib.ma_kernel_launch_count() - before
    try:
        assert lib.ma_biquad_set_coefficients(h, vp(old), 2, vp(old_map)) == 0
        assert run(old, old_map) == 2      # split: end states, then chunks
        assert lib.ma_test_inject_fault(device.handle, L.FAULT_BIQUAD_MAP, 2) == 0   # cudaErrorMemoryAllocation
        assert lib.ma_biquad_set_coefficients(h, vp(new), 2, vp(new_map)) == L.MA_ERR_ALLOC
        assert run(old, old_map) == 2
        assert lib.ma_test_inject_fault(device.handle, L.FAULT_BIQUAD_LADDER, 2) == 0
        assert lib.ma_biquad_set_coefficients(h, vp(new), 2, vp(new_map)) == 0
        assert run(new, new_map) == 1
        assert lib.ma_biquad_set_coefficients(h, vp(new), 2, vp(new_map)) == 0
        assert run(new, new_map) == 2
    finally:
        lib.ma_biquad_destroy(h)


def test_time_splits_of_very_long_channels(device, lib):
    """74 channels, the most that are split, so long that a chunk holds more than 511 tiles: still split, and the last
    chunk's samples are the filter's."""
    import torch
    channels, sections, length = 74, 3, 4 * 513 * 4096 - 77
    coef = np.stack([rp.biquad_coefficients("lowpass", 200.0, 48000.0, 4.0, 0.0), rp.biquad_coefficients("peaking", 40.0, 48000.0, 8.0, 9.0),
                     rp.biquad_coefficients("highpass", 30.0, 48000.0, 0.7, 0.0)]).astype(np.float32)
    x = torch.rand((channels, length), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)) * 2.0 - 1.0
    picked = {c: x[c].cpu().numpy().astype(np.float64) for c in (0, 73)}
    torch.cuda.synchronize()
    h = ctypes.c_void_p()
    assert lib.ma_biquad_create(device.handle, channels, sections, ctypes.byref(h)) == 0
    try:
        assert lib.ma_biquad_set_coefficients(h, coef.ctypes.data_as(ctypes.c_void_p), 1, None) == 0
        before = lib.ma_kernel_launch_count()
        assert lib.ma_biquad_process_dev(h, ctypes.c_void_p(x.data_ptr()), length, ctypes.c_void_p(x.data_ptr()), length, length) == 0
        assert lib.ma_kernel_launch_count() - before == 2   # end states, then chunks
        device.synchronize(30)
        for c, y in picked.items():
            for s in range(sections):
                y, _ = rp.biquad_process(y, coef[s], dtype=np.float64)
            assert o64.rel_rms(x[c].cpu().numpy(), y) <= TOL
    finally:
        lib.ma_biquad_destroy(h)
