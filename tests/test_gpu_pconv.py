"""GPU parity of uniformly partitioned convolution against the float32 port of the
reference's block loop and the float64 linear-convolution oracle."""
import ctypes

import numpy as np
import pytest

from oracle import float64 as o64
from oracle import reference_path as rp
from oracle import configs

pytestmark = pytest.mark.gpu
TOL = 1e-5


def conv(device, block, channels=1):
    from metalaudio_b200 import Convolution
    return Convolution(device, Convolution.Mode.partitioned(blockSize=block), channels=channels)


def test_identity_kernel(device):
    """ConvolutionTests: delta kernel, block 64, 256-sample ramp reproduces the input."""
    c = conv(device, 64)
    c.setKernel(np.array([1.0], np.float32))
    x = np.arange(256, dtype=np.float32) / 256
    y = c.process(x)
    assert y.shape == (256,)
    assert np.max(np.abs(y - x)) < 100 * 1e-6


@pytest.mark.parametrize("block,taps,length", [(64, 1, 256), (64, 64, 640), (64, 200, 1000), (128, 1000, 5000),
                                               (256, 4096, 10000), (512, 3000, 7777), (1, 5, 17), (2, 7, 33),
                                               (4, 9, 40), (16, 100, 333), (1024, 5000, 9000), (4096, 9000, 20000)])
def test_process_matches_port_and_oracle(device, block, taps, length):
    rng = np.random.default_rng(block + taps)
    h = (rng.standard_normal(taps) * np.exp(-np.arange(taps) / max(1, taps / 4))).astype(np.float32)
    x = rng.standard_normal(length).astype(np.float32)
    c = conv(device, block)
    c.setKernel(h)
    assert c.partitionCount == (taps + block - 1) // block
    y = c.process(x)
    assert y.shape == (length + taps - 1,)
    ref = o64.convolve_full(x, h)
    assert o64.rel_rms(y, ref) <= TOL
    port = rp.PartitionedConvolution(block)
    port.set_kernel(h)
    assert o64.rel_rms(y, port.process(x)) <= TOL
    assert c.expectedOutputSize(length) == length + taps - 1 and c.kernelTailLength == taps - 1
    assert c.maxInputSize == 0


def test_consecutive_calls_and_reset(device):
    """The delay line survives across process() calls (Convolution.swift ring semantics), but
    every call pushes ceil((L+K-1)/B) >= ceil(L/B) + P - 1 blocks, so the input-bearing
    spectra have aged out of reach (p <= P-1) by the next call: consecutive calls agree with
    the port and with a fresh convolution.  reset() then same input -> same output, bit-stable."""
    block, taps = 64, 257
    rng = np.random.default_rng(4)
    h = rng.standard_normal(taps).astype(np.float32)
    x1 = rng.standard_normal(128).astype(np.float32)
    x2 = rng.standard_normal(500).astype(np.float32)
    c = conv(device, block)
    c.setKernel(h)
    port = rp.PartitionedConvolution(block)
    port.set_kernel(h)
    a1, p1 = c.process(x1), port.process(x1)
    a2, p2 = c.process(x2), port.process(x2)
    assert o64.rel_rms(a1, p1) <= TOL and o64.rel_rms(a2, p2) <= TOL
    assert o64.rel_rms(a2, o64.convolve_full(x2, h)) <= TOL
    c.reset()
    a3 = c.process(x2)
    assert np.array_equal(a3, a2)
    c.reset()
    assert np.array_equal(c.process(x2), a3)


def test_multichannel_shared_and_per_pair_irs(device):
    block, taps, length, ch = 64, 1000, 3000, 8
    rng = np.random.default_rng(8)
    x = (0.1 * rng.standard_normal((ch, length))).astype(np.float32)
    # shared IR (configuration 3 shape)
    h = configs.decaying_ir(taps, 77, rt60_s=0.01)
    c = conv(device, block, channels=ch)
    c.setKernel(h)
    y = c.process(x)
    for i in range(ch):
        assert o64.rel_rms(y[i], o64.convolve_full(x[i], h)) <= TOL
    # one IR per channel pair (configuration 4 shape)
    hs = np.stack([configs.decaying_ir(taps, [78, i], rt60_s=0.01) for i in range(ch // 2)])
    c2 = conv(device, block, channels=ch)
    c2.setKernel(hs, channelToKernel=[i // 2 for i in range(ch)])
    y2 = c2.process(x)
    for i in range(ch):
        assert o64.rel_rms(y2[i], o64.convolve_full(x[i], hs[i // 2])) <= TOL
    # arbitrary mapping, odd channel count
    c3 = conv(device, block, channels=3)
    c3.setKernel(hs, channelToKernel=[2, 0, 2])
    y3 = c3.process(x[:3])
    for i, ir in enumerate([2, 0, 2]):
        assert o64.rel_rms(y3[i], o64.convolve_full(x[i], hs[ir])) <= TOL


@pytest.mark.parametrize("block,taps,channels", [(64, 1000, 4), (256, 5000, 3), (1, 3, 2), (2, 9, 5), (32, 700, 8), (64, 30, 2),
                                                 (128, 128, 3), (128, 129, 4)])
def test_streaming_step_equals_whole_signal(device, lib, block, taps, channels):
    """The causal one-block step (the HBM-streaming kernel) produces the same samples as
    the whole-signal call."""
    rng = np.random.default_rng(block * 3 + taps)
    h = (rng.standard_normal(taps) / np.sqrt(taps)).astype(np.float32)
    n_blocks = 40
    length = n_blocks * block
    x = rng.standard_normal((channels, length)).astype(np.float32)
    c = conv(device, block, channels=channels)
    c.setKernel(h)
    from metalaudio_b200 import Tensor
    tin = Tensor(device, (channels, length)); tin.copy(x)
    tout = Tensor(device, (channels, length))
    for t in range(n_blocks):
        st = lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(tin.pointer + 4 * t * block), length,
                                   ctypes.c_void_p(tout.pointer + 4 * t * block), length)
        assert st == 0
    device.synchronize()
    y = tout.toArray()
    for i in range(channels):
        ref = o64.convolve_full(x[i], h)[:length]
        assert o64.rel_rms(y[i], ref) <= TOL
    # whole-signal call after reset agrees on the same samples
    c.reset()
    z = c.process(x)
    assert o64.rel_rms(y, z[:, :length]) <= TOL


@pytest.mark.parametrize("splits", [1, 3, 16, 18, 20, 37, 40])
def test_streaming_step_with_forced_partition_splits(device, lib, splits):
    """ma_pconv_step_splits: the step's multiply-accumulate split into 1, 3, 16, 18, 20, 37 or 40 ranges of
    the 100 partitions gives the same samples.  From 16 splits up, consecutive splits form thread-block
    clusters of 8, 4 or 2 CTAs (16 and 40: eight; 20: four; 18: two; 37: none, and then the partial spectra
    go through their own summing kernel) that add their sums up on chip.  Changing the count between steps
    of a running stream is allowed."""
    from metalaudio_b200 import Tensor
    block, taps, channels, n_blocks = 64, 6400, 8, 30
    rng = np.random.default_rng(splits)
    h = (rng.standard_normal(taps) / np.sqrt(taps)).astype(np.float32)
    length = n_blocks * block
    x = rng.standard_normal((channels, length)).astype(np.float32)
    c = conv(device, block, channels=channels)
    c.setKernel(h)
    got = ctypes.c_int32(0)
    assert lib.ma_pconv_step_splits(c._h, 0, ctypes.byref(got)) == 0 and got.value >= 1
    chosen = got.value
    assert lib.ma_pconv_step_splits(c._h, 101, None) != 0 and lib.ma_pconv_step_splits(c._h, 65, None) != 0
    tin = Tensor(device, (channels, length)); tin.copy(x)
    tout = Tensor(device, (channels, length))
    for t in range(n_blocks):
        if t == 10:   # switch in mid-stream
            assert lib.ma_pconv_step_splits(c._h, splits, ctypes.byref(got)) == 0 and got.value == splits
        if t == 20:
            assert lib.ma_pconv_step_splits(c._h, chosen, None) == 0
        assert lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(tin.pointer + 4 * t * block), length,
                                     ctypes.c_void_p(tout.pointer + 4 * t * block), length) == 0
    device.synchronize()
    y = tout.toArray()
    for i in range(channels):
        assert o64.rel_rms(y[i], o64.convolve_full(x[i], h)[:length]) <= TOL


@pytest.mark.parametrize("block,taps,length", [(128, 1001, 5000), (512, 1025, 4096), (32, 65, 1000), (1024, 4097, 20480)])
def test_whole_signal_writes_only_its_rows(device, lib, block, taps, length):
    """Rows packed at exactly len + taps - 1 samples (an even count: the paired plans' overlap-add):
    the samples behind every row belong to the next channel, those behind the last one to nobody."""
    from metalaudio_b200 import Tensor
    channels = 3
    rng = np.random.default_rng(block)
    h = (rng.standard_normal(taps) / np.sqrt(taps)).astype(np.float32)
    x = rng.standard_normal((channels, length)).astype(np.float32)
    full = length + taps - 1
    c = conv(device, block, channels=channels)
    c.setKernel(h)
    guard = 4 * block
    tin = Tensor(device, x.shape); tin.copy(x)
    tout = Tensor(device, (channels * full + guard,)); tout.copy(np.full(channels * full + guard, 7.0, np.float32))
    assert lib.ma_pconv_reserve(c._h, length) == 0
    assert lib.ma_pconv_process_dev(c._h, ctypes.c_void_p(tin.pointer), length, length, ctypes.c_void_p(tout.pointer), full) == 0
    device.synchronize()
    y = tout.toArray()
    assert np.all(y[channels * full:] == 7.0)
    for i in range(channels):
        assert o64.rel_rms(y[i * full:(i + 1) * full], o64.convolve_full(x[i], h)) <= TOL


@pytest.mark.parametrize("block,taps", [(64, 1023), (64, 1024), (128, 2048), (64, 9001), (256, 33000)])
def test_whole_signal_after_steps_and_back(device, lib, block, taps):
    """Whole-signal calls on a clear delay line run on a coarser partition (from 16 partitions up); a call that
    follows streaming steps continues with their history on the caller's block size, and the calls and
    steps after it start clear again."""
    from metalaudio_b200 import Tensor
    channels, steps, length = 2, 3, 5000
    rng = np.random.default_rng(taps)
    h = (rng.standard_normal(taps) / np.sqrt(taps)).astype(np.float32)
    x = rng.standard_normal((channels, steps * block + length)).astype(np.float32)
    c = conv(device, block, channels=channels)
    c.setKernel(h)
    tail = np.ascontiguousarray(x[:, steps * block:])
    ref = np.stack([o64.convolve_full(tail[i], h) for i in range(channels)])
    tin = Tensor(device, x.shape); tin.copy(x)
    tout = Tensor(device, (channels, block))

    def step(t):
        assert lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(tin.pointer + 4 * t * block), x.shape[1],
                                     ctypes.c_void_p(tout.pointer), block) == 0
        device.synchronize()
        return tout.toArray()

    assert o64.rel_rms(c.process(tail), ref) <= TOL           # clear
    for t in range(steps):
        y = step(t)                                           # the call before left nothing behind
    want = np.stack([o64.convolve_full(x[i, :steps * block], h)[(steps - 1) * block:steps * block] for i in range(channels)])
    assert o64.rel_rms(y, want) <= TOL
    # continues the stream: the block products of the steps' input reach into the call (all but the kept tail)
    z = c.process(tail)
    port = rp.PartitionedConvolution(block)
    for i in range(channels):
        port.set_kernel(h)
        for t in range(steps):
            padded = np.concatenate([x[i, t * block:(t + 1) * block], np.zeros(block, np.float32)])
            port.ring[port.write_index] = np.fft.fft(padded).astype(np.complex64)
            port.write_index = (port.write_index + 1) % port.partitions
        assert o64.rel_rms(z[i], port.process(tail[i])) <= TOL
    assert o64.rel_rms(c.process(tail), ref) <= TOL           # clear again
    y = step(0)
    assert o64.rel_rms(y, np.stack([o64.convolve_full(x[i, :block], h)[:block] for i in range(channels)])) <= TOL


@pytest.mark.parametrize("block,taps,length", [(32, 1, 32), (32, 33, 500), (32, 255, 2049), (32, 511, 1500), (4096, 65536, 5000),
                                               (4096, 65537, 60000), (4096, 135000, 130000), (4096, 262144, 9000),
                                               (4096, 262145, 9000)])
def test_whole_signal_products_at_chunk_and_tile_edges(device, block, taps, length):
    """1 to 65 partitions (64 is the last count whose rows are brought in as boxes), whole and partial chunks of
    16, one to four warps of output blocks per CTA, one response per channel."""
    rng = np.random.default_rng(taps)
    channels = 3
    h = (rng.standard_normal((2, taps)) / np.sqrt(taps)).astype(np.float32)
    x = rng.standard_normal((channels, length)).astype(np.float32)
    c = conv(device, block, channels=channels)
    c.setKernel(h, channelToKernel=[1, 0, 1])
    y = c.process(x)
    for i, ir in enumerate([1, 0, 1]):
        assert o64.rel_rms(y[i], o64.convolve_full(x[i], h[ir])) <= TOL


def test_config3_scaled(device):
    """Configuration 3 at reduced channel count / length: one shared exponentially decaying
    noise IR, block 256, float64 oracle plus exact dot-product spot checks."""
    h = configs.c3_ir(16384)
    x = configs.c3_input(channels=8, length=1 << 15)
    c = conv(device, 256, channels=8)
    c.setKernel(h)
    assert c.partitionCount == 64
    y = c.process(x)
    ref = np.stack([o64.convolve_full(x[i], h) for i in range(8)])
    assert o64.rel_rms(y, ref) <= TOL
    idx = np.random.default_rng(0).integers(0, y.shape[1], 200)
    spot = o64.convolve_spot(x[3], h, idx)
    assert np.sqrt(np.mean((y[3, idx] - spot) ** 2)) / np.sqrt(np.mean(ref[3] ** 2)) <= TOL


def test_config4_scaled(device):
    """Configuration 4 at reduced size: block 64, one IR per channel pair, long partition
    count (accumulation over 512 partitions)."""
    irs = configs.c4_irs(n_irs=4, taps=32768)
    x = configs.c4_input(channels=8, length=1 << 14)
    c = conv(device, 64, channels=8)
    c.setKernel(irs, channelToKernel=[i // 2 for i in range(8)])
    assert c.partitionCount == 512
    y = c.process(x)
    ref = np.stack([o64.convolve_full(x[i], irs[i // 2]) for i in range(8)])
    assert o64.rel_rms(y, ref) <= TOL
    assert o64.max_over_rms(y, ref) <= 1e-4


C4_BLOCK, C4_TAPS = 64, 262144          # configuration 4's own block size and tap count: P = 4096


def _c4_case(channels=4, extra_blocks=256):
    """Input long enough that every one of the 4096 partitions meets a non-zero block spectrum:
    4096 + extra_blocks input blocks per channel, two impulse responses for four channels."""
    irs = configs.c4_irs(n_irs=channels // 2, taps=C4_TAPS)
    x = configs.c4_input(channels=channels, length=(C4_TAPS // C4_BLOCK + extra_blocks) * C4_BLOCK)
    ref = np.stack([o64.convolve_full(x[i], irs[i // 2]) for i in range(channels)])
    return irs, x, ref


def test_config4_true_partition_count_whole_signal(device):
    """Configuration 4's block size and taps (block 64, 262144 taps, one impulse response per channel pair), a
    whole-signal call on a clear delay line: it runs on 64 partitions of 4096 samples.  Against the float64 linear
    convolution and the float32 port of the reference loop, which sums 4096 products per output bin."""
    irs, x, ref = _c4_case()
    c = conv(device, C4_BLOCK, channels=4)
    c.setKernel(irs, channelToKernel=[0, 0, 1, 1])
    assert c.partitionCount == 4096
    y = c.process(x)
    assert y.shape == ref.shape
    assert o64.rel_rms(y, ref) <= TOL
    assert o64.max_over_rms(y, ref) <= 5e-5
    # the steady-state part alone (all 4096 partitions active), where the sums are longest
    lo = C4_TAPS
    assert o64.rel_rms(y[:, lo:lo + 16384], ref[:, lo:lo + 16384]) <= TOL
    # the reference's own float32 block loop on one channel's first 32 blocks past the ramp-up
    port = rp.PartitionedConvolution(C4_BLOCK)
    port.set_kernel(irs[0])
    short = x[0, :(4096 + 32) * C4_BLOCK]
    yp = port.process(short)
    ys = c.process(np.stack([short] * 4))[0]
    assert o64.rel_rms(ys, yp) <= TOL


@pytest.mark.parametrize("partitions", [2047, 2048, 4096])
def test_whole_signal_sums_of_thousands_of_partitions(device, lib, partitions):
    """Whole-signal calls that continue a stream keep the caller's partition: up to 4096 products of block 64 per output
    bin, from 2048 partitions up as sums of at most 256 that are added up in a second level.  Inputs reach past the
    ramp-up, so that every partition meets a non-zero spectrum."""
    taps = partitions * C4_BLOCK - 5
    irs = configs.c4_irs(n_irs=2, taps=taps)
    x = configs.c4_input(channels=2, length=(partitions + 130) * C4_BLOCK + 13)
    ref = np.stack([o64.convolve_full(x[i], irs[i]) for i in range(2)])
    c = conv(device, C4_BLOCK, channels=2)
    c.setKernel(irs, channelToKernel=[0, 1])
    assert c.partitionCount == partitions
    zero_step(lib, device, c, C4_BLOCK, 2)
    y = c.process(x)
    # float32 sums of n terms err by about 2^-24 sqrt(n): 256 terms 9.5e-7, 2047 terms 2.7e-6
    bound = 1e-6 if partitions >= 2048 else 2.7e-6
    assert o64.rel_rms(y, ref) <= bound
    lo, hi = taps, x.shape[1]
    assert o64.rel_rms(y[:, lo:hi], ref[:, lo:hi]) <= bound
    print("partitions", partitions, o64.rel_rms(y, ref), o64.rel_rms(y[:, lo:hi], ref[:, lo:hi]), o64.max_over_rms(y, ref))


def test_config4_true_partition_count_streaming(device, lib):
    """The same case through the causal streaming step (every step reads all 4096 delay-line
    spectra of every channel): 4352 steps, compared with the float64 linear convolution."""
    from metalaudio_b200 import Tensor
    irs, x, ref = _c4_case()
    channels, length = x.shape
    c = conv(device, C4_BLOCK, channels=channels)
    c.setKernel(irs, channelToKernel=[0, 0, 1, 1])
    tin = Tensor(device, (channels, length)); tin.copy(x)
    tout = Tensor(device, (channels, length))
    for t in range(length // C4_BLOCK):
        st = lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(tin.pointer + 4 * t * C4_BLOCK), length,
                                   ctypes.c_void_p(tout.pointer + 4 * t * C4_BLOCK), length)
        assert st == 0
    device.synchronize(60)
    y = tout.toArray()
    assert o64.rel_rms(y, ref[:, :length]) <= TOL
    assert o64.max_over_rms(y, ref[:, :length]) <= 5e-5
    assert o64.rel_rms(y[:, C4_TAPS:], ref[:, C4_TAPS:length]) <= TOL


def test_step_after_other_library_work_reads_fresh_input(device, lib):
    """A streaming step whose input block was produced by another kernel of the library queued
    just before it (here a biquad) must see that kernel's output: the step's first kernel is only
    allowed to start early when it directly follows the previous step."""
    from metalaudio_b200 import Tensor
    block, taps, channels, steps = 64, 300, 4, 24
    rng = np.random.default_rng(77)
    h = (rng.standard_normal(taps) / np.sqrt(taps)).astype(np.float32)
    x = rng.standard_normal((channels, steps * block)).astype(np.float32)
    c = conv(device, block, channels=channels)
    c.setKernel(h)
    bq = ctypes.c_void_p()
    assert lib.ma_biquad_create(device.handle, channels, 1, ctypes.byref(bq)) == 0
    gain = np.array([[0.5, 0.0, 0.0, 0.0, 0.0]], np.float32)    # y = 0.5 x, no memory
    assert lib.ma_biquad_set_coefficients(bq, gain.ctypes.data_as(ctypes.c_void_p), 1, None) == 0
    tin = Tensor(device, x.shape); tin.copy(x)
    mid = Tensor(device, (channels, block))
    tout = Tensor(device, x.shape)
    n = steps * block
    for t in range(steps):
        assert lib.ma_biquad_process_dev(bq, ctypes.c_void_p(tin.pointer + 4 * t * block), n,
                                         ctypes.c_void_p(mid.pointer), block, block) == 0
        assert lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(mid.pointer), block,
                                     ctypes.c_void_p(tout.pointer + 4 * t * block), n) == 0
    device.synchronize()
    y = tout.toArray()
    lib.ma_biquad_destroy(bq)
    for i in range(channels):
        assert o64.rel_rms(y[i], 0.5 * o64.convolve_full(x[i], h)[:n]) <= TOL


def zero_step(lib, device, c, block, channels=1):
    """One streaming step of silence: the delay line stays zero but no longer counts as clear, so the next
    whole-signal call runs on the caller's own block size."""
    from metalaudio_b200 import Tensor
    t = Tensor(device, (channels, block))
    t.copy(np.zeros((channels, block), np.float32))
    assert lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(t.pointer), block, ctypes.c_void_p(t.pointer), block) == 0
    device.synchronize()


@pytest.mark.parametrize("site", ["spectra", "buffers", "both"])
def test_reserve_without_memory_for_the_coarse_partition(lib, device, site):
    """ma_pconv_reserve when the coarser partition's spectra, or the signals' buffers beside them, cannot be had:
    the call succeeds and whole-signal calls run on the caller's block size, with the results of that size.  When the
    buffers fail on that size too the call reports it, and the next one starts afresh."""
    from metalaudio_b200 import _lib as L
    block, taps, length, channels = 64, 3000, 9000, 3
    rng = np.random.default_rng(31)
    h = (rng.standard_normal((channels, taps)) * np.exp(-np.arange(taps) / 500.0)).astype(np.float32)
    x = rng.standard_normal((channels, length)).astype(np.float32)

    def fresh():
        c = conv(device, block, channels=channels)
        c.setKernel(h, channelToKernel=list(range(channels)))
        return c
    own = fresh()
    zero_step(lib, device, own, block, channels)
    ref_own = own.process(x)
    ref_coarse = fresh().process(x)
    assert not np.array_equal(ref_own, ref_coarse)
    c = fresh()
    assert lib.ma_pconv_reserve(c._h, length) == 0   # a first reservation has the coarse spectra ...
    if site == "spectra":
        c = fresh()
        assert lib.ma_test_inject_fault(device.handle, L.FAULT_RESERVE_SPECTRA, 2) == 0   # cudaErrorMemoryAllocation
        assert lib.ma_pconv_reserve(c._h, length) == 0
        assert np.array_equal(c.process(x), ref_own)
    elif site == "buffers":
        for c in (c, fresh()):                        # ... and gives them back where a longer one does not fit beside them
            assert lib.ma_test_inject_fault(device.handle, L.FAULT_RESERVE_BUFFERS, 2) == 0
            assert lib.ma_pconv_reserve(c._h, 2 * length) == 0
            assert np.array_equal(c.process(x), ref_own)
    else:
        c = fresh()
        assert lib.ma_test_inject_fault(device.handle, L.FAULT_RESERVE_BUFFERS, 1) == 0   # not a matter of memory
        assert lib.ma_pconv_reserve(c._h, length) == L.MA_ERR_CUDA
        assert np.array_equal(c.process(x), ref_coarse)
    for i in range(channels):
        assert o64.rel_rms(c.process(x)[i], o64.convolve_full(x[i], h[i])) <= TOL
    # new taps: the coarse partition again
    c.setKernel(h, channelToKernel=list(range(channels)))
    assert np.array_equal(c.process(x), ref_coarse)


def test_taps_take_no_device_memory_before_a_reservation(lib, device):
    """A convolver that only streams holds its spectra, its delay line and nothing else on the device: not the taps,
    which only ma_pconv_reserve lays out a second time."""
    import torch
    block, taps, irs = 64, 65536, 256
    h = np.random.default_rng(5).standard_normal((irs, taps)).astype(np.float32)
    c = conv(device, block, channels=irs)
    c.setKernel(h[:, :64], channelToKernel=list(range(irs)))   # creates the plan and the object
    free0 = torch.cuda.mem_get_info()[0]
    c.setKernel(h, channelToKernel=list(range(irs)))           # the temporary copy of the taps joins the pool
    c.setKernel(h[:, :64], channelToKernel=list(range(irs)))
    pool = free0 - torch.cuda.mem_get_info()[0]
    c.setKernel(h, channelToKernel=list(range(irs)))
    held = free0 - torch.cuda.mem_get_info()[0] - pool
    need = 2 * 8 * irs * taps                                  # spectra and delay line
    assert held <= need + (40 << 20)                           # the taps would be 64 MiB more


@pytest.mark.parametrize("block,taps,length,where", [
    (64, 3000, 9000, [(0, 4000)]), (64, 3000, 9000, [(0, 0)]), (64, 3000, 9000, [(1, 8999)]), (64, 3000, 9000, [(0, 255), (0, 256)]),
    (32, 70000, 150001, [(0, 5), (0, 100000), (2, 149999)]), (256, 4096, 20000, [(1, 3), (1, 10001), (2, 511)]),
    (1, 40, 3000, [(0, 100), (0, 1700)]), (2, 333, 5000, [(2, 2048)]), (128, 9000, 4097, [(0, 4096)]), (512, 40000, 70000, [(1, 33333)])])
def test_non_finite_samples_spoil_the_callers_blocks_only(lib, device, block, taps, length, where):
    """A NaN or infinity in the input of a call on the coarse partition: lost are exactly the outputs that the caller's
    own block size loses, the others are the convolution's.  Also in place and through the host form."""
    from metalaudio_b200 import Tensor
    channels, full = 3, length + taps - 1
    rng = np.random.default_rng(block + taps)
    h = (rng.standard_normal((2, taps)) * np.exp(-np.arange(taps) / max(8, taps / 6))).astype(np.float32)
    cmap = [0, 1, 1]
    x = rng.standard_normal((channels, length)).astype(np.float32)
    clean = x.copy()
    for k, (c, at) in enumerate(where):
        x[c, at] = (np.nan, np.inf, -np.inf)[k % 3]
        clean[c, at] = 0.0
    finite = np.ones((channels, full), bool)
    for c, at in where:                      # block i of the output: input blocks i - P .. i
        first = at // block * block
        finite[c, first:first + (-(-taps // block) + 1) * block] = False
    c = conv(device, block, channels=channels)
    c.setKernel(h, channelToKernel=cmap)
    zero_step(lib, device, c, block, channels)
    assert np.array_equal(np.isfinite(c.process(x)), finite)      # the caller's block size
    ref = np.stack([o64.convolve_full(clean[i], h[cmap[i]]) for i in range(channels)])

    def check(y):
        assert np.array_equal(np.isfinite(y), finite)
        for i in range(channels):
            assert o64.rel_rms(y[i][finite[i]], ref[i][finite[i]]) <= TOL
    check(c.process(x))
    buf = Tensor(device, (channels, full))
    buf.copy(np.pad(x, ((0, 0), (0, taps - 1))))
    assert lib.ma_pconv_process_dev(c._h, ctypes.c_void_p(buf.pointer), length, full, ctypes.c_void_p(buf.pointer), full) == 0
    device.synchronize(30)
    check(buf.toArray())
    y = c.process(clean)                       # nothing is left behind
    assert all(o64.rel_rms(y[i], ref[i]) <= TOL for i in range(channels))


class Recorded:
    """Calls on the library's stream recorded into a CUDA graph."""

    def __init__(self, lib, device, calls):
        import torch
        self.stream = torch.cuda.ExternalStream(lib.ma_context_stream(device.handle))
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(self.stream):
            self.graph.capture_begin(capture_error_mode="relaxed")
            try:
                calls()
            finally:
                self.graph.capture_end()

    def replay(self):
        import torch
        with torch.cuda.stream(self.stream):
            self.graph.replay()


def test_recorded_whole_signal_calls_and_streaming_between_them(lib, device):
    """Whole-signal calls recorded into a graph, on a clear delay line: neither the recording (nothing runs then) nor
    calls that continue a stream, before or between replays, leave rows behind that the next call takes for the zeros
    in front of the signal."""
    from metalaudio_b200 import Tensor
    block, taps, length, channels = 64, 3000, 9000, 2
    full = length + taps - 1
    rng = np.random.default_rng(51)
    h = (rng.standard_normal(taps) * np.exp(-np.arange(taps) / 500.0)).astype(np.float32)
    x = rng.standard_normal((channels, length)).astype(np.float32)
    ref = np.stack([o64.convolve_full(x[i], h) for i in range(channels)])
    c = conv(device, block, channels=channels)
    c.setKernel(h)
    tin, out, blk = Tensor(device, x.shape), Tensor(device, (channels, full)), Tensor(device, (channels, block))
    tin.copy(x)
    blk.copy(np.full((channels, block), 50.0, np.float32))
    assert lib.ma_pconv_reserve(c._h, length) == 0

    def whole():
        assert lib.ma_pconv_process_dev(c._h, ctypes.c_void_p(tin.pointer), length, length, ctypes.c_void_p(out.pointer), full) == 0

    def stream():   # fills the delay line, and the buffer by the caller's block size; clear afterwards
        for _ in range(3):
            assert lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(blk.pointer), block, ctypes.c_void_p(out.pointer), full) == 0
        whole()

    def check(call):
        out.zero()
        call()
        device.synchronize()
        y = out.toArray()
        assert all(o64.rel_rms(y[i], ref[i]) <= TOL for i in range(channels))
    check(whole)
    stream()
    g = Recorded(lib, device, whole)
    check(whole)
    check(g.replay)
    stream()
    check(g.replay)
    check(whole)
    check(g.replay)


def test_recorded_steps_fill_the_delay_line(lib, device):
    """A graph of one turn of the delay line (as many steps as partitions): after its replay a whole-signal call
    continues that stream, as after the same steps called directly, also when the object was reset in between."""
    from metalaudio_b200 import Tensor
    block, taps, length = 64, 1500, 4000
    parts, full = -(-taps // block), length + taps - 1
    rng = np.random.default_rng(52)
    h = (rng.standard_normal(taps) * np.exp(-np.arange(taps) / 300.0)).astype(np.float32)
    past = rng.standard_normal((1, parts * block)).astype(np.float32)
    x = rng.standard_normal((1, length)).astype(np.float32)
    tin, tpast, out, blk = Tensor(device, x.shape), Tensor(device, past.shape), Tensor(device, (1, full)), Tensor(device, past.shape)
    tin.copy(x)
    tpast.copy(past)
    results = []
    for recorded in (False, True):
        c = conv(device, block)
        c.setKernel(h)
        assert lib.ma_pconv_reserve(c._h, length) == 0

        def steps():
            for b in range(parts):
                assert lib.ma_pconv_step_dev(c._h, ctypes.c_void_p(tpast.pointer + 4 * b * block), past.shape[1],
                                             ctypes.c_void_p(blk.pointer + 4 * b * block), past.shape[1]) == 0
        steps()
        assert lib.ma_pconv_reset(c._h) == 0
        if recorded:
            g = Recorded(lib, device, steps)
            assert lib.ma_pconv_reset(c._h) == 0
            g.replay()
        else:
            steps()
        assert lib.ma_pconv_process_dev(c._h, ctypes.c_void_p(tin.pointer), length, length, ctypes.c_void_p(out.pointer), full) == 0
        device.synchronize()
        results.append((blk.toArray(), out.toArray()))
    assert np.array_equal(results[0][0], results[1][0])
    assert np.array_equal(results[0][1], results[1][1])
    alone = o64.convolve_full(x[0], h)
    assert o64.rel_rms(results[0][1][0], alone) > 0.05   # the stream before it is heard


def test_errors(device):
    from metalaudio_b200 import Convolution, ConvolutionError, MetalAudioError
    c = conv(device, 64)
    with pytest.raises(ConvolutionError) as e:
        c.setKernel(np.zeros(0, np.float32))
    assert e.value.case == "emptyKernel"
    with pytest.raises(ConvolutionError):
        c.process(np.ones(10, np.float32))
    assert c.process(np.zeros(0, np.float32)).size == 0
    with pytest.raises(MetalAudioError):
        Convolution(device, Convolution.Mode.partitioned(blockSize=0)).setKernel(np.ones(4, np.float32))
