"""The shared-memory FFT core and the kernels over it, at the lengths where
their plans change: row transforms (affine and other 7-smooth lengths, primes,
lengths over one CTA's shared memory that split and that do not), the Doppler
estimator's blocks (each radix, two to four passes, one or more blocks per
line) with odd burst sizes through the time unfolding, and the FP32 phases of
the differentiable chain."""
import numpy as np
import pytest

from conftest import rel_l2
from sentinel1_decode_gb300 import S1Decoder, synth


def burst(lines, quads, swath="IW2", pulse=None, seed=5, targets=6):
    rp = synth.RadarParams() if pulse is None else synth.RadarParams(pulse_length_us=pulse)
    sweep = 820 if swath.startswith("IW") else 0
    return synth.generate(synth.StreamSpec(
        [synth.BurstSpec(num_lines=lines, num_quads=quads, swath=swath, beam_start=100 if sweep else 512,
                         beam_sweep=sweep, num_targets=targets)], seed=seed, radar=rp))


# Tolerances: a transform's relative L2 error is near eps sqrt(log2 n), three
# of them in a chirp-z one; 1e-13 and 2e-6 leave an order above that.
@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-13), ("fp32", 2e-6), ("fp32_plain", 2e-6)])
@pytest.mark.parametrize("lines", [2, 7, 96, 487, 1500, 14009, 14010, 28672])
def test_row_transforms(lib_path, prec, tol, lines):
    data = burst(lines, 9, "S1", pulse=0.2, targets=0)
    d = S1Decoder(data, precision=prec)
    rc = d.get_range_compressed_burst("S1", 0)
    rd = d.get_range_compressed_burst("S1", 0, range_doppler=True)
    d.close()
    assert rel_l2(rd, np.fft.fftshift(np.fft.fft(rc, axis=0), axes=0)) < tol


# FP32 against FP64: the SLC moves by 7e-5 per 1e-5 Hz of centroid, so a wrong
# estimate shows; 1e-4 is the bound of the FP32 SLCs.
@pytest.mark.gpu
@pytest.mark.parametrize("lines,quads,pulse", [(149, 100, 1.0), (257, 151, 3.0), (150, 400, 5.0), (201, 333, 10.0),
                                               (311, 1500, 62.0), (330, 3001, 40.0), (277, 2500, 100.0)])
def test_slc_at_odd_sizes(lib_path, lines, quads, pulse):
    data = burst(lines, quads, pulse=pulse)
    out = []
    for prec in ("fp64", "fp32"):
        d = S1Decoder(data, precision=prec)
        out.append(d.get_azimuth_compressed_burst("IW2", 0))
        d.close()
    assert rel_l2(out[1], out[0]) < 1e-4


# The FP32 chain's rounding is 2e-7 per transform of a unit-norm image; the
# entropy's derivative with respect to the polynomial does not cancel.
@pytest.mark.gpu
@pytest.mark.parametrize("lines,quads", [(131, 65), (144, 512), (257, 1031)])
def test_chain_phases(lib_path, lines, quads):
    data = burst(lines, quads, "S1", pulse=2.0)
    res = []
    for prec in ("fp64", "fp32"):
        d = S1Decoder(data, precision=prec)
        res.append(d.azimuth_adjoint("S1", 0, [3.0, -2.0], 5.0))
        d.close()
    (l64, t64, _), (l32, t32, _) = res
    assert abs(l32 - l64) < 1e-5 * abs(l64)
    assert np.linalg.norm(np.asarray(t32) - np.asarray(t64)) < 1e-4 * np.linalg.norm(t64)


def knot_of_near(u, S, TS):
    """The interval and the step from its first sample, as the time unfolding
    forms them: float32 estimates, products that wrap in 32 bits."""
    q = np.trunc(u.astype(np.float32) * np.float32((S - 1) / (TS - 1))).astype(np.int64)
    num = (u * (S - 1) - q * (TS - 1)).astype(np.uint32).astype(np.int32).astype(np.int64)
    low, high = num < 0, num >= TS - 1
    q = q - low + high
    num = num + (TS - 1) * low - (TS - 1) * high
    end = q > S - 2
    q = np.where(end, S - 2, q)
    num = np.where(end, num + TS - 1, num)
    return q, np.trunc((num.astype(np.float32) + np.float32(0.5)) * np.float32(1.0 / (S - 1))).astype(np.int64)


@pytest.mark.parametrize("S,T", [(61, 2), (1201, 9), (6908, 6), (13801, 3), (1048575, 16)])
def test_interval_and_step_in_32_bits(S, T):
    TS = S * T
    u = np.arange(TS, dtype=np.int64) if TS < 1 << 20 else np.unique(
        np.concatenate([np.random.default_rng(1).integers(0, TS, 200000), [0, 1, TS - 2, TS - 1]]))
    q, d = knot_of_near(u, S, TS)
    want = np.minimum(u * (S - 1) // (TS - 1), S - 2)
    np.testing.assert_array_equal(q, want)
    np.testing.assert_array_equal(d, u + (-want * (TS - 1) // (S - 1)))


# FP64 products do not depend on whether the unfolding's transforms run over
# the band alone: the oracle's transforms are whole ones.  1e-8 is the bound of
# the FP64 products.
@pytest.mark.gpu
@pytest.mark.parametrize("lines,quads", [(601, 300), (640, 257), (433, 500), (1000, 200)])
def test_fp64_band_transforms_vs_oracle(lib_path, lines, quads):
    import s1_oracle as O
    data = burst(lines, quads, pulse=5.0, seed=11)
    ref = O.S1Decoder(data).get_azimuth_compressed_burst("IW2", 0)
    d = S1Decoder(data, precision="fp64")
    out = d.get_azimuth_compressed_burst("IW2", 0)
    d.close()
    assert rel_l2(out, ref) < 1e-8
