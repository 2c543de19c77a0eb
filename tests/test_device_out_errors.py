"""A product call that fails leaves the caller's device buffer as it was, also
where the product is formed in that buffer, and the handle goes on working."""
import numpy as np
import pytest

from sentinel1_decode_gb300 import S1Decoder, synth

BAD_BRC = -9


def streams(swath, shapes):
    """A good stream and the same with a bit-rate code of 7 in the middle of the last burst."""
    sweep = 820 if swath == "IW2" else 0
    good = synth.generate(synth.StreamSpec(
        [synth.BurstSpec(num_lines=n, num_quads=q, swath=swath, beam_start=100 if sweep else 512, beam_sweep=sweep,
                         gap_lines=200, num_targets=4) for n, q in shapes], seed=9,
        radar=synth.RadarParams(pulse_length_us=5.0)))
    d = S1Decoder(good)
    at = d.packet_offset(d.num_packets() - shapes[-1][0] // 2) + 68
    d.close()
    bad = bytearray(good)
    bad[at] |= 0xE0
    return good, bytes(bad)


@pytest.mark.gpu
@pytest.mark.parametrize("swath,shapes,level", [
    ("S1", [(300, 511)], 0), ("S1", [(300, 511)], 1), ("S1", [(257, 1000)], 2), ("S1", [(257, 1000)], 3),
    ("IW2", [(301, 400)], 1), ("IW2", [(301, 400)], 3), ("IW2", [(1000, 96), (1003, 101)], 3)])
def test_failed_decode_leaves_the_buffer(lib_path, swath, shapes, level):
    torch = pytest.importorskip("torch")
    good, bad = streams(swath, shapes)
    d = S1Decoder(bad, precision="fp32")
    lib, burst = d._lib, len(shapes) - 1
    if swath == "S1" and level == 3:
        rows, cols = d.burst_shape(swath, 0, 1)
        call = lambda p: lib.s1g_swath_product(d.handle, b"S1", 3, p, rows, cols, 0, 1)  # noqa: E731
    else:
        rows, cols = d.burst_shape(swath, burst, level)
        call = lambda p: lib.s1g_burst_product(d.handle, swath.encode(), burst, level, p, rows, cols, 0, 1)  # noqa: E731
    buf = torch.full((rows, cols), 7.0 + 0j, dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        assert call(buf.data_ptr()) == BAD_BRC
        assert bool((buf == 7.0).all())
    d.reload(good)
    assert call(buf.data_ptr()) == 0
    fresh = S1Decoder(good, precision="fp32")
    if swath == "S1" and level == 3:
        want = fresh.get_azimuth_compressed_swath(swath, dtype=np.complex64)
    else:
        want = fresh._burst(swath, burst, level, np.complex64)
    np.testing.assert_array_equal(buf.cpu().numpy(), want)
    d.close()
    fresh.close()


@pytest.mark.gpu
def test_burst_of_two_formats(lib_path):
    """Bypass packets and one FDBAQ packet (of zero bits) among them: both
    decoders write the burst's status words, a good burst is delivered and a
    bad one is not."""
    torch = pytest.importorskip("torch")
    data = bytearray(synth.generate(synth.StreamSpec(
        [synth.BurstSpec(num_lines=300, num_quads=200, swath="S1", beam_start=512, beam_sweep=0, num_targets=4, baq_mode=0)],
        seed=9, radar=synth.RadarParams(pulse_length_us=5.0))))
    d = S1Decoder(bytes(data), precision="fp32")
    a, b = d.packet_offset(150), d.packet_offset(151)
    data[a + 37] = data[a + 37] & 0xE0 | 12
    data[a + 68:b] = bytes(b - a - 68)
    d.reload(bytes(data))
    want = d.get_range_compressed_burst("S1", 0, dtype=np.complex64)
    rows, cols = want.shape
    buf = torch.full((rows, cols), 7.0 + 0j, dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    call = lambda: d._lib.s1g_burst_product(d.handle, b"S1", 0, 1, buf.data_ptr(), rows, cols, 0, 1)  # noqa: E731
    good = bytes(data)
    data[a + 68] |= 0xE0
    d.reload(bytes(data))
    assert call() == BAD_BRC
    assert bool((buf == 7.0).all())
    d.reload(good)
    assert call() == 0
    np.testing.assert_array_equal(buf.cpu().numpy(), want)
    d.close()
