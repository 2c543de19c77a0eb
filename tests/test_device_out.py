"""Products written straight into the caller's device buffer (where the shape,
type and alignment allow it) equal those delivered to host memory; a buffer of
another shape is refused and keeps its contents."""
import numpy as np
import pytest

from sentinel1_decode_gb300 import S1Decoder, synth

LEVELS = {"range_compressed": 1, "range_doppler": 2, "azimuth": 3}


@pytest.mark.gpu
@pytest.mark.parametrize("level", sorted(LEVELS))
@pytest.mark.parametrize("swath,lines,quads", [("S1", 300, 511), ("S1", 257, 1000), ("IW2", 301, 400)])
@pytest.mark.parametrize("offset", [0, 1])
def test_device_buffer_equals_host_buffer(lib_path, level, swath, lines, quads, offset):
    torch = pytest.importorskip("torch")
    sweep = 820 if swath == "IW2" else 0
    data = synth.generate(synth.StreamSpec(
        [synth.BurstSpec(num_lines=lines, num_quads=quads, swath=swath, beam_start=100 if sweep else 512,
                         beam_sweep=sweep, num_targets=4)], seed=9, radar=synth.RadarParams(pulse_length_us=5.0)))
    d = S1Decoder(data, precision="fp32")
    lv = LEVELS[level]
    if lv == 3:
        host = d.get_azimuth_compressed_burst(swath, 0, dtype=np.complex64) if sweep else \
            d.get_azimuth_compressed_swath(swath, dtype=np.complex64)
    else:
        host = d.get_range_compressed_burst(swath, 0, range_doppler=lv == 2, dtype=np.complex64)
    rows, cols = host.shape
    buf = torch.full((rows * cols + 2,), 7.0 + 0j, dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    lib, name = d._lib, swath.encode()
    call = (lambda r: lib.s1g_swath_product(d.handle, name, lv, buf.data_ptr() + 8 * offset, r, cols, 0, 1)) \
        if lv == 3 and not sweep else \
        (lambda r: lib.s1g_burst_product(d.handle, name, 0, lv, buf.data_ptr() + 8 * offset, r, cols, 0, 1))
    assert call(rows + 1) != 0
    assert bool((buf == 7.0).all())
    assert call(rows) == 0
    got = buf.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + rows * cols].reshape(rows, cols), host)
    assert (got[:offset] == 7.0).all() and (got[offset + rows * cols:] == 7.0).all()
    d.close()
