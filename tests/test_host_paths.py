"""The library's host code on a CUDA runtime without a GPU (fake_cudart): what
it launches, keeps, replays and orders, watched from outside.  Kernels do
nothing there, so nothing here looks at samples."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, %r)
from sentinel1_decode_gb300 import S1Decoder, S1GError, load_library, process_swath_batch, synth
rt = ctypes.CDLL("libcudart.so.13")
rt.fake_count.restype = ctypes.c_longlong
rt.fake_last_unordered.restype = ctypes.c_char_p

def count(what):
    return rt.fake_count(what.encode())

def bursts(*shapes, seed=1, swath="IW2", **kw):
    return [synth.BurstSpec(num_lines=n, num_quads=q, swath=swath, num_targets=1, gap_lines=200, **kw) for n, q in shapes]

def stream(*specs, seed=1):
    return synth.generate(synth.StreamSpec(list(specs), seed=seed))
""" % ROOT


@pytest.fixture(scope="module")
def fake(lib_path, tmp_path_factory):
    """Runs a script in a child process on the fake runtime."""
    from sentinel1_decode_gb300.build import nvcc
    out = tmp_path_factory.mktemp("fake_cudart")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    src = os.path.join(HERE, "fake_cudart")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", include,
                    os.path.join(src, "fake_cudart.cpp"), "-o", str(out / "libcudart.so.13"),
                    "-Wl,-soname,libcudart.so.13,--version-script=" + os.path.join(src, "libcudart.map")], check=True)
    # freed memory stays mapped and is overwritten, so that a late reader shows
    env = dict(os.environ, LD_LIBRARY_PATH=str(out), S1G_AUTOTUNE="0", S1G_FFT_TUNE_FILE=str(out / "tune.txt"),
               MALLOC_PERTURB_="165", MALLOC_MMAP_THRESHOLD_=str(1 << 40), MALLOC_TRIM_THRESHOLD_=str(1 << 40))

    def run(script):
        r = subprocess.run([sys.executable, "-c", PRELUDE + script], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_reload_of_the_same_layout_decodes_again(fake):
    """Headers and packet lengths alike, other user data: samples of the stream
    before must not be served."""
    fake("""
data = bytearray(stream(*bursts((1000, 24), (1003, 24))))
d = S1Decoder(bytes(data))
d.get_range_compressed_burst("IW2", 0)
once = count("launch:k_decode_fdbaq")
d.get_range_compressed_burst("IW2", 1)
assert count("launch:k_decode_fdbaq") == once          # the swath was decoded as a whole
data[-1] ^= 0x10
d.reload(bytes(data))
d.get_range_compressed_burst("IW2", 0)
assert count("launch:k_decode_fdbaq") == once + 1
d.get_range_compressed_burst("IW2", 1)
assert count("launch:k_decode_fdbaq") == once + 1
""")


@pytest.mark.gpu
def test_reload_of_the_same_layout_gives_its_own_samples(lib_path):
    """The same with the samples: in every packet the sign of the first IE sample
    (the bit after its block's rate code) turned round."""
    import numpy as np
    from sentinel1_decode_gb300 import S1Decoder, synth
    data = synth.generate(synth.StreamSpec(
        [synth.BurstSpec(num_lines=n, num_quads=40, swath="IW2", num_targets=1, gap_lines=200) for n in (1000, 1003)],
        seed=3))
    d = S1Decoder(data)
    other = bytearray(data)
    for p in range(d.num_packets()):
        other[d.packet_offset(p) + 68] ^= 0x10
    before = d.get_burst("IW2", 1, dtype=np.complex64)
    d.reload(bytes(other))
    fresh = S1Decoder(bytes(other))
    for b in range(2):
        got = d.get_burst("IW2", b, dtype=np.complex64)
        np.testing.assert_array_equal(got, fresh.get_burst("IW2", b, dtype=np.complex64))
    assert not np.array_equal(got, before)
    d.close()
    fresh.close()


GROWTH = """
data = stream(*bursts((1000, 24), (1003, 24)), *bursts((1000, 40), (1001, 44), swath="IW3"))
d = S1Decoder(data)
for _ in range(3):                                      # eager, capture, replay
    process_swath_batch([d], "IW2")
assert (count("capture"), count("replay")) == (1, 2)
"""


@pytest.mark.parametrize("grow", [
    'process_swath_batch([d], "IW3")',                                     # longer lines, same handle
    'd.get_range_compressed_burst("IW3", 1)',                              # a per-burst call
    'd.set_precision("fp64"); d.get_range_compressed_burst("IW3", 1); d.set_precision("fp32")',
])
def test_no_replay_over_buffers_that_moved(fake, grow):
    """A captured batch holds the addresses of the handle's buffers: once one of
    them has been replaced by a larger one, the batch is run and captured anew."""
    fake(GROWTH + grow + """
captured, replayed = count("capture"), count("replay")
process_swath_batch([d], "IW2")
assert (count("capture"), count("replay")) == (captured, replayed)      # eager
process_swath_batch([d], "IW2")
process_swath_batch([d], "IW2")
assert (count("capture"), count("replay")) == (captured + 1, replayed + 2)
""")


def test_no_replay_for_another_handle_at_the_same_address(fake):
    """The key of a captured batch tells handles apart by more than their address."""
    fake("""
data = stream(*bursts((1000, 24)))
a = S1Decoder(data)
for _ in range(40):
    b = S1Decoder(data)
    for _ in range(2):
        process_swath_batch([a, b], "IW2")
    at = b.handle.value
    b.close()
    c = S1Decoder(data)
    if c.handle.value == at:
        break
    c.close()
else:
    sys.exit("no handle at the same address")
captured, replayed = count("capture"), count("replay")
process_swath_batch([a, c], "IW2")
assert (count("capture"), count("replay")) == (captured, replayed)
""")


def test_replay_goes_on_while_nothing_moves(fake):
    """Smaller products in between and reloads of the same bytes cost no capture."""
    fake("""
data = stream(*bursts((1000, 24), (1003, 24)))
d = S1Decoder(data)
for _ in range(2):
    process_swath_batch([d], "IW2")
d.get_range_compressed_burst("IW2", 0)
d.get_burst("IW2", 0)
d.reload(data)
for _ in range(3):
    process_swath_batch([d], "IW2")
assert (count("capture"), count("replay")) == (1, 4), (count("capture"), count("replay"))
""")


@pytest.mark.gpu
def test_batch_after_growth_equals_a_fresh_handle(lib_path):
    """Batches of two swaths in turn, the second of longer lines, and per-burst
    products in between: every SLC is a fresh handle's."""
    import numpy as np
    from sentinel1_decode_gb300 import S1Decoder, batch_outputs, process_swath_batch, synth
    from test_batch import fetch
    spec = [synth.BurstSpec(num_lines=n, num_quads=q, swath=sw, num_targets=2, gap_lines=200)
            for sw, n, q in (("IW2", 1000, 96), ("IW2", 1003, 96), ("IW3", 1010, 130), ("IW3", 1031, 136))]
    data = synth.generate(synth.StreamSpec(spec, seed=4))
    want = {}
    for sw in ("IW2", "IW3"):
        f = S1Decoder(data, precision="fp32")
        want[sw] = [f.get_azimuth_compressed_burst(sw, b, dtype=np.complex64) for b in range(2)]
        f.close()
    d = S1Decoder(data, precision="fp32")
    for sw in ("IW2", "IW2", "IW2", "IW3", "IW2", "IW2", "product", "IW2", "IW3", "IW3", "IW2", "IW2"):
        if sw == "product":
            d.set_precision("fp64")
            d.get_range_compressed_burst("IW3", 1)
            d.set_precision("fp32")
            continue
        process_swath_batch([d], sw)
        for got, ref in zip([fetch(*o) for o in batch_outputs(d)], want[sw]):
            np.testing.assert_array_equal(got, ref)
    d.close()


def test_kernels_get_their_shared_memory_on_every_device(fake):
    """The limit of dynamic shared memory belongs to a kernel and a device: one
    process with handles on two of them."""
    fake("""
data = stream(*bursts((300, 1000)))
for device in (0, 1):
    for precision in ("fp32", "fp32_plain", "fp64"):
        d = S1Decoder(data, device=device, precision=precision)
        d.apply_eccm(1000, 10)
        if precision == "fp32":
            d.get_azimuth_compressed_burst("IW2", 0, dtype=np.complex64)
        d.get_range_compressed_burst("IW2", 0, range_doppler=True, dtype=np.complex64)
        d.close()
    assert count("refused") == 0, device
assert count("launch:k_rc_dc") and count("launch:k_transpose_tma") and count("launch:k_eccm_notch")
""")


ORDER = {
    "products": """
for precision in ("fp32", "fp32_plain", "fp64"):
    d = S1Decoder(stream(*bursts((1000, 31), (1003, 31))), precision=precision)
    for eccm in (False, True):
        d.get_range_compressed_burst("IW2", 0, range_doppler=True, dtype=np.complex64)
        if precision == "fp32":
            d.get_azimuth_compressed_burst("IW2", 1, dtype=np.complex64)
        d.apply_eccm(1000, 10)
    if precision == "fp32":
        for _ in range(2):
            process_swath_batch([d], "IW2")
for precision in ("fp32_plain", "fp64"):
    d = S1Decoder(stream(*bursts((1000, 31))), precision=precision)
    try:                                # as far as they come: tile counts are read back from kernels
        d.get_azimuth_compressed_burst("IW2", 0, dtype=np.complex64)
    except S1GError:
        pass
""",
    # one 20-line group of a stripmap among others: packets that are not in a row
    "scattered": """
d = S1Decoder(stream(*[x for k in range(6) for x in bursts((40, 40 + k), swath="S%d" % (k % 2 + 1))]))
d.apply_eccm(1000, 10)
for precision in ("fp32", "fp64"):
    d.set_precision(precision)
    for level in ("raw", "range"):
        try:
            (d.get_swath if level == "raw" else d.get_range_compressed_swath)("S1", dtype=np.complex64)
        except S1GError:
            pass
""",
    "stripmap": """
for precision in ("fp32", "fp32_plain", "fp64"):
    d = S1Decoder(stream(*bursts((300, 40), swath="S1", beam_start=512, beam_sweep=0)), precision=precision)
    d.get_azimuth_compressed_swath("S1", dtype=np.complex64)
""",
    "adjoint": """
d = S1Decoder(stream(*bursts((300, 40), swath="S1", beam_start=512, beam_sweep=0)))
try:
    d.azimuth_adjoint("S1", 0, [1.0], 0.0)
except S1GError as e:
    assert "zero" in str(e) or "empty" in str(e), e       # kernels do nothing: the image is 0
assert count("launch:k_entropy_sums") == 1
""",
    "noalloc": """
lib = load_library()
x = np.zeros(4096, np.uint8)
p = x.ctypes.data
assert lib.s1g_decode_fdbaq_noalloc(p, 1000, p + 2048, 2, 8, p, 16, p + 3000, 0x1000) == 0
assert count("launch:k_decode_fdbaq") == 1
""",
    "packet": """
d = S1Decoder(stream(*bursts((300, 40))))
x = np.zeros(80, np.complex64)
assert d._lib.s1g_packet_samples(d.handle, 3, x.ctypes.data, 80, 0, 1) == 0
""",
}


@pytest.mark.parametrize("what", sorted(ORDER))
def test_tables_reach_the_device_before_their_readers(fake, what):
    """The handles' streams do not wait for the legacy stream, and a copy from
    pageable memory on that one may return before the device has the data; an
    asynchronous copy may read its source until the stream has been waited for."""
    fake(ORDER[what] + """
assert count("unordered") == 0, (count("unordered"), rt.fake_last_unordered())
assert count("pending") == 0
assert count("stale") == 0, count("stale")
""")


def test_swath_padding_is_done_when_the_call_returns(fake):
    """The rows of zeros between the bursts of a focused IW swath, in the caller's
    device buffer."""
    fake("""
d = S1Decoder(stream(*bursts((1000, 24), (1003, 24), (1001, 24))))
for level in range(4):
    rows, cols = ctypes.c_int64(), ctypes.c_int64()
    assert d._lib.s1g_swath_shape(d.handle, b"IW2", level, ctypes.byref(rows), ctypes.byref(cols)) == 0
    out = np.zeros((rows.value, cols.value), np.complex64)
    assert d._lib.s1g_swath_product(d.handle, b"IW2", level, out.ctypes.data, *out.shape, 0, 1) == 0
    assert count("pending") == 0, level
""")
