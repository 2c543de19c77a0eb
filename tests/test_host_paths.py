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
    env = dict(os.environ, LD_LIBRARY_PATH=str(out), S1G_AUTOTUNE="0", S1G_FFT_TUNE_FILE=str(out / "tune.txt"))

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
