"""The warp-cooperative FDBAQ walk against the oracle's serial one, bit for
bit, where its pieces can go wrong: blocks of one code up to full ones, every
bit-rate code, blocks of only the shortest codes (a block in a few of its 32
pieces) and only the longest (a block over more than 32 pieces), packets whose
symbols leave room for one warp per CTA, misaligned packet starts (every
packet of odd length shifts the next one)."""
import numpy as np
import pytest

import s1_oracle as O
from sentinel1_decode_gb300 import S1Decoder, synth


def packet_bytes(nq, codes, rng):
    """FDBAQ user data of one packet: `codes(brc)` draws the m-codes of a block."""
    nb = (2 * nq + 255) // 256
    brc = rng.integers(0, 5, nb) if codes != "short60k" else np.zeros(nb, int)
    out = []
    for ch in range(4):
        bits = ""
        for b in range(nb):
            n = 128 if b < nb - 1 else nq - 128 * (nb - 1)
            if ch == 0:
                bits += format(brc[b], "03b")
            if ch == 2:
                bits += format(int(rng.integers(0, 256)), "08b")
            table = synth.HUFFMAN[brc[b]]
            lens = np.array([l for _, l in table])
            if codes == "mixed":
                m = rng.integers(0, len(table), n)
            elif codes == "long":
                m = np.full(n, int(np.argmax(lens)))
            else:
                m = np.full(n, int(np.argmin(lens)))
            sign = rng.integers(0, 2, n)
            bits += "".join(str(s) + format(table[k][0], "0%db" % table[k][1]) for s, k in zip(sign, m))
        bits += "0" * (-len(bits) % 16)
        out.append(bits)
    bits = "".join(out)
    return int(bits, 2).to_bytes(len(bits) // 8, "big") if bits else b""


def stream(nq, codes, lines, seed):
    rng = np.random.default_rng(seed)
    user = [packet_bytes(nq, codes, rng) for _ in range(lines)]
    # an odd byte after some packets: the next ones start on another alignment
    user = [u + b"\0" * int(rng.integers(0, 2)) for u in user]
    hf = synth.RadarParams().fields(nq)
    fields = []
    for i in range(lines):
        f = dict(hf)
        f.update(coarse_time=1_000_000, fine_time=1 + i, sync_marker=synth.SYNC_MARKER, ecc_number=1, pri_count=1000 + i,
                 sc_data_word_index=i % 64 + 1, space_packet_count=i, baq_mode=12, baq_block_length=31, polarisation=4,
                 azimuth_beam_address=512, swath_number=synth.SWATH_NUMBERS["S1"], num_quadratures=nq)
        fields.append(f)
    head = synth.build_headers(fields, [len(u) for u in user])
    return b"".join(h.tobytes() + u for h, u in zip(head, user))


@pytest.mark.gpu
@pytest.mark.parametrize("nq,codes,lines", [
    (1, "mixed", 3), (31, "mixed", 5), (127, "short", 4), (128, "long", 4), (129, "mixed", 7), (256, "long", 3),
    (385, "mixed", 33), (1000, "short", 5), (1021, "long", 5), (6250, "mixed", 9), (60000, "short60k", 3)])
def test_walk_equals_the_serial_walk(lib_path, nq, codes, lines):
    data = stream(nq, codes, lines, seed=nq + lines)
    ref, status = O.decode_packets(data, O.get_packets(data))
    assert not status.any()
    d64 = S1Decoder(data, precision="fp64")
    got = d64.get_burst("S1", 0)
    np.testing.assert_array_equal(got.view(np.uint64), np.ascontiguousarray(ref[:, :2 * nq]).view(np.uint64))
    d64.close()
    d32 = S1Decoder(data, precision="fp32_plain")
    got = d32.get_burst("S1", 0, dtype=np.complex64)
    np.testing.assert_array_equal(got, ref[:, :2 * nq].astype(np.complex64))
    d32.close()
