"""Timed cases of the library's work, through its public entry points.

A case is a dict of plain values; `prepare` makes its Level-0 byte streams on
the GPU from a seed (headers by the package's synthetic generator, echoes and
FDBAQ user data by the torch code below) and opens the decoder handles that a
program keeps, `run` is one pass as a program calls it, `work` what the pass
cannot do without and `exact` its result in 64 bits from plain torch.

The scenes: point scatterers with their range chirp and azimuth phase history
(TOPS-steered for IW) over complex-Gaussian noise, FDBAQ blocks with a random
bit-rate code each and the THIDX of the block's RMS.
"""
import math

import numpy as np
import torch

from sentinel1_decode_gb300 import S1Decoder, batch_outputs, load_library, process_swath_batch, synth
from sentinel1_decode_gb300.decoder import batch_host_outputs

RAW, RANGE_COMPRESSED, AZIMUTH_COMPRESSED = 0, 1, 3
CF32, CF64 = 0, 1
C0 = 299792458.0
CARRIER = 5.405000454334350e9
WAVELENGTH = C0 / CARRIER
PI = 3.14159265358979          # the radar chain's own constant
BRC_CODES = [4, 5, 7, 10, 16]  # magnitudes per bit-rate code


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a quicklook over a few echo lines of a narrow stripmap window: the smallest call, launches and latency
        {"name": "sm_quicklook", "kind": "range", "swath": "S1", "lines": 64, "samples": 1000, "precision": "fp32"},
        # FDBAQ decode of one IW burst inside a program that allocates nothing: packets in, samples out
        {"name": "decode_iw", "kind": "decode", "swath": "IW2", "lines": 1500, "samples": 12000},
        # range-compressed IW burst (interferometry and RFI screening work on these), ragged sizes
        {"name": "range_iw", "kind": "range", "swath": "IW2", "lines": 1481, "samples": 11926, "precision": "fp32"},
        # the 1024 x 2048 stripmap scene of the benchmark, packets to focused image
        {"name": "stripmap", "kind": "stripmap", "swath": "S1", "lines": 1024, "samples": 2048, "precision": "fp32"},
        # a stripmap scene of ordinary size with odd lengths
        {"name": "stripmap_scene", "kind": "stripmap", "swath": "S3", "lines": 3301, "samples": 9250, "precision": "fp32"},
        # one IW burst to SLC at the benchmark's size
        {"name": "slc_iw2", "kind": "slc", "swath": "IW2", "lines": 1500, "samples": 12000, "precision": "fp32", "eccm": False},
        # one IW burst of another sub-swath, whose lengths have large prime factors (most real window lengths do)
        {"name": "slc_iw1", "kind": "slc", "swath": "IW1", "lines": 1457, "samples": 11838, "precision": "fp32", "eccm": False},
        # the same under radio interference with the notch on
        {"name": "slc_eccm", "kind": "slc", "swath": "IW2", "lines": 1500, "samples": 12000, "precision": "fp32", "eccm": True},
        # the 64-bit path, used to validate products
        {"name": "slc_fp64", "kind": "slc", "swath": "IW3", "lines": 1083, "samples": 3002, "precision": "fp64", "eccm": False},
        # the production unit: bursts of uneven size, both polarisations, one captured batch
        {"name": "swath_dualpol", "kind": "swath", "swath": "IW2", "lines": 1490, "samples": 12162, "bursts": 3, "pols": 2},
        # the same from new bytes in host memory to SLCs in host memory, one polarisation
        {"name": "swath_host", "kind": "host", "swath": "IW2", "lines": 1510, "samples": 11946, "bursts": 2, "pols": 1},
        # one evaluation of the autofocus objective: forward and adjoint of the azimuth chain
        {"name": "focus", "kind": "focus", "swath": "S1", "lines": 1024, "samples": 4096, "precision": "fp32", "terms": 2},
    ]


def draw(rng):
    kind = rng.choice(["range", "decode", "range", "stripmap", "slc", "slc", "slc", "swath", "host", "focus"])
    span = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    even = lambda n: n + (n & 1)  # noqa: E731
    c = {"kind": kind, "swath": rng.choice(["IW1", "IW2", "IW3"])}
    if kind == "range":
        if rng.random() < 0.5:
            c["swath"] = rng.choice(["S1", "S2", "S4", "S6"])
        c.update(lines=span(64, 1560), samples=even(span(700, 12500)), precision=rng.choice(["fp32", "fp32", "fp64"]))
    elif kind == "decode":
        c.update(lines=span(64, 1560), samples=even(span(500, 12500)))
    elif kind == "stripmap":
        c.update(swath=rng.choice(["S1", "S2", "S3", "S5_N"]), lines=span(512, 3301), samples=even(span(1200, 9250)),
                 precision=rng.choice(["fp32", "fp32", "fp64"]))
    elif kind == "slc":
        c.update(lines=rng.randint(1000, 1560), samples=even(span(2400, 12500)), precision="fp32", eccm=rng.random() < 0.3)
        if not c["eccm"] and rng.random() < 0.2:
            c.update(precision="fp64", lines=rng.randint(1000, 1100), samples=even(span(1500, 3000)))
    elif kind == "swath":
        c.update(lines=rng.randint(1060, 1540), samples=even(span(6000, 12100)), bursts=rng.randint(1, 3), pols=rng.randint(1, 2))
    elif kind == "host":
        c.update(lines=rng.randint(1060, 1540), samples=even(span(6000, 12100)), bursts=rng.randint(1, 2), pols=1)
    else:
        c.update(swath="S1", lines=span(512, 1024), samples=even(span(1500, 4096)), precision="fp32", terms=rng.randint(1, 4))
    return c


# ------------------------------------------------------------------ inputs
def _bursts(case, seed):
    """(lines, samples) of each burst; the bursts of a swath differ by a few lines and samples."""
    out = []
    for b in range(case.get("bursts", 1)):
        dl, ds = ((0, 0), (-37, 34), (23, -58))[b % 3]
        out.append((case["lines"] + dl, case["samples"] + ds))
    return out


def _beam(swath, lines):
    if swath.startswith("IW"):
        return np.rint(100 + np.arange(lines) * (820 / (lines - 1))).astype(int)
    return np.full(lines, 512, dtype=int)


def _chirp(p):
    t = np.arange(p["replica_len"]) / p["fs_mhz"]
    return torch.from_numpy(np.exp(2j * np.pi * (p["txpsf"] * t + 0.5 * p["txprr"] * t * t))).to("cuda", torch.complex64)


def _echo(swath, lines, samples, eccm, g):
    """Echo lines [lines, samples] of the scene, complex64."""
    radar = synth.RadarParams()
    p = synth.decoded_params(radar.fields(samples // 2), samples // 2)
    prf, fs = 1.0 / p["pri"], p["fs_mhz"] * 1e6
    eta = (torch.arange(lines, device="cuda", dtype=torch.float64) - lines / 2) / prf
    psi = -0.018 + _beam(swath, lines) * (0.036 / 1023)
    k_dc = -2 * radar.velocity_mps * ((psi[-1] - psi[0]) / (lines / prf)) / WAVELENGTH
    v = radar.velocity_mps * 0.95
    n_ch = p["replica_len"]
    spots = torch.zeros(lines, samples, dtype=torch.complex64, device="cuda")
    rows = torch.arange(lines, device="cuda")
    draws = torch.rand(150, 4, generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    for u0, u1, u2, u3 in draws:
        r0 = (p["delay_near"] + (0.03 + 0.94 * u0) * samples / fs) * C0 / 2
        if swath.startswith("IW"):
            c = (0.8 * u1 - 0.4) * lines / prf
            k, width = c + WAVELENGTH * r0 * k_dc * c / (2 * v * v), 0.12 * lines / prf
        else:
            c = (0.7 * u1 - 0.35) * lines / prf
            k, width = c, 0.35 * lines / prf
        rr = torch.sqrt(r0 ** 2 + (v * (eta - k)) ** 2)
        a = 20.0 * (0.3 + 1.2 * u3) * torch.exp(-0.5 * ((eta - c) / width) ** 2)
        at = torch.round((2 * rr / C0 - p["delay_near"]) * fs).long() - n_ch // 2
        ok = (at >= 0) & (at < samples)
        turn = torch.remainder(2 * rr / WAVELENGTH, 1.0) - u2
        spots[rows, at.clamp(0, samples - 1)] += torch.polar(torch.where(ok, a, 0.0), -2 * math.pi * turn).to(torch.complex64)
    nfft = 1 << int(math.ceil(math.log2(samples + n_ch)))
    echo = torch.fft.ifft(torch.fft.fft(spots, nfft, dim=1) * torch.fft.fft(_chirp(p), nfft), dim=1)[:, :samples]
    echo = echo + torch.view_as_complex(torch.randn(lines, samples, 2, generator=g, device="cuda")) * 5.0
    if eccm:  # tones and a chirped interferer on three lines out of ten
        t = torch.arange(samples, device="cuda", dtype=torch.float64) / fs
        hit = (torch.rand(lines, generator=g, device="cuda") < 0.3).float()
        level = hit * 6.0 * 10 ** ((10 + 20 * torch.rand(lines, generator=g, device="cuda")) / 20) / math.sqrt(6)
        f = (torch.rand(lines, 5, generator=g, device="cuda", dtype=torch.float64) - 0.5) * 0.9 * fs
        for k in range(5):
            echo += level[:, None] * torch.polar(torch.ones_like(t), 2 * math.pi * torch.remainder(f[:, k, None] * t, 1.0)).to(torch.complex64)
        kr = (torch.rand(lines, generator=g, device="cuda", dtype=torch.float64) - 0.5) * 4e12
        u = t - t.mean()
        echo += level[:, None] * torch.polar(torch.ones_like(t), math.pi * kr[:, None] * u * u).to(torch.complex64)
    return echo


_TABLES = {}


def _tables():
    """Levels [5][16], thresholds [5][15] (both in units of the sigma factor), code words and lengths, on the GPU."""
    if not _TABLES:
        lev = torch.tensor(synth.NORMALIZED_RECONSTRUCTION, dtype=torch.float64)
        mid = torch.full((5, 15), float("inf"), dtype=torch.float64)
        code, length = torch.zeros(5, 16, dtype=torch.int64), torch.zeros(5, 16, dtype=torch.int64)
        for b, n in enumerate(BRC_CODES):
            mid[b, : n - 1] = (lev[b, : n - 1] + lev[b, 1:n]) / 2
            for m, (word, bits) in enumerate(synth.HUFFMAN[b]):
                code[b, m], length[b, m] = word, bits
        _TABLES.update(lev=lev.cuda(), mid=mid.cuda(), code=code.cuda(), length=length.cuda(),
                       sf=torch.tensor(synth.THIDX_TO_SF, dtype=torch.float64).cuda())
    return _TABLES


def _encode(echo, g):
    """FDBAQ user data of echo lines: (bytes uint8, bytes per packet, decoded samples complex128)."""
    T = _tables()
    lines, samples = echo.shape
    nq, nb = samples // 2, (samples + 255) // 256
    parts, sizes, decoded = [], [], []
    blk = (torch.arange(nq, device="cuda") // 128).clamp(max=nb - 1)
    first = (torch.arange(nb, device="cuda") * 128).clamp(max=nq - 1)
    brc_all = torch.randint(0, 5, (lines, nb), generator=g, device="cuda")
    head = torch.tensor([3, 0, 8, 0], device="cuda")
    for l0 in range(0, lines, 256):
        e, brc = echo[l0:l0 + 256], brc_all[l0:l0 + 256]
        n = e.shape[0]
        ch = torch.stack([e[:, 0::2].real, e[:, 1::2].real, e[:, 0::2].imag, e[:, 1::2].imag], 1).double()   # IE IO QE QO
        pad = torch.nn.functional.pad(ch, (0, nb * 128 - nq)).reshape(n, 4, nb, 128)
        count = torch.full((nb,), 512.0, device="cuda", dtype=torch.float64)
        count[-1] = 4 * (nq - 128 * (nb - 1))
        rms = torch.sqrt((pad ** 2).sum(dim=(1, 3)) / count)
        th = torch.bucketize(rms, (T["sf"][1:] + T["sf"][:-1]) / 2).clamp(9, 254)
        b_q, sf = brc[:, None, blk], T["sf"][th][:, None, blk]
        mag = ch.abs() / sf
        m = torch.zeros(ch.shape, dtype=torch.int64, device="cuda")
        for k in range(15):
            m += mag > T["mid"][:, k][b_q]
        neg = (ch < 0) & (m > 0)
        value = torch.where(neg, -1.0, 1.0) * (T["lev"][b_q.expand_as(m), m] * sf)
        z = torch.empty(n, samples, dtype=torch.complex128, device="cuda")
        z[:, 0::2], z[:, 1::2] = torch.complex(value[:, 0], value[:, 2]), torch.complex(value[:, 1], value[:, 3])
        decoded.append(z)
        hl = T["length"][b_q.expand_as(m), m]
        word, width = (neg.long() << hl) | T["code"][b_q.expand_as(m), m], hl + 1
        before = torch.cumsum(width, 2) - width
        bits = width.sum(2) + nb * head
        padded = (bits + 15) // 16 * 16
        starts = torch.cumsum(padded.reshape(-1), 0).reshape(n, 4) - padded
        at = starts[:, :, None] + before + head[None, :, None] * (blk + 1)
        at_head = starts[:, :, None] + before[:, :, first] + head[None, :, None] * torch.arange(nb, device="cuda")
        total = int(padded.sum())
        stream = torch.zeros(total, dtype=torch.uint8, device="cuda")
        for pos, val, wid in ((at, word, width), (at_head[:, 0], brc, torch.full_like(brc, 3)), (at_head[:, 2], th, torch.full_like(th, 8))):
            for k in range(int(wid.max())):
                # past its own width a value writes nothing: it is sent to its last bit again
                j = torch.minimum(torch.full_like(wid, k), wid - 1)
                stream[pos + j] = ((val >> (wid - 1 - j)) & 1).to(torch.uint8)
        weight = torch.tensor([128, 64, 32, 16, 8, 4, 2, 1], device="cuda", dtype=torch.uint8)
        parts.append((stream.reshape(-1, 8) * weight).sum(1).to(torch.uint8))
        sizes.append(padded.sum(1) // 8)
    return torch.cat(parts), torch.cat(sizes), torch.cat(decoded)


def _orbit():
    p0 = np.array([6.0e6, 1.0e6, 3.6e6])
    d = np.cross(p0, np.array([0.3, -0.2, 1.0]))
    return p0, synth.RadarParams().velocity_mps * d / np.linalg.norm(d)


START = 1_000_000.3


def _headers(swath, shapes, pol, sizes):
    """Packet headers [packets][68] and, per burst, the first packet's fields."""
    fields, firsts, number, pri_count, t = [], [], 0, 100_000, START
    p0, v0 = _orbit()
    words = None
    for lines, samples in shapes:
        hf = synth.RadarParams().fields(samples // 2)
        pri = hf["pri"] / synth.F_REF * 1e-6
        beam = _beam(swath, lines)
        t += 300 * pri
        pri_count += 300
        for a in range(lines):
            tt = t + a * pri
            if number % 64 == 0:
                t_sv = math.floor(2 * (START + number * pri)) / 2
                words = synth.subcomm_words(t_sv, p0 + v0 * (t_sv - START), v0)
            f = dict(hf)
            f.update(coarse_time=int(tt), fine_time=max(1, int((tt - int(tt)) * 65536)), sync_marker=synth.SYNC_MARKER,
                     data_take_id=0x0D6D0C0, ecc_number=8 if swath.startswith("IW") else 1, rx_channel_id=pol,
                     instrument_configuration_id=7, sc_data_word_index=number % 64 + 1, sc_data_word=words[number % 64],
                     space_packet_count=number, pri_count=pri_count + a, baq_mode=12, baq_block_length=31, rx_gain=8,
                     polarisation=4, temperature_compensation=3, elevation_beam_address=6, azimuth_beam_address=int(beam[a]),
                     tx_pulse_number=6, swap=1, swath_number=synth.SWATH_NUMBERS[swath], num_quadratures=samples // 2,
                     packet_sequence_count=number)
            if a == 0:
                firsts.append(f)
            fields.append(f)
            number += 1
        t += lines * pri
        pri_count += lines
    return synth.build_headers(fields, sizes), firsts


def _stream(case, seed, pol=0):
    """(Level-0 bytes on the GPU, packet offsets, decoded samples of each burst)."""
    shapes = _bursts(case, seed)
    data, sizes, decoded = [], [], []
    for b, (lines, samples) in enumerate(shapes):
        g = torch.Generator("cuda").manual_seed(1_000_003 * seed + 1009 * pol + b)
        d, s, z = _encode(_echo(case["swath"], lines, samples, case.get("eccm", False), g), g)
        data.append(d)
        sizes.append(s)
        decoded.append(z)
    user, size = torch.cat(data), torch.cat(sizes)
    head, firsts = _headers(case["swath"], shapes, pol, size.tolist())
    packets = size.numel()
    begin = torch.cumsum(size + 68, 0) - (size + 68)
    out = torch.zeros(int(size.sum()) + 68 * packets, dtype=torch.uint8, device="cuda")
    which = torch.repeat_interleave(torch.arange(packets, device="cuda"), size)
    out[torch.arange(user.numel(), device="cuda") + 68 * (which + 1)] = user
    out[begin[:, None] + torch.arange(68, device="cuda")] = torch.from_numpy(np.ascontiguousarray(head)).cuda()
    return out, begin, decoded, firsts


def _ok(decoder, code):
    if code:
        raise RuntimeError("s1g error %d: %s" % (code, load_library().s1g_last_error(decoder.handle).decode()))


def _open(stream, precision):
    host = stream.cpu().numpy()
    return S1Decoder.from_pointer(host.ctypes.data, host.size, precision=precision)


class _Device:
    """A device buffer of the library seen as an array; the tensor made of it keeps the handles that own the memory open."""

    def __init__(self, handles, ptr, rows, cols, pitch):
        self.handles = handles
        self.__cuda_array_interface__ = {"shape": (rows, cols, 2), "typestr": "<f4", "data": (ptr, False), "version": 3,
                                         "strides": (pitch * 8, 8, 4)}


THETA = [3.1, -1.7, 0.6, 0.4]
CENTROID = 12.5


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "decode":
        s["bytes"], s["offsets"], _, _ = _stream(case, seed)
        s["out"] = torch.empty(case["lines"], case["samples"], dtype=torch.complex64, device="cuda")
        s["status"] = torch.empty(case["lines"], dtype=torch.int32, device="cuda")
        return s
    precision = case.get("precision", "fp32")
    streams = [_stream(case, seed, pol)[0] for pol in range(case.get("pols", 1))]
    s["handles"] = [_open(x, precision) for x in streams]
    h = s["handles"][0]
    if case.get("eccm"):
        h.apply_eccm(13000, 100)
    if kind in ("range", "slc", "stripmap"):
        rows, cols = case["lines"], case["samples"]
        if kind == "slc":
            rows = h.unfold_shape(case["swath"], 0)[1]
        s["out"] = torch.empty(rows, cols, dtype=torch.complex128 if precision == "fp64" else torch.complex64, device="cuda")
    if kind == "host":
        # what the program reads each acquisition from and delivers it to: page-locked host memory
        s["bytes"] = streams[0].cpu().pin_memory()
        s["out"] = [torch.empty(h.unfold_shape(case["swath"], b)[1], n, dtype=torch.complex64).pin_memory()
                    for b, (_, n) in enumerate(_bursts(case, seed))]
        batch_host_outputs(h, [x.data_ptr() for x in s["out"]])
    return s


def run(s):
    case = s["case"]
    kind, swath = case["kind"], case["swath"].encode()
    lib = load_library()
    if kind == "decode":
        out = s["out"]
        lib.s1g_decode_fdbaq_noalloc(s["bytes"].data_ptr(), s["bytes"].numel(), s["offsets"].data_ptr(), case["lines"],
                                     case["samples"] // 2, out.data_ptr(), out.shape[1], s["status"].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return {"samples": out, "status": s["status"]}
    h = s["handles"][0]
    if kind in ("range", "slc", "stripmap"):
        out = s["out"]
        typ = CF64 if out.dtype == torch.complex128 else CF32
        rows, cols = out.shape
        if kind == "stripmap":
            code = lib.s1g_swath_product(h.handle, swath, AZIMUTH_COMPRESSED, out.data_ptr(), rows, cols, typ, 1)
        else:
            level = RANGE_COMPRESSED if kind == "range" else AZIMUTH_COMPRESSED
            code = lib.s1g_burst_product(h.handle, swath, 0, level, out.data_ptr(), rows, cols, typ, 1)
        _ok(h, code)
        return out
    if kind == "swath":
        process_swath_batch(s["handles"], case["swath"])
        return [torch.view_as_complex(torch.as_tensor(_Device(s["handles"], p, r, c, pitch), device="cuda"))
                for p, r, c, pitch, _ in batch_outputs(h)]
    if kind == "host":
        h.reload_from_pointer(s["bytes"].data_ptr(), s["bytes"].numel())
        process_swath_batch(s["handles"], case["swath"])
        return s["out"]
    loss, theta, centroid = h.azimuth_adjoint(case["swath"], 0, THETA[: case["terms"]], CENTROID)
    # the chain's arithmetic is 32-bit: so are the values a caller gets out of it
    return {"loss": np.float32(loss), "theta": theta.astype(np.float32), "centroid": np.float32(centroid)}


# ------------------------------------------------------------------ the work
def _fft(n):
    return 5.0 * n * math.log2(max(n, 2))


def work(case):
    """Bytes: each stage's input read once and its output written once where a burst does not stay on the chip (a corner
    turn lies between the stages). Flops: one transform of the line's own length for each that the chain names."""
    kind, eight = case["kind"], 16 if case.get("precision") == "fp64" else 8
    total = {"bytes": 0.0, "flops": 0.0}
    for _ in range(case.get("pols", 1)):
        for n_a, n_r in _bursts(case, 0):
            coded = n_a * (68 + n_r * 0.83)
            burst = eight * n_a * n_r
            if kind == "decode":
                b, f = coded + burst, 0.0
            elif kind == "range":
                b, f = coded + burst, 2 * n_a * _fft(n_r + 2573)
            elif kind == "stripmap":
                b, f = coded + 7 * burst, 2 * n_a * _fft(n_r + 2573) + 2 * n_r * _fft(n_a) + n_a * _fft(n_r)
            elif kind == "focus":
                b, f = coded + 15 * burst, 2 * n_a * _fft(n_r + 2573) + 4 * n_r * _fft(n_a) + 4 * n_a * _fft(n_r)
            else:
                S, tiles = 4.6 * n_a, 6 if case["swath"] == "IW2" else 5
                b = coded + eight * n_r * (2 * n_a + 4 * S + n_a)
                f = 2 * n_a * _fft(n_r + 2573) + n_r * (_fft(n_a) + 3 * _fft(S) + 2 * _fft(tiles * S)) + 2 * S * _fft(n_r)
                if kind == "host":
                    b += coded + burst
            total["bytes"] += b
            total["flops"] += f
    return total


# ------------------------------------------------------------------ the results in 64 bits
def _lin(a, b, n):
    return a + torch.arange(n, device="cuda", dtype=torch.float64) * ((b - a) / (n - 1))


def _cis(th):
    return torch.polar(torch.ones_like(th), th)


class _Geometry:
    """What the chain takes from the packet headers of a burst (one burst per stream)."""

    def __init__(self, case, f, lines, samples):
        self.n_a, self.n_r, self.swath = lines, samples, f["swath_number"]
        p = synth.decoded_params(f, samples // 2)
        self.psf, self.prr, self.pl, self.L = p["txpsf"], p["txprr"], p["txpl"], p["replica_len"]
        self.fs, self.pri = p["fs_mhz"] * 1e6, f["pri"] / synth.F_REF * 1e-6
        self.prf, self.T = 1 / self.pri, lines * self.pri
        swst = f["swst"] / synth.F_REF * 1e-6
        self.near = f["rank"] * self.pri + swst + synth.DELTA_T_SUPPRESSED
        self.far = self.near + samples / self.fs
        self.slant = _lin(self.near * C0 / 2, self.far * C0 / 2, samples)
        i = torch.arange(samples, device="cuda", dtype=torch.float64)
        self.tc = (swst + 1.439e-6) + (swst + f["rank"] * self.pri - i / self.fs) / 2
        self.fr = _lin(-self.fs / 2, self.fs / 2, samples)
        self.t0 = float(f["coarse_time"]) + 1.0 / float(f["fine_time"])
        # state vectors: one per complete 64-packet cycle after the first, equal times dropped
        p0, v0 = _orbit()
        times = []
        for c in range(1, (lines - 1) // 64):
            t = math.floor(2 * (START + 64 * c * self.pri)) / 2
            if not times or t > times[-1]:
                times.append(t)
        self.times, self.p0 = times, p0
        self.v0, self.vel = v0, v0.astype(np.float32).astype(np.float64)
        self.speed = float(np.linalg.norm(self.vel))
        self.bd = 675.0 if self.swath == 11 else 600.0
        beam = _beam(case["swath"], lines)
        angle = -0.018 + beam * (0.036 / 1023)
        self.rate = -2 * self.speed * ((angle[-1] - angle[0]) / (self.pri * lines)) / WAVELENGTH

    def v2_eff(self, t, slant):
        """Squared effective velocity at times t (rows) and slant ranges (columns)."""
        t = torch.clamp(t, self.times[0], self.times[-1])
        pos = torch.as_tensor(self.p0, device="cuda") + torch.as_tensor(self.v0, device="cuda") * (t[:, None] - START)
        lat = pos[:, 2] / pos[:, 0]
        a, b = 6378137.0, 6356752.3142
        re = torch.sqrt(((a * a * torch.cos(lat)) ** 2 + (b * b * torch.sin(lat)) ** 2) / ((a * torch.cos(lat)) ** 2 + (b * torch.sin(lat)) ** 2))
        h = torch.linalg.norm(pos, dim=1)
        beta = ((re * re + h * h)[:, None] - slant[None, :] ** 2) / (2 * re * h)[:, None]
        return self.speed * (re / h)[:, None] * self.speed * beta



def _range_compress(g, z):
    L, M = g.L, g.n_r + 2 * g.L
    t = _lin(0.0, g.pl, L)
    ref = torch.zeros(M, dtype=torch.complex128, device="cuda")
    ref[(M - L) // 2:(M - L) // 2 + L] = _cis(2.0 * PI * (g.psf * t + 0.5 * g.prr * t * t)) / L
    energy = float(((ref.abs() ** 2) ** 2 / M).sum())
    ref = torch.fft.fft(ref).conj() / energy
    out = torch.empty_like(z)
    for a in range(0, g.n_a, 512):
        y = torch.fft.ifft(torch.fft.fft(torch.nn.functional.pad(z[a:a + 512], (L, L)), dim=1) * ref, dim=1)
        out[a:a + 512] = torch.roll(y, M // 2, dims=1)[:, L:M - L]
    return out


def _notch(z, det, mit):
    """Zeroes the short-time bins whose spectrum changes fast, on the lines whose spectrum reaches `det`."""
    n = z.shape[1]
    windows = math.floor(n / 128 * 2)
    hot = torch.nonzero(~(torch.fft.fft(z, dim=1).abs().amax(1) < det))[:, 0]
    lines = z[hot]
    span = [(64 * i, 64 * i + 128 if 64 * i + 128 <= n else n - 1) for i in range(windows)]
    spec = torch.zeros(len(hot), windows, 128, dtype=torch.complex128, device="cuda")
    for i, (a, b) in enumerate(span):
        spec[:, i, : b - a] = lines[:, a:b]
    spec = torch.fft.fft(spec, dim=2)
    grad = torch.empty_like(spec)
    grad[..., 1:-1] = (spec[..., 2:] - spec[..., :-2]) / 2
    grad[..., 0], grad[..., -1] = spec[..., 1] - spec[..., 0], spec[..., -1] - spec[..., -2]
    back = torch.fft.ifft(torch.where(grad.abs() < mit, spec, 0.0), dim=2)
    for i, (a, b) in enumerate(span):
        lines[:, a:b] = back[:, i, : b - a]
    z[hot] = lines
    return z


def _centroid(g, rc):
    """Doppler centroid per range bin: lag-1 phases, 30 block means, unwrap, quadratic fit."""
    t = _lin(0.0, 1.06, g.n_a)
    d = _cis(PI * g.rate * (t - 0.53) ** 2)[:, None]
    sums = ((rc[:-1] * d[:-1]) * (rc[1:] * d[1:]).conj()).sum(0).cpu().numpy()
    prf = g.prf
    wrapped = -prf * np.angle(sums) / (2 * PI)
    blocks = 30
    size = g.n_r // blocks
    fine = np.array([wrapped[b * size:min((b + 1) * size, g.n_r - 1) if (b + 1) * size >= g.n_r else (b + 1) * size].mean() for b in range(blocks)])
    rt = np.linspace(g.near, g.far, blocks) - g.near
    spec = np.zeros(blocks * 8, dtype=np.complex128)
    spec[:blocks] = np.floor(np.abs(np.cos(2 * PI * fine / prf) + 1j * np.sin(2 * PI * fine / prf)))
    spec = np.fft.fft(spec)
    k = int(np.argmax(np.abs(spec) ** 2))
    step = float(np.float32(rt[1]))
    slope = np.fft.fftfreq(blocks * 8, step)[k] / step
    line = slope * rt + np.angle(spec[k]) / (2 * PI)
    rest = np.angle(np.exp(1j * (2 * PI * fine / prf - line)))
    poly = np.polynomial.polynomial.polyfit(rt / rt[-1], (line + rest / (2 * PI)) * prf, 2)
    x = _lin(0.0, 1.0, g.n_r)
    return poly[0] + poly[1] * x + poly[2] * x * x


def _unfold_frequency(g, rc):
    S = math.floor(abs(g.rate * g.T / g.prf) * g.n_a)
    half = abs(g.rate * g.T / g.prf) * g.prf / 2
    start, end = int(S // 2 - math.floor(g.bd) / 2), int(S // 2 + math.floor(g.bd) / 2)
    ramp = _cis(-PI / g.rate * _lin(-half, half, S) ** 2)[:, None]
    out = torch.empty(S, g.n_r, dtype=torch.complex128, device="cuda")
    for c in range(0, g.n_r, 1024):
        x = torch.roll(torch.fft.fft(rc[:, c:c + 1024], dim=0), g.n_a // 2, dims=0)
        reps = math.floor(abs(g.rate * g.T / g.prf))
        tile = reps * g.n_a + math.floor((abs(g.rate * g.T / g.prf) - reps) * g.n_a)
        y = x.repeat(reps + 1, 1)[:S]
        y[tile:] = 0
        y = torch.fft.fft(y * ramp, dim=0)
        band = torch.zeros_like(y)
        band[: end - start] = y[start:end]
        out[:, c:c + 1024] = torch.fft.ifft(band, dim=0) * ramp.conj()
    return out


def _row_pass(g, x, fa, t, fdc, tops):
    """Range transforms, secondary range compression, scale, migration phase and azimuth filter; also the FM rates."""
    out, rate = torch.empty_like(x), torch.empty(x.shape if tops else (0,), dtype=torch.float64, device="cuda")
    scale = 1 / torch.sqrt((g.slant[g.n_r // 2] / g.slant) ** 3)
    for a in range(0, x.shape[0], 512):
        v2 = g.v2_eff(t[a:a + 512], g.slant)
        f = fa[a:a + 512, None] + fdc
        D = torch.sqrt(1 - WAVELENGTH ** 2 * f * f / (4 * v2))
        y = torch.fft.fft(x[a:a + 512], dim=1) if tops else x[a:a + 512]
        y = torch.fft.ifft(y * _cis(-PI * g.fr ** 2 * C0 * g.slant * f * f / (2 * v2 * CARRIER ** 3 * D * D)), dim=1) * g.n_r
        th = 4 * PI * g.slant * D / WAVELENGTH + 2 * PI * f * g.tc
        if tops:
            th = th - 4 * PI * g.fr * (g.slant / D - g.slant) / C0
            rate[a:a + 512] = -2 * v2 * D ** 3 / (WAVELENGTH * g.slant)
        out[a:a + 512] = y * scale * _cis(th)
    return out, rate


def _resample(v, n):
    """Rows of v resampled to n points, linearly."""
    m = v.shape[1]
    at = torch.arange(n, device="cuda") * (m - 1)
    i = torch.clamp(at // (n - 1), max=m - 2)
    w = (at - i * (n - 1)).double() / (n - 1)
    return v[:, i] * (1 - w) + v[:, i + 1] * w


def _unfold_time(g, x, ka, fdc):
    S, n_r = x.shape
    width = abs(g.rate * g.T / g.prf) * g.prf - g.bd
    span = g.T + (width - 2 * g.bd) / abs(float(ka[:, 0].mean()))
    inside = S // 2 < n_r and n_r // 2 < S
    mid = float(ka[n_r // 2, S // 2]) if inside else float(ka[S // 2, n_r // 2])
    n_ref = float(fdc[n_r // 2]) / mid
    span *= 1.05 if g.swath == 11 else 0.9
    tiles = math.ceil((n_ref + span / 2) / g.T) - math.floor((n_ref - span / 2) / g.T)
    rows = math.floor(g.prf * g.T)
    down = rows + math.floor(g.bd * (1.15 if g.swath == 11 else 0.26))
    n = tiles * S
    start, end = int(n // 2 - width / 2), int(n // 2 + width / 2)
    t_in, t_out = _lin(-span / 2, span / 2, n), _lin(n_ref - span / 2, n_ref + span / 2, down)
    at = torch.arange(down, device="cuda") * (n - 1)
    i = torch.clamp(at // (down - 1), max=n - 2)
    u = (at - i * (down - 1)).double() / (down - 1)
    lo = down // 2 - rows // 2
    keep = slice(lo, down // 2 + rows // 2)
    out = torch.empty(keep.stop - keep.start, n_r, dtype=torch.complex128, device="cuda")

    def phase(k, dc, t):
        kt = -k * g.rate / (g.rate - k)
        tt = -dc / k + t
        return PI * kt * tt * tt - 2 * PI * (kt + k) * (-dc / k) * tt

    for c in range(0, n_r, 256):
        k, dc = ka[:, c:c + 256].T.contiguous(), fdc[c:c + 256, None]
        y = x[:, c:c + 256].T.repeat(1, tiles) * _cis(-phase(_resample(k, n), dc, t_in))
        y = torch.fft.fft(y, dim=1)
        band = torch.zeros_like(y)
        band[:, : end - start] = y[:, start:end]
        y = torch.fft.ifft(band, dim=1)
        o = (0.5 * u * (u - 1)) * y[:, torch.clamp(i - 1, min=0)] + (1 - u * u) * y[:, i] + (0.5 * u * (u + 1)) * y[:, i + 1]
        out[:, c:c + 256] = (o * _cis(phase(_resample(k, down), dc, t_out)))[:, keep].T
    return out


def _image(case, g, z):
    if case.get("eccm"):
        z = _notch(z.clone(), 13000, 100)
    rc = _range_compress(g, z)
    if case["kind"] == "range":
        return rc
    if case["kind"] == "stripmap":
        x = torch.roll(torch.fft.fft(rc, dim=0), g.n_a // 2, dims=0)
        fa, t = _lin(-g.prf / 2, g.prf / 2, g.n_a), g.t0 + g.T / g.prf * torch.arange(g.n_a, device="cuda", dtype=torch.float64)
        return torch.fft.ifft(_row_pass(g, x, fa, t, torch.zeros_like(g.slant), False)[0], dim=0)
    fdc = _centroid(g, rc)
    x = _unfold_frequency(g, rc)
    S = x.shape[0]
    half = abs(g.rate * g.T / g.prf) * g.prf / 2
    t = g.t0 + g.T / g.prf / (S / g.n_a) * torch.arange(S, device="cuda", dtype=torch.float64)
    x, ka = _row_pass(g, x, _lin(-half, half, S), t, fdc, True)
    return _unfold_time(g, torch.fft.ifft(x, dim=0), ka, fdc)


def _entropy(case, g, z):
    """Loss and gradients of the azimuth chain by automatic differentiation."""
    x = _range_compress(g, z)
    theta = torch.tensor(THETA[: case["terms"]], dtype=torch.float64, device="cuda", requires_grad=True)
    fc = torch.tensor(CENTROID, dtype=torch.float64, device="cuda", requires_grad=True)
    xa = torch.linspace(-1, 1, g.n_a, device="cuda", dtype=torch.float64)
    phi = sum(theta[j] * xa ** (j + 2) for j in range(case["terms"]))
    y = torch.fft.fft(x * _cis(-phi)[:, None], dim=0)
    r_ref = g.slant[g.n_r // 2]
    v2 = g.v2_eff(torch.tensor([g.t0 + 0.5 * g.T], device="cuda", dtype=torch.float64), r_ref[None])[0, 0]
    f = torch.fft.fftfreq(g.n_a, 1 / g.prf, device="cuda", dtype=torch.float64) + fc
    D = torch.sqrt(1 - WAVELENGTH ** 2 * f * f / (4 * v2))
    fr = torch.fft.fftfreq(g.n_r, 1 / g.fs, device="cuda", dtype=torch.float64)
    y = torch.fft.ifft(torch.fft.fft(y, dim=1) * _cis(4 * math.pi * r_ref * (1 / D - 1)[:, None] * fr / C0), dim=1)
    y = torch.fft.ifft(y * _cis(-4 * math.pi / WAVELENGTH * g.slant * (1 - D)[:, None]), dim=0)
    p = y.real ** 2 + y.imag ** 2
    p = p / p.sum()
    loss = -(p * torch.log(p)).sum()
    loss.backward()
    return {"loss": loss.detach(), "theta": theta.grad, "centroid": fc.grad}


def exact(case, seed):
    _, _, decoded, firsts = _stream(case, seed)
    if case["kind"] == "decode":
        return {"samples": decoded[0], "status": None}
    if case["kind"] in ("swath", "host"):
        return None   # several bursts one after another: the single bursts' cases say it
    g = _Geometry(case, firsts[0], case["lines"], case["samples"])
    if case["kind"] == "focus":
        return _entropy(case, g, decoded[0])
    return _image(case, g, decoded[0])
