"""Frames whose record chains are walked by guessing that the next records have
the size of the last (FoR sub-blocks, ALP sub-blocks, ALP-RD exceptions), and
the DICT and ALP-RD frames decoded as warp items with their dictionary written
before and their exceptions after.  Each frame is the oracle's encoding of a
block; its values must come back bit for bit through the device reader and the
host reader, with and without nulls."""
import numpy as np
import pytest

from test_device_reader import F64, I64, device_decode

pytestmark = pytest.mark.gpu

M_ALP, M_DICT, M_FOR, M_ALP_RD = 9, 19, 50, 52


def widths(rng, n, run):
    """i64 values whose range in each 1,024 has a width redrawn every `run` sub-blocks."""
    nsub = (n + 1023) // 1024
    w = np.repeat(rng.integers(0, 60, (nsub + run - 1) // run), run)[:nsub]
    hi = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
    u = rng.integers(0, 1 << 62, n, dtype=np.int64).astype(np.uint64)
    return u & np.repeat(hi, 1024)[:n]


def decimals(rng, n, exc):
    """Two-decimal f64 values with `exc(k)` random ones in sub-block k."""
    v = np.floor(rng.random(n) * 1e5) / 100.0
    bits = v.view(np.uint64).copy()
    for k in range((n + 1023) // 1024):
        at = k * 1024 + rng.permutation(min(1024, n - k * 1024))[: exc(k)]
        bits[at] = rng.random(at.size).view(np.uint64)
    return bits


def rd_exceptions(rng, n, rate):
    bits = (np.uint64(0x3FF00) << np.uint64(46)) | rng.integers(0, 1 << 46, n, dtype=np.int64).astype(np.uint64)
    m = rng.random(n) < rate
    bits[m] = rng.integers(0, 1 << 62, int(m.sum()), dtype=np.int64).astype(np.uint64)
    return bits


def distinct(rng, n, card):
    d = rng.integers(0, 1 << 62, card, dtype=np.int64).astype(np.uint64)
    return d[rng.integers(0, card, n)]


CASES = [
    ("for_one_value", M_FOR, lambda r: widths(r, 1, 1)),
    ("for_each_width_new", M_FOR, lambda r: widths(r, 40 * 1024 + 1, 1)),
    ("for_runs_of_5", M_FOR, lambda r: widths(r, 131072, 5)),
    ("for_runs_of_33", M_FOR, lambda r: widths(r, 131071, 33)),
    ("for_one_width", M_FOR, lambda r: widths(r, 131072, 128)),
    ("alp_no_exceptions", M_ALP, lambda r: decimals(r, 70_001, lambda k: 0)),
    ("alp_mixed_exceptions", M_ALP, lambda r: decimals(r, 70_001, lambda k: k % 3 * 7)),
    ("alp_same_exceptions", M_ALP, lambda r: decimals(r, 40_960, lambda k: 5)),
    ("rd_no_exceptions", M_ALP_RD, lambda r: rd_exceptions(r, 5_000, 0.0)),
    ("rd_few_exceptions", M_ALP_RD, lambda r: rd_exceptions(r, 32_768, 0.001)),
    ("rd_exceptions", M_ALP_RD, lambda r: rd_exceptions(r, 131_072, 0.1)),
    ("dict_one_value", M_DICT, lambda r: distinct(r, 1_500, 1)),
    ("dict_small", M_DICT, lambda r: distinct(r, 33_000, 200)),
    ("dict_two_subblocks", M_DICT, lambda r: distinct(r, 20_001, 2_049)),
    ("dict_large", M_DICT, lambda r: distinct(r, 131_072, 40_000)),
]


def stream_of(payload, mode, wire, n, valid=None):
    """A one-frame stream; with `valid` (bool per position) a RAW validity blob."""
    s = b"FCR1" + bytes([2, 0 if valid is None else 1, 16, wire])
    s += (n if valid is None else valid.size).to_bytes(8, "little")
    if valid is not None:
        blob = b"\0" + np.packbits(valid, bitorder="little").tobytes()
        ln, v = b"", len(blob)
        while v > 127:
            ln += bytes([v & 127 | 128])
            v >>= 7
        s += ln + bytes([v]) + blob
    return s + bytes([mode]) + n.to_bytes(4, "little") + len(payload).to_bytes(4, "little") + payload


@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("name,mode,make", CASES, ids=[c[0] for c in CASES])
def test_frame_decodes(qb, oracle, name, mode, make, nulls):
    rng = np.random.default_rng(len(name) + 100 * mode)
    vals = make(rng)
    wire = I64 if mode == M_FOR else F64
    payload = oracle.encode_mode(mode, vals, oracle.DT_U64 if mode == M_FOR else oracle.DT_F64, level=1)
    assert payload is not None
    valid, want = None, vals
    if nulls:
        valid = np.zeros(vals.size + vals.size // 5 + 3, bool)
        valid[rng.permutation(valid.size)[: vals.size]] = True
        want = np.zeros(valid.size, np.uint64)
        want[valid] = vals
    s = stream_of(bytes(payload), mode, wire, vals.size, valid)
    rc, w, n, got, _ = device_decode(qb, s, 8 * want.size, offset=3)
    assert (rc, w, n) == (0, wire, want.size)
    assert got == want.tobytes()
    assert np.ascontiguousarray(qb.decompress_column(s).values).view(np.uint64).tobytes() == want.tobytes()


def test_damaged_chains_match_oracle(qb, oracle):
    """A width over 64, a cut chain and a cut last sub-block, at sub-blocks the guess reaches and the first one."""
    from test_entropy_decode import _agree
    vals = widths(np.random.default_rng(5), 36 * 1024, 36)
    p = bytes(oracle.encode_mode(M_FOR, vals, oracle.DT_U64, level=1))
    size = 9 + 128 * p[3]
    assert len(p) == 3 + 36 * size
    for k in (0, 17, 32, 35):
        at = 3 + k * size
        for bad in (p[:at] + b"\x41" + p[at + 1:], p[:at], p[:at + 5], p[:at + size - 1]):
            _agree(qb, oracle, stream_of(bad, M_FOR, I64, vals.size))
