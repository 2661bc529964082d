"""Short columns: the encoder's start of a nullable stream without the host's
knowledge of the valid count, and the decoder's walk of a few frames with the
tables made in one launch.  Bitmap lengths around words, CTAs and the short
form's limit; no, few, alternating and all nulls (RAW and RLE blobs); frame
counts around the walk's limit; destinations that just fit; streams cut
anywhere."""
import ctypes

import numpy as np
import pytest

from test_device_reader import check_same, device_decode, host_decode, host_parse

pytestmark = pytest.mark.gpu

F64, I64, I32 = 0, 1, 3


def bitmaps(rng, n):
    yield "all", np.ones(n, bool)
    yield "none", np.zeros(n, bool)
    yield "one_null", np.arange(n) != n // 2
    yield "one_valid", np.arange(n) == n - 1
    yield "runs", (np.arange(n) // 300) % 2 == 1
    yield "alternate", np.arange(n) % 2 == 0
    yield "random", rng.random(n) < 0.8


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 32_767, 32_768, 32_769, 65_537, 262_144, 262_145])
@pytest.mark.parametrize("dt", [I64, I32, F64])
def test_nullable_columns_match_oracle(qb, oracle, n, dt):
    rng = np.random.default_rng(n + dt)
    v = {I64: np.cumsum(rng.integers(0, 99, n)), I32: rng.integers(-5, 6, n).astype(np.int32),
         F64: np.floor(rng.random(n) * 1e5) / 100}[dt]
    for name, valid in bitmaps(rng, n):
        bm = np.packbits(valid, bitorder="little")
        for bs in ((None, 700) if n < 70_000 else (None,)):
            want = oracle.compress_column(v, dt, bm, level=1, block_size=bs)
            got = qb.compress_column(v, bm, qb.Config(level=qb.Level.FAST, block_size=bs), dtype=dt)
            assert got == want, (name, bs)
            exp = v.copy()
            exp[~valid] = 0
            check_same(qb, got, device_read=False)
            assert np.asarray(qb.decompress_column(got).values).tobytes() == exp.tobytes(), (name, bs)


@pytest.mark.parametrize("frames", [1, 2, 47, 48, 49, 96, 97, 98, 400])
def test_frame_counts(qb, oracle, frames):
    rng = np.random.default_rng(frames)
    n = frames * 130 - 7
    for v, dt in ((np.cumsum(rng.integers(0, 1 << 20, n)), I64), (np.repeat(rng.integers(0, 9, n), 3)[:n], I64),
                  (np.floor(rng.random(n) * 1e4) / 100, F64)):
        for bm in (None, np.packbits(rng.random(n) < 0.9, bitorder="little")):
            s = oracle.compress_column(v, dt, bm, level=1, block_size=130)
            check_same(qb, s, device_read=True)


def test_destination_sizes(qb):
    import torch
    rng = np.random.default_rng(1)
    n = 5000
    v, valid = np.cumsum(rng.integers(0, 99, n)), rng.random(n) < 0.8
    bm = np.packbits(valid, bitorder="little")
    stream = qb.compress_column(v, bm, qb.Config(level=qb.Level.FAST), dtype=I64)
    d_v, d_bm = torch.from_numpy(v).cuda(), torch.from_numpy(bm).cuda()
    for cap in (len(stream) + 9, len(stream), len(stream) - 1, 700, 669, 668, 642, 641, 100, 16, 15, 0):
        d_dst = torch.zeros(len(stream) + 200, dtype=torch.uint8, device="cuda")
        olen, cfg = ctypes.c_size_t(), qb._cfg(qb.Config(level=qb.Level.FAST))
        rc = qb.lib.quoin_b200_compress_column_device(None, I64, n, d_v.data_ptr(), d_bm.data_ptr(), 0, 0,
                                                      ctypes.byref(cfg), d_dst.data_ptr(), cap, ctypes.byref(olen), None)
        got = d_dst.cpu().numpy()
        assert not got[cap:].any()
        if cap >= len(stream):
            assert rc == 0 and got[: olen.value].tobytes() == stream
        else:
            assert rc == -2 and olen.value >= len(stream)


def test_cut_streams_report_as_the_host_reader(qb, oracle):
    rng = np.random.default_rng(4)
    n = 3000
    v = np.floor(rng.random(n) * 1e4) / 100
    bm = np.packbits(rng.random(n) < 0.9, bitorder="little")
    s = oracle.compress_column(v, F64, bm, level=1, block_size=1000)
    for cut in list(range(0, 60, 7)) + list(rng.integers(60, len(s), 40)):
        b = s[: int(cut)]
        rc, _, _ = host_parse(qb, b)
        want = host_decode(qb, b, F64, n)[0] if rc == 0 else rc
        assert device_decode(qb, b, 8 * n)[0] == want, cut
