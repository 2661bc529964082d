"""Batch calls whose columns are compressed in groups (one launch per kernel
for many columns): every stream, length and status is the single-column
call's.  All wire types, bitmaps around the one-CTA stretch of 262,144
positions and with RAW and RLE blobs, all and no nulls, fixed block sizes,
every level, destinations that are too small, columns at and past the longest
that a group takes, and more values than one group holds."""
import ctypes

import numpy as np
import pytest

from test_batch import CompressJob, P, batch_api  # noqa: F401

pytestmark = pytest.mark.gpu

DTYPES = list(range(8))  # f64 i64 u64 i32 u32 f32 decimal128 decimal256
NULLS = ["none", "all_valid", "all_null", "runs", "alternate", "random", "last"]


def column(rng, dt, n, nulls):
    if dt in (0, 5):
        v = np.floor(rng.random(n) * 1e5) / 100 if rng.random() < 0.7 else rng.standard_normal(n)
        v = v.astype(np.float64 if dt == 0 else np.float32)
    elif dt >= 6:
        v = np.zeros((n, 2 if dt == 6 else 4), np.uint64)
        v[:, 0] = rng.integers(0, 1 << 40, n, dtype=np.uint64)
        v[rng.random(n) < 0.3] = np.uint64((1 << 64) - 12345)  # small negatives
    else:
        base = np.cumsum(rng.integers(0, 99, n)) if rng.random() < 0.5 else rng.integers(0, 7, n) * 1000
        v = base.astype({1: np.int64, 2: np.uint64, 3: np.int32, 4: np.uint32}[dt])
    pos = np.arange(n)
    valid = {"none": None, "all_valid": pos >= 0, "all_null": pos < 0, "runs": (pos // 500) % 2 == 1,
             "alternate": pos % 2 == 0, "random": rng.random(n) < 0.9, "last": pos == n - 1}[nulls]
    return v, None if valid is None else np.packbits(valid, bitorder="little")


def check(qb, L, cols, cfg, caps=None, workers=3):
    import torch
    c = qb._cfg(cfg)
    jobs = (CompressJob * len(cols))()
    keep = []
    for j, (dt, v, bm) in enumerate(cols):
        n = len(v)
        dv = torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1).copy()).cuda()
        db = None if bm is None else torch.from_numpy(bm.copy()).cuda()
        bound = qb._stream_bound(dt, n, bm is not None) + 9 * (n // max(cfg.block_size or n, 1) + 1)
        want_cap = caps[j] if caps else bound
        one, got = (torch.zeros(bound + 64, dtype=torch.uint8, device="cuda") for _ in range(2))
        sc, pr = (4, 18) if dt >= 6 else (0, 0)
        olen = ctypes.c_size_t()
        ptr = None if db is None else db.data_ptr()
        rc = qb.lib.quoin_b200_compress_column_device(None, dt, n, dv.data_ptr(), ptr, sc, pr, ctypes.byref(c),
                                                      one.data_ptr(), want_cap, ctypes.byref(olen), None)
        jobs[j] = CompressJob(dt, sc, pr, n, dv.data_ptr(), ptr, got.data_ptr(), want_cap, 0, 99)
        keep.append((dv, db, one, got, rc, olen.value))
    torch.cuda.synchronize()
    b = P(L.quoin_b200_batch_create(workers))
    try:
        for _ in range(2):  # the second call reuses the first's memory
            rc = L.quoin_b200_compress_batch_device(b, jobs, len(cols), ctypes.byref(c))
            assert rc == next((k[4] for k in keep if k[4]), 0)
            for j, (dv, db, one, got, rc1, n1) in enumerate(keep):
                what = (j, cols[j][0], len(cols[j][1]))
                assert (jobs[j].status, jobs[j].out_len) == (rc1, n1), what
                if rc1 == 0:
                    assert torch.equal(one[:n1], got[:n1]), what
                assert not got[jobs[j].dst_cap:].any(), what
    finally:
        L.quoin_b200_batch_free(b)


@pytest.mark.parametrize("level", ["FASTEST", "FAST", "SAMPLE", "BALANCED_INPOOL"])
@pytest.mark.parametrize("bs", [None, 700, 200_000])
def test_types_and_bitmaps(qb, batch_api, level, bs):  # noqa: F811
    rng = np.random.default_rng(len(level) + (bs or 0))
    cfg = qb.Config(level=qb.Level.FAST, block_size=bs, selection=qb.Selection.SAMPLE) if level == "SAMPLE" else \
        qb.Config(level=getattr(qb.Level, level), block_size=bs)
    cols = []
    for i, dt in enumerate(DTYPES * 3):
        for k, nulls in enumerate(NULLS):
            n = [1, 33, 1024, 5000, 32_769, 70_001][(i * 5 + k) % 6]
            cols.append((dt, *column(rng, dt, n, nulls)))
    check(qb, batch_api, cols, cfg)


@pytest.mark.parametrize("n", [262_144, 262_145, 524_289, 1 << 20, (1 << 20) + 1])
def test_long_bitmaps(qb, batch_api, n):  # noqa: F811
    rng = np.random.default_rng(n)
    cols = [(dt, *column(rng, dt, n, nulls)) for dt, nulls in zip([0, 1, 3, 6, 7, 5, 2], NULLS)]
    cols += [(3, *column(rng, 3, n, nulls)) for nulls in NULLS]
    check(qb, batch_api, cols, qb.Config(level=qb.Level.FAST))


def test_small_destinations(qb, batch_api):  # noqa: F811
    rng = np.random.default_rng(2)
    cols, caps = [], []
    for dt in (0, 1, 3, 6, 7):
        for nulls in ("none", "random", "all_null"):
            v, bm = column(rng, dt, 3000, nulls)
            for cap in (0, 15, 16, 17, 50, 51, 60, 400, 430, 480, 1200, 5000, 9000):
                cols.append((dt, v, bm))
                caps.append(cap)
    check(qb, batch_api, cols, qb.Config(level=qb.Level.FAST), caps)


def test_many_groups(qb, batch_api):  # noqa: F811
    rng = np.random.default_rng(3)
    cols = [(DTYPES[i % 8], *column(rng, DTYPES[i % 8], int(rng.integers(1, 400_000)), NULLS[i % 7])) for i in range(60)]
    check(qb, batch_api, cols, qb.Config(level=qb.Level.FAST), workers=2)
