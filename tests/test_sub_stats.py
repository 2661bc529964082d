"""The encoder's sub-block statistics at the ends of their ranges: whole and
partial sub-blocks and windows, mixed signs, wrapping deltas, repeats, every
4- and 8-byte type; streams equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F64, I64, U64, I32, U32, F32 = range(6)
NP = {F64: np.float64, I64: np.int64, U64: np.uint64, I32: np.int32, U32: np.uint32, F32: np.float32}


def values(rng, n, dt, kind):
    w = np.dtype(NP[dt]).itemsize
    u = rng.integers(0, 256, n * w, dtype=np.uint8).view(NP[dt] if dt not in (F64, F32) else {8: np.uint64, 4: np.uint32}[w])
    u = u.copy()
    top = u.dtype.type(np.iinfo(u.dtype).max)
    if kind == "ends":  # the type's least and greatest values side by side
        u[::3], u[1::3] = np.iinfo(u.dtype).min, top
    elif kind == "near_zero":
        u = (rng.integers(-3, 4, n)).astype(np.int64).astype(u.dtype)
    elif kind == "one_sign_change":
        u = (np.arange(n, dtype=np.int64) - n // 2).astype(u.dtype)
    elif kind == "constant":
        u[:] = top
    elif kind == "repeats":
        u = np.repeat(u, 7)[:n].copy()
    elif kind == "stride":
        u = (np.arange(n, dtype=np.int64) * -977 + 5).astype(u.dtype)
    if dt in (F64, F32):
        f = u.view(NP[dt]).copy()
        f[~np.isfinite(f)] = 1.5
        return f if kind != "near_zero" else (rng.integers(-300, 300, n) / 4.0 + 0.0).astype(NP[dt])
    return u


@pytest.mark.parametrize("dt", range(6))
@pytest.mark.parametrize("kind", ["random", "ends", "near_zero", "one_sign_change", "constant", "repeats", "stride"])
def test_streams_match_oracle(qb, oracle, dt, kind):
    if dt in (F64, F32) and kind == "ends":
        return  # integer ranges; a float's least and greatest bit patterns are no numbers
    rng = np.random.default_rng(dt * 10 + len(kind))
    for n in (1, 2, 1023, 1024, 1025, 8 * 1024, 32_768, 32_769, 70_001):
        v = values(rng, n, dt, kind)
        for bs in (None, 1024, 5000):
            for level in (0, 1):
                cfg = qb.Config(level=qb.Level(level), block_size=bs)
                assert qb.compress_column(v, None, cfg, dtype=dt) == oracle.compress_column(
                    v, dt, None, level=level, block_size=bs), (n, bs, level)
