"""Decimal containers written limb after limb on the device: limbs of more
blocks than one CTA lays out, columns without a valid value, one value, extreme
significands, and destination buffers that just fit or just do not."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEC128, DEC256 = 6, 7


def column(rng, n, wire, kind):
    nl = 2 if wire == DEC128 else 4
    v = rng.integers(-(1 << 63), 1 << 63, (n, nl), dtype=np.int64)
    if kind == "small":
        v[:, 0] = rng.integers(0, 1 << 40, n)
        v[:, 1:] = 0
    elif kind == "signed":
        v[:, 0] = rng.integers(-10**14, 10**14, n)
        v[:, 1:] = (v[:, :1] >> 63)
    elif kind == "extreme" and n > 2:
        v[n // 2, :] = 0
        v[n // 2, -1] = -(1 << 63)  # the least significand
        v[n // 3, :] = -1
        v[n // 3, -1] = (1 << 63) - 1  # the largest
    return np.ascontiguousarray(v)


@pytest.mark.parametrize("wire", [DEC128, DEC256])
@pytest.mark.parametrize("kind", ["small", "signed", "extreme"])
@pytest.mark.parametrize("n,bs", [(1, None), (257, None), (30_000, 3), (70_001, None)])
def test_containers_match_oracle(qb, oracle, wire, kind, n, bs):
    rng = np.random.default_rng(n + wire)
    v = column(rng, n, wire, kind)
    cfg = qb.Config(level=qb.Level.FAST, block_size=bs)
    for valid in (None, rng.random(n) < 0.7, np.zeros(n, bool), np.arange(n) >= n // 2):
        bm = None if valid is None else np.packbits(valid, bitorder="little")
        want = oracle.compress_column(v, wire, bm, level=1, block_size=bs, scale=4, precision=18)
        got = qb.compress_column(v, bm, cfg, dtype=wire, scale=4, precision=18)
        assert got == want
        d = qb.decompress_column(got)
        exp = v.copy()
        if valid is not None:
            exp[~valid] = 0
        assert d.values.tobytes() == exp.tobytes()


def test_destination_sizes(qb):
    import torch
    v = column(np.random.default_rng(1), 5000, DEC128, "signed")
    stream = qb.compress_column(v, None, qb.Config(level=qb.Level.FAST), dtype=DEC128, scale=4, precision=18)
    d_v = torch.from_numpy(v).cuda()
    for cap in (len(stream) + 100, len(stream), len(stream) - 1, len(stream) // 2, 200, 36, 35, 34, 0):
        d_dst = torch.zeros(len(stream) + 200, dtype=torch.uint8, device="cuda")
        olen, cfg = ctypes.c_size_t(), qb._cfg(qb.Config(level=qb.Level.FAST))
        rc = qb.lib.quoin_b200_compress_column_device(None, DEC128, 5000, d_v.data_ptr(), None, 4, 18,
                                                      ctypes.byref(cfg), d_dst.data_ptr(), cap, ctypes.byref(olen), None)
        got = d_dst.cpu().numpy()
        assert not got[max(cap, 0):].any()  # nothing past the buffer
        if cap >= len(stream):
            assert rc == 0 and olen.value == len(stream) and got[: len(stream)].tobytes() == stream
        else:
            assert rc == -2 and olen.value >= len(stream)
