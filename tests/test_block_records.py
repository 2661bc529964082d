"""The encoder's block passes whose results the emission reads from records: bit
packing at every width and byte alignment, ALP-RD dictionaries whose sample
names other left parts than the block's eight most frequent ones, few or very
many left parts, run starts kept for RLE beside small and large dictionaries,
blocks shared by several CTAs.  Streams equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F64, I64, U64 = 0, 1, 2


def check(qb, oracle, v, dt, block_size=None, level=None, modes=None):
    cfg = qb.Config(level=level or qb.Level.FAST, block_size=block_size)
    want = oracle.compress_column(v, dt, None, level=2 if level else 1, block_size=block_size)
    got = qb.compress_column(v, None, cfg, dtype=dt)
    assert got == want
    if modes is not None:
        pos, seen = 16, set()
        while pos < len(got):
            seen.add(got[pos])
            pos += 9 + int.from_bytes(got[pos + 5: pos + 9], "little")
        assert modes & seen, seen


def bits_of(rng, n, w):
    u = rng.integers(0, 1 << 63, n, dtype=np.int64).astype(np.uint64) * np.uint64(2) + rng.integers(0, 2, n).astype(np.uint64)
    u = u >> np.uint64(64 - w) if w else np.zeros(n, np.uint64)
    if w and n > 1:  # both ends of the range in every 1,024
        u[::512], u[1::512] = 0, (1 << w) - 1
    return u


@pytest.mark.parametrize("w", range(0, 65))
def test_pack_widths(qb, oracle, w):
    """FoR sub-blocks of every width, in frames of odd sizes so that their payloads start at every alignment."""
    rng = np.random.default_rng(w)
    for n, bs in ((5 * 1025, 1025), (4 * 1024 + 1023, 2047), (40_000, None)):
        check(qb, oracle, bits_of(rng, n, w) + np.uint64(12345 if w < 60 else 0), U64, block_size=bs)


def left_parts(rng, n, counts, other):
    """f64 lanes with left parts k drawn with the given weights, random low bits, and a share of random left parts."""
    p = np.asarray(counts, float)
    k = rng.choice(p.size, n, p=p / p.sum()).astype(np.uint64)
    bits = (np.uint64(0x3F0) + k) << np.uint64(52) | rng.integers(0, 1 << 52, n, dtype=np.int64).astype(np.uint64)
    m = rng.random(n) < other
    bits[m] = rng.integers(0, 1 << 62, int(m.sum()), dtype=np.int64).astype(np.uint64)
    return bits.view(np.float64)


RD = [
    ("nine_alike", [1.0] * 9, 0.0),
    ("twelve_alike", [1.0] * 12, 0.02),
    ("eight_and_close", [40, 20, 10, 8, 6, 3, 1.1, 1.0, 0.9, 0.85], 0.03),
    ("three", [5, 3, 1], 0.0),
    ("three_and_others", [5, 3, 1], 0.05),
    ("one", [1], 0.01),
    ("many_exceptions", [5, 3, 1], 0.2),
]


@pytest.mark.parametrize("n", [700, 4095, 32_768, 140_000])
@pytest.mark.parametrize("name,counts,other", RD, ids=[c[0] for c in RD])
def test_alprd_dictionaries(qb, oracle, name, counts, other, n):
    rng = np.random.default_rng(n + len(name))
    v = left_parts(rng, n, counts, other)
    check(qb, oracle, v, F64, modes={52, 5, 50, 51, 3})
    check(qb, oracle, v[: n // 2 + 1], F64, block_size=1000)
    if n == 4095:
        check(qb, oracle, v, F64, level=qb.Level.BALANCED_INPOOL)


def test_alprd_is_reached(qb, oracle):
    rng = np.random.default_rng(3)
    check(qb, oracle, left_parts(rng, 40_000, [5, 3, 1], 0.03), F64, modes={52})


@pytest.mark.parametrize("card", [2, 300, 1535, 1537, 6000])
@pytest.mark.parametrize("run", [1, 4, 40])
@pytest.mark.parametrize("n", [3_000, 33_000, 200_001])
def test_runs_and_dictionaries(qb, oracle, card, run, n):
    rng = np.random.default_rng(card + run + n)
    d = rng.integers(0, 1 << 62, card, dtype=np.int64)
    d[0] = -1  # the all-ones key
    lens = rng.geometric(1.0 / run, n)
    v = np.repeat(d[rng.integers(0, card, n)], lens)[:n]
    check(qb, oracle, v, I64)
    check(qb, oracle, v, I64, block_size=50_000)
