"""The rANS coder's four states as four lanes: inputs whose lengths end a step,
an encoder chunk (4,096 bytes) or a batch of the decoder (32 symbols) anywhere,
streams longer than the decoder's 16 KB ring, and symbol tables at the ends of
the frequency range (one symbol of frequency 4096, symbols of frequency 1, 256
equal ones).  The parts are BYTE_TRANSPOSE frames of 8n bytes."""
import numpy as np
import pytest

from test_entropy_decode import _agree
from test_entropy_encode import check

pytestmark = pytest.mark.gpu

M_BYTE_TRANSPOSE, U64, F64 = 11, 2, 0


def one(rng, m):
    return np.full(m, 7, np.uint8)


def rare(rng, m):
    b = np.full(m, 200, np.uint8)
    at = rng.permutation(m)[: m // 500 + 1]
    b[at] = rng.integers(0, 256, at.size)
    return b


def flat(rng, m):
    return rng.integers(0, 256, m).astype(np.uint8)


def skewed(rng, m):
    return (rng.geometric(0.2, m) % 256).astype(np.uint8)


def frame(oracle, data):
    n = data.size // 8
    payload = b"\x02" + oracle.rans_compress(data.tobytes())
    head = b"FCR1" + bytes([2, 0, 16, U64]) + n.to_bytes(8, "little")
    return head + bytes([M_BYTE_TRANSPOSE]) + n.to_bytes(4, "little") + len(payload).to_bytes(4, "little") + payload


@pytest.mark.parametrize("make", [one, rare, flat, skewed], ids=lambda f: f.__name__)
@pytest.mark.parametrize("n", [1, 3, 4, 5, 255, 256, 257, 511, 513, 2049, 4100, 131_072])
def test_decoder_lengths(qb, oracle, make, n):
    data = make(np.random.default_rng(n), 8 * n)
    assert _agree(qb, oracle, frame(oracle, data)) == "ok"


@pytest.mark.parametrize("cut", [1, 2, 8, 40, 5000])
def test_truncated_streams_match_oracle(qb, oracle, cut):
    """A stream that ends early, in the last batch or before."""
    data = skewed(np.random.default_rng(cut), 8 * 3000)
    s = bytearray(frame(oracle, data))
    s = s[: len(s) - cut]
    s[16 + 5: 16 + 9] = (len(s) - 25).to_bytes(4, "little")
    assert _agree(qb, oracle, bytes(s)) == "Truncated"


@pytest.mark.parametrize("n", [1, 2, 5, 63, 511, 513, 1025, 4099])
@pytest.mark.parametrize("bits", [0, 3, 9])
def test_encoder_lengths(qb, oracle, n, bits):
    """Columns whose bytes take the coded forms, at lengths around the encoder's steps and chunks."""
    rng = np.random.default_rng(100 * n + bits)
    planes = rng.geometric(0.3, (n, 8)).astype(np.uint64) % np.uint64(1 << bits if bits else 1)
    v = (planes << (np.uint64(8) * np.arange(8, dtype=np.uint64))).sum(1, dtype=np.uint64)
    check(qb, oracle, v, U64)
    check(qb, oracle, np.round(np.cumsum(rng.standard_normal(n)), 2) + 0.0, F64)
