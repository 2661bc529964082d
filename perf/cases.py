"""What a user of this library has it do, as cases that can be timed.

A case names an operation, the columns it works on and their length:

  op       "compress" / "decompress": device-resident columns, one call per column;
           "compress_batch" / "decompress_queue": many uneven columns in one call;
           "roundtrip": device-resident columns compressed and decompressed again;
           "host_roundtrip": the Python calls on host arrays.
  columns  a column kind, several joined by "+", or "mixed" (`count` columns of
           uneven length up to n, kinds in turn).
  n        values per column.
  null_pct percentage of nulls (0: no validity bitmap).
  level, selection, block_size: the encoder's options.

The columns have the shapes of the benchmark workloads (quoin_b200/synth.py),
generated on the GPU from the seed.  Streams are returned in the buffer they
were written to, zero behind their end, with their lengths; decoded values as
their bit patterns (the codec is lossless, so floats too are compared bit for
bit).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import quoin_b200 as Q

L = Q.lib
P, S = ctypes.c_void_p, ctypes.c_size_t

LEVELS = {"fastest": Q.Level.FASTEST, "fast": Q.Level.FAST, "balanced_inpool": Q.Level.BALANCED_INPOOL}
INTEGER = "timestamps_i64+runs_u64+categories_i32"
FLOAT = "random_walk_f64+sensor_f32+decimal128"
# Column kinds: wire dtype, bytes of a value, and about how many stream bytes a
# valid value takes at Level.FAST (only for work()'s lower bound of a pass).
KINDS = {
    "timestamps_i64": (Q.I64, 8, 2.85),
    "runs_u64": (Q.U64, 8, 3.43),
    "categories_i32": (Q.I32, 4, 0.56),
    "categories_u32": (Q.U32, 4, 0.56),
    "prices_f64": (Q.F64, 8, 7.27),
    "random_walk_f64": (Q.F64, 8, 5.7),
    "sensor_f32": (Q.F32, 4, 1.2),
    "decimal128": (Q.DECIMAL128, 16, 6.0),
}
MIXED = ["prices_f64", "sensor_f32", "timestamps_i64", "runs_u64", "categories_i32", "categories_u32", "decimal128",
         "random_walk_f64"]


class CompressJob(ctypes.Structure):
    """QuoinB200CompressJob (include/quoin.h)."""
    _fields_ = [("wire_dtype", ctypes.c_int32), ("scale", ctypes.c_int8), ("precision", ctypes.c_uint8), ("n", S),
                ("d_values", P), ("d_validity", P), ("d_dst", P), ("dst_cap", S), ("out_len", S),
                ("status", ctypes.c_int32)]


class DecodeJob(ctypes.Structure):
    """QuoinB200DeviceDecodeJob (include/quoin.h)."""
    _fields_ = [("d_src", P), ("src_len", S), ("d_values_out", P), ("values_cap_bytes", S), ("d_validity_out", P),
                ("wire", ctypes.c_int32), ("n", ctypes.c_uint64), ("status", ctypes.c_int32)]


L.quoin_b200_batch_create.restype = P
L.quoin_b200_batch_create.argtypes = [ctypes.c_int]
L.quoin_b200_compress_batch_device.argtypes = [P, ctypes.POINTER(CompressJob), S, ctypes.POINTER(Q._QuoinConfig)]
L.quoin_b200_decompress_queue_device.argtypes = [P, ctypes.POINTER(DecodeJob), S, P]

_batch = None


def batch_handle():
    """The process's batch of eight contexts (a program creates one and keeps it)."""
    global _batch
    if _batch is None:
        _batch = P(L.quoin_b200_batch_create(8))
    return _batch


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def case(op, columns, n, null_pct=0, level="fast", selection="full", block_size=0, count=1, name=None):
    c = {"op": op, "columns": columns, "n": n, "null_pct": null_pct, "level": level, "selection": selection,
         "block_size": block_size, "count": count}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small column of a service's row group, through the Python calls: launches and latency
        case("host_roundtrip", "timestamps_i64", 5_003, 10, name="host_small"),
        # one data page of a table file, written at the fastest level
        case("compress", "categories_u32", 65_537, 20, level="fastest", name="page_compress"),
        # the same size read back
        case("decompress", "timestamps_i64", 65_537, 10, name="page_decompress"),
        # the price column of the benchmark (1,048,576 f64, 3 % exceptions)
        case("compress", "prices_f64", 1_048_576, name="prices_compress"),
        case("decompress", "prices_f64", 1_048_576, name="prices_decompress"),
        # the benchmark's integer columns at full length, 10 % nulls
        case("compress", INTEGER, 67_108_864, 10, name="integer_compress"),
        case("decompress", INTEGER, 67_108_864, 10, name="integer_decompress"),
        # the benchmark's float columns at an ordinary, odd length
        case("compress", FLOAT, 10_000_019, name="float_compress"),
        case("decompress", FLOAT, 10_000_019, name="float_decompress"),
        # a table of uneven columns written and read in one call each
        case("compress_batch", "mixed", 1 << 20, 10, count=192, name="batch_compress"),
        case("decompress_queue", "mixed", 1 << 20, 10, count=192, name="queue_decompress"),
        # the entropy-coded level, written and read back
        case("roundtrip", "sensor_f32+prices_f64", 1_000_003, level="balanced_inpool", name="balanced_roundtrip"),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]; mostly odd and ragged."""
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(sorted(KINDS))
    nulls = rng.choice([0, 0, 5, 10, 20])
    if kind.startswith("runs") or kind.startswith("categ"):
        nulls = rng.choice([0, 10, 20])
    level = rng.choice(["fast", "fast", "fast", "fastest"])
    selection = "sample" if rng.random() < 0.15 else "full"
    block = rng.choice([0, 0, 0, 0, 0, 0, 4096, 65536])
    pick = rng.random()
    if pick < 0.36:
        return case("compress", kind, _size(rng, 1 << 12, 1 << 26), nulls, level, selection, block)
    if pick < 0.72:
        return case("decompress", kind, _size(rng, 1 << 12, 1 << 26), nulls, level, selection, block)
    if pick < 0.80:
        return case("compress_batch", "mixed", _size(rng, 1 << 14, 1 << 20), nulls, level, count=_size(rng, 16, 192))
    if pick < 0.88:
        return case("decompress_queue", "mixed", _size(rng, 1 << 14, 1 << 20), nulls, level, count=_size(rng, 16, 192))
    if pick < 0.94:
        return case("host_roundtrip", kind, _size(rng, 1_000, 200_000), nulls, level)
    return case("roundtrip", kind, _size(rng, 1 << 14, 1 << 20), nulls, "balanced_inpool")


# ---------------------------------------------------------------------------
# Columns
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _timestamps_i64(n, g):
    """ns timestamps from 1.7e18 with steps 1,000,000 + Poisson(5000)."""
    rate = torch.full((n,), 5000.0, dtype=torch.float32, device="cuda")
    d = 1_000_000 + torch.poisson(rate, generator=g).to(torch.int64)
    d[:1] = 0
    return 1_700_000_000_000_000_000 + d.cumsum(0)


def _runs_u64(n, g):
    """base + U[0, 2^k), k ~ U{3..40} redrawn every 1,024 values (held as int64)."""
    base = torch.randint(0, 1 << 40, (1,), device="cuda", generator=g)
    k = torch.randint(3, 41, ((n + 1023) // 1024,), device="cuda", generator=g)
    masks = (torch.ones_like(k) << k) - 1
    u = torch.randint(0, 1 << 62, (n,), device="cuda", generator=g)
    return base + (u & masks.repeat_interleave(1024)[:n])


def _categories_i32(n, g, ncat=64, s=1.1, mean_run=16):
    """Zipf(s) symbols of `ncat` random i32 values in Geometric(1/mean_run) runs."""
    cats = torch.randint(-(1 << 31), 1 << 31, (ncat,), device="cuda", generator=g).to(torch.int32)
    p = torch.arange(1, ncat + 1, dtype=torch.float64, device="cuda") ** -s
    runs = n // mean_run + n // (4 * mean_run) + 64
    sym = torch.multinomial(p, runs, replacement=True, generator=g)
    u = torch.rand(runs, dtype=torch.float64, device="cuda", generator=g)
    lens = (torch.log1p(-u) / math.log1p(-1.0 / mean_run)).floor().to(torch.int64) + 1
    lens[-1] += n  # the last run reaches the end whatever the others drew
    ends = lens.cumsum(0).clamp_(max=n)
    lens = ends - torch.cat([ends.new_zeros(1), ends[:-1]])
    return cats[sym].repeat_interleave(lens, output_size=n)


def _prices_f64(n, g):
    """Two-decimal prices below 10,000, 3 % replaced by random finite bit patterns."""
    v = torch.floor(torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 1e6 + 0.5) / 100.0
    bits = v.view(torch.int64)
    ne = int(0.03 * n)
    at = torch.randperm(n, device="cuda", generator=g)[:ne]
    r = torch.randint(-(1 << 62), 1 << 62, (ne,), device="cuda", generator=g) * 2
    r |= torch.randint(0, 2, (ne,), device="cuda", generator=g)
    r = torch.where((r >> 52) & 0x7FF == 0x7FF, r ^ (1 << 52), r)
    bits[at] = r
    return bits.view(torch.float64)


def _random_walk_f64(n, g):
    """20.0 + a walk of N(0, 1e-3) steps at full precision (steps in units of 2^-48, so that their sum is exact)."""
    step = torch.randn(n, dtype=torch.float64, device="cuda", generator=g) * 1e-3
    k = torch.round(step * 2.0**48).to(torch.int64)
    k[:1] = 0
    return 20.0 + k.cumsum(0).to(torch.float64) * 2.0**-48


def _sensor_f32(n, g):
    """One-decimal readings round(N(25, 5), 1)."""
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g) * 5.0 + 25.0
    return (torch.round(x * 10.0) / 10.0).to(torch.float32)


def _decimal128(n, g):
    """Decimal128(18, 4) significands in [-1e14, 1e14), as (n, 2) limbs."""
    v = torch.randint(-10**14, 10**14, (n,), device="cuda", generator=g)
    return torch.stack([v, v >> 63], dim=1)


def _values(kind, n, g):
    if kind == "categories_u32":
        return _categories_i32(n, g)
    return globals()["_" + kind](n, g).contiguous()


def _bitmap(valid):
    """Arrow LSB-first bitmap of a bool tensor."""
    n = valid.numel()
    padded = torch.zeros((n + 7) // 8 * 8, dtype=torch.uint8, device=valid.device)
    padded[:n] = valid
    weights = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=valid.device)
    return (padded.view(-1, 8) * weights).sum(1, dtype=torch.uint8)


def _bits(t):
    """The values' bit patterns as whole numbers."""
    return t.view(torch.int32 if t.element_size() == 4 else torch.int64)


def _columns(c, seed):
    """[(kind, values, valid bool or None)] of a case."""
    g = _generator(seed)
    if c["columns"] == "mixed":
        want = torch.rand(c["count"], generator=torch.Generator().manual_seed(c["count"])).tolist()
        lo = math.log(1024)
        todo = [(MIXED[i % len(MIXED)], int(math.exp(lo + u * (math.log(c["n"]) - lo)))) for i, u in enumerate(want)]
    else:
        todo = [(kind, c["n"]) for kind in c["columns"].split("+")]
    out = []
    for kind, n in todo:
        v = _values(kind, n, g)
        valid = torch.rand(n, device="cuda", generator=g) >= c["null_pct"] / 100.0 if c["null_pct"] else None
        out.append((kind, v, valid))
    return out


# ---------------------------------------------------------------------------
# Preparation
# ---------------------------------------------------------------------------
def _config(c):
    return Q.Config(level=LEVELS[c["level"]], block_size=c["block_size"] or None,
                    selection=Q.Selection.SAMPLE if c["selection"] == "sample" else Q.Selection.FULL)


def _round16(x):
    return (x + 63) // 64 * 64


def prepare(c, seed):
    """Input columns on the GPU with room for the results; for a decode the
    columns' streams, as the encoder wrote them."""
    st = {"op": c["op"], "cfg": Q._cfg(_config(c)), "config": _config(c), "cols": []}
    cols = _columns(c, seed)
    if c["op"] == "host_roundtrip":
        kind, v, valid = cols[0]
        st["wire"] = KINDS[kind][0]
        st["values"] = v.cpu().numpy()
        st["validity"] = None if valid is None else _bitmap(valid).cpu().numpy()
        st["stream"] = np.zeros(Q._stream_bound(st["wire"], c["n"], valid is not None), dtype=np.uint8)
        return st
    dst_off = out_off = bm_off = 0
    for kind, v, valid in cols:
        wire, width, _ = KINDS[kind]
        n = v.shape[0]
        col = {"wire": wire, "n": n, "values": v, "validity": None if valid is None else _bitmap(valid),
               "scale": 4 if wire == Q.DECIMAL128 else 0, "precision": 18 if wire == Q.DECIMAL128 else 0,
               "cap": Q._stream_bound(wire, n, valid is not None, c["block_size"] or None), "len": 0,
               "dst_off": dst_off, "out_off": out_off, "bm_off": bm_off, "width": width}
        dst_off += _round16(col["cap"])
        out_off += _round16(n * width)
        bm_off += _round16((n + 7) // 8)
        st["cols"].append(col)
    st["dst"] = torch.zeros(dst_off, dtype=torch.uint8, device="cuda")
    decodes = c["op"] != "compress" and c["op"] != "compress_batch"
    if decodes:
        st["out"] = torch.zeros(out_off, dtype=torch.uint8, device="cuda")
        st["bitmaps"] = torch.zeros(bm_off, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    if c["op"] in ("compress_batch", "decompress_queue"):
        st["jobs"] = (CompressJob * len(cols))()
        for j, col in zip(st["jobs"], st["cols"]):
            j.wire_dtype, j.scale, j.precision, j.n = col["wire"], col["scale"], col["precision"], col["n"]
            j.d_values = col["values"].data_ptr()
            j.d_validity = None if col["validity"] is None else col["validity"].data_ptr()
            j.d_dst, j.dst_cap = st["dst"].data_ptr() + col["dst_off"], col["cap"]
    if c["op"] == "decompress":
        _compress(st)
    elif c["op"] == "decompress_queue":
        _compress_batch(st)
        st["decode_jobs"] = (DecodeJob * len(cols))()
        for d, j, col in zip(st["decode_jobs"], st["jobs"], st["cols"]):
            d.d_src, d.src_len = j.d_dst, j.out_len
            d.d_values_out = st["out"].data_ptr() + col["out_off"]
            d.values_cap_bytes = col["n"] * col["width"]
            d.d_validity_out = None if col["validity"] is None else st["bitmaps"].data_ptr() + col["bm_off"]
    if decodes and c["op"] != "roundtrip":  # a reader holds streams, not the values they came from
        for col in st["cols"]:
            col["nullable"] = col["validity"] is not None
            col["values"] = col["validity"] = None
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _compress(st):
    base, cfg = st["dst"].data_ptr(), ctypes.byref(st["cfg"])
    length = S()
    for col in st["cols"]:
        bm = col["validity"]
        Q._check(L.quoin_b200_compress_column_device(
            None, col["wire"], col["n"], col["values"].data_ptr(), None if bm is None else bm.data_ptr(), col["scale"],
            col["precision"], cfg, base + col["dst_off"], col["cap"], ctypes.byref(length), None))
        col["len"] = length.value
    return {"lengths": np.array([col["len"] for col in st["cols"]], dtype=np.int64), "streams": st["dst"]}


def _decompress(st):
    src, out, bitmaps = st["dst"].data_ptr(), st["out"].data_ptr(), st["bitmaps"].data_ptr()
    wire, n = ctypes.c_int32(), ctypes.c_uint64()
    for col in st["cols"]:
        Q._check(L.quoin_b200_decompress_column_device(
            None, src + col["dst_off"], col["len"], out + col["out_off"], col["n"] * col["width"],
            bitmaps + col["bm_off"], ctypes.byref(wire), ctypes.byref(n), None))
    return _decoded(st)


def _decoded(st):
    """The decoded columns (bit patterns) and their bitmaps."""
    vals = [st["out"][col["out_off"]:col["out_off"] + col["n"] * col["width"]].view(
        torch.int32 if col["width"] == 4 else torch.int64) for col in st["cols"]]
    return {"values": vals, "bitmaps": st["bitmaps"]}


def _compress_batch(st):
    Q._check(L.quoin_b200_compress_batch_device(batch_handle(), st["jobs"], len(st["jobs"]), ctypes.byref(st["cfg"])))
    return {"lengths": np.array([j.out_len for j in st["jobs"]], dtype=np.int64), "streams": st["dst"]}


def run(st):
    op = st["op"]
    if op == "compress":
        return _compress(st)
    if op == "decompress":
        return _decompress(st)
    if op == "roundtrip":
        return {"compressed": _compress(st), "decoded": _decompress(st)}
    if op == "compress_batch":
        return _compress_batch(st)
    if op == "decompress_queue":
        Q._check(L.quoin_b200_decompress_queue_device(None, st["decode_jobs"], len(st["decode_jobs"]), None))
        return {"values": st["out"].view(torch.int64), "bitmaps": st["bitmaps"]}
    stream = Q.compress_column(st["values"], st["validity"], st["config"], dtype=st["wire"],
                               scale=4 if st["wire"] == Q.DECIMAL128 else 0,
                               precision=18 if st["wire"] == Q.DECIMAL128 else 0)
    got = Q.decompress_column(stream)
    st["stream"][:len(stream)] = np.frombuffer(stream, dtype=np.uint8)
    return {"length": len(stream), "stream": st["stream"], "values": got.values.view(np.uint8),
            "bitmap": None if got.validity is None else np.frombuffer(got.validity, dtype=np.uint8)}


def exact(c, seed):
    """The decoded values and bitmaps: the inputs with nulls as 0 (streams have
    no such value)."""
    if c["op"] in ("compress", "compress_batch"):
        return None
    cols = _columns(c, seed)
    vals, maps = [], []
    for kind, v, valid in cols:
        b = _bits(v)
        if valid is not None:
            b = torch.where(valid if b.dim() == 1 else valid[:, None], b, torch.zeros_like(b))
        vals.append(b.reshape(-1).contiguous())
        n = v.shape[0]
        m = torch.zeros(_round16((n + 7) // 8), dtype=torch.uint8, device="cuda")
        if valid is not None:
            m[:(n + 7) // 8] = _bitmap(valid)
        maps.append(m)
    if c["op"] == "host_roundtrip":
        n = c["n"]
        return {"length": None, "stream": None, "values": vals[0].view(torch.uint8),
                "bitmap": maps[0][:(n + 7) // 8] if c["null_pct"] else None}
    if c["op"] == "decompress_queue":
        whole = []
        for v in vals:
            b = torch.zeros(_round16(v.numel() * v.element_size()), dtype=torch.uint8, device="cuda")
            b[:v.numel() * v.element_size()] = v.view(torch.uint8)
            whole.append(b)
        return {"values": torch.cat(whole).view(torch.int64), "bitmaps": torch.cat(maps)}
    got = {"values": vals, "bitmaps": torch.cat(maps)}
    return {"compressed": None, "decoded": got} if c["op"] == "roundtrip" else got


def work(c):
    """Bytes of a pass: each value and bitmap once on one side, the stream once on the other."""
    if c["columns"] == "mixed":  # lengths exp(U[ln 1024, ln n]): their mean
        todo = MIXED
        values = c["count"] * (c["n"] - 1024) / math.log(c["n"] / 1024)
    else:
        todo = c["columns"].split("+")
        values = c["n"] * len(todo)
    valid = 1 - c["null_pct"] / 100.0
    one = sum(KINDS[k][1] + KINDS[k][2] * valid for k in todo) / len(todo)
    if c["null_pct"]:
        one += 0.25
    passes = 2 if "roundtrip" in c["op"] else 1
    return {"bytes": passes * values * one, "flops": 0}
