"""The sort path's workload: what programs have this library do, from a thousand rows to fifty million.

Columns start in HBM (imported from CUDA memory without a copy) unless a case says otherwise, and results
are taken as CUDA arrays through am_export_device, the library's zero-copy interop, so every pass ends with
its result complete. Indices are returned as signed integers of their own width (the same bits).
"""
import ctypes
import json
import math

import numpy as np
import torch

import arrowmetal_b200 as am

DEV = "cuda"
FULL = (-(1 << 63), (1 << 63) - 1)
TYPESTR = {"i": "<i4", "I": "<i4", "l": "<i8", "L": "<i8", "f": "<f4", "g": "<f8"}
WIDTH = {"int32": 4, "float32": 4, "int64": 8, "float64": 8}
FORMAT = {"int32": "i", "float32": "f", "int64": "l", "float64": "g"}


def listed():
    return [
        # The smallest calls, where launches and latency are all there is: one small column's order
        # (the smallest arrays of the segmented workload hold 1e3 rows).
        {"name": "argsort_2k", "op": "argsort", "rows": 2003, "dtype": "int64", "bits": 40, "nulls": 0.1, "descending": False,
         "wide": False},
        # A small served request: ORDER BY over a slice-sized table with two payload columns.
        {"name": "order_by_30k", "op": "order_by", "rows": 30011, "dtype": "int64", "bits": 64, "nulls": 0.0, "descending": False},
        # The single-key scale case: full-range int64, uint64 indices as pyarrow returns them.
        {"name": "argsort_1m", "op": "argsort", "rows": 1000000, "dtype": "int64", "bits": 64, "nulls": 0.0, "descending": False,
         "wide": True},
        # A mid-sized ORDER BY ... DESC on a float64 key (ieee order): the float key is gathered with the payload.
        {"name": "order_by_f64_6m", "op": "order_by", "rows": 6000007, "dtype": "float64", "bits": 64, "nulls": 0.02,
         "descending": True},
        # The benchmark's headline: ORDER BY int64 in [0, 2^40), 10% nulls, payload float64 + int32, 50M rows.
        {"name": "order_by_50m", "op": "order_by", "rows": 50000000, "dtype": "int64", "bits": 40, "nulls": 0.1,
         "descending": False},
        # A sorted copy of a 4-byte column.
        {"name": "sort_f32_20m", "op": "sort", "rows": 20000003, "dtype": "float32", "bits": 32, "nulls": 0.0, "descending": False},
        # The multi-key configuration: int32 Zipf key DESC, float64 key with specials and 5% nulls, all columns taken.
        {"name": "multikey_16m", "op": "multikey", "rows": 16000001, "descending": True},
        # The segmented configuration, one call: int64 and float32 arrays of 1e3 to 1e6 rows.
        {"name": "batch_48", "op": "batch", "arrays": 48, "lo": 1000, "hi": 1000000, "descending": False},
        # ORDER BY ... LIMIT over a large key column.
        {"name": "top_k_30m", "op": "top_k", "rows": 30000000, "dtype": "int64", "bits": 40, "nulls": 0.1, "k": 1000,
         "descending": True},
        # The order of a utf8 column (0 to 24 lowercase letters, 5% nulls) and a payload taken through it.
        {"name": "strings_2m", "op": "strings", "rows": 2000003, "letters": 24, "nulls": 0.05, "descending": False},
        # A sort consumer: Arrow rank ("min" ties) of a key with nulls.
        {"name": "rank_8m", "op": "rank", "rows": 8000009, "dtype": "int64", "bits": 40, "nulls": 0.1, "descending": False},
        # End to end from host buffers, as a query engine's ORDER BY node calls it: import, plan, export.
        {"name": "host_order_by_3m", "op": "host_order_by", "rows": 3000001, "dtype": "int64", "bits": 40, "nulls": 0.1,
         "descending": False},
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n + rng.randint(-9, 9)))


def draw(rng):
    op = rng.choice(["argsort", "argsort", "order_by", "order_by", "order_by", "sort", "multikey", "batch", "top_k",
                     "strings", "rank", "host_order_by"])
    c = {"op": op, "descending": rng.random() < 0.4}
    if op == "batch":
        c.update(arrays=rng.randint(8, 48), lo=1000, hi=_size(rng, 20000, 1000000))
        return c
    if op == "multikey":
        c["rows"] = _size(rng, 100000, 16000000)
        return c
    if op == "strings":
        c.update(rows=_size(rng, 10000, 2000000), letters=rng.choice([8, 16, 24]), nulls=rng.choice([0.0, 0.05]))
        return c
    top = {"argsort": 30000000, "order_by": 50000000, "sort": 40000000, "top_k": 50000000, "rank": 10000000,
           "host_order_by": 4000000}[op]
    low = {"argsort": 1000, "order_by": 1000, "sort": 1000, "top_k": 1000000, "rank": 10000, "host_order_by": 10000}[op]
    c["rows"] = _size(rng, low, top)
    c["dtype"] = rng.choice(["int64", "int64", "int32", "float32", "float64"])
    c["bits"] = 8 * WIDTH[c["dtype"]]
    if c["dtype"] == "int64":
        c["bits"] = rng.choice([40, 64])
    c["nulls"] = rng.choice([0.0, 0.02, 0.1])
    if op == "argsort":
        c["wide"] = rng.random() < 0.3
    if op == "top_k":
        c["k"] = _size(rng, 10, min(1000000, c["rows"] // 8))
    return c


# ---- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 20260906)
    return g


def _values(n, dtype, bits, g):
    if dtype == "float64":
        return torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    if dtype == "float32":
        return torch.randn(n, generator=g, device=DEV, dtype=torch.float32)
    if dtype == "int32":
        return torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    lo, hi = (0, 1 << bits) if bits < 64 else FULL
    return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=torch.int64)


def _bitmap(valid):
    """A packed little-endian validity bitmap of a boolean tensor."""
    n = valid.numel()
    v = torch.zeros((n + 7) // 8 * 8, dtype=torch.uint8, device=DEV)
    v[:n] = valid
    weight = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=DEV)
    return (v.view(-1, 8) * weight).sum(1, dtype=torch.int64).to(torch.uint8)


def _column(t, fmt, valid=None):
    """A CUDA column wrapped without a copy."""
    if valid is None:
        return am.MetalArray.from_device(t.data_ptr(), t.numel(), fmt, keep=t)
    bits = _bitmap(valid)
    nulls = int((~valid).sum())
    torch.cuda.synchronize()
    return am.MetalArray.from_device(t.data_ptr(), t.numel(), fmt, validity_ptr=bits.data_ptr(), null_count=nulls,
                                     keep=(t, bits))


def _valid(n, nulls, g):
    return None if not nulls else torch.rand(n, generator=g, device=DEV) >= nulls


def _key(case, seed):
    g = _gen(seed)
    t = _values(case["rows"], case["dtype"], case["bits"], g)
    return t, _valid(case["rows"], case["nulls"], g), g


def _payload(n, g):
    return (torch.randn(n, generator=g, device=DEV, dtype=torch.float64),
            torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int64).to(torch.int32))


def _multikey(case, seed):
    """key1 int32 from 200 values, bounded Zipf(1.1); key2 float64 N(0, 1e6) with signed zeros, infinities, NaN
    and 5% nulls; payload float64."""
    n, g = case["rows"], _gen(seed)
    p = torch.arange(1, 201, device=DEV, dtype=torch.float64) ** -1.1
    cdf = torch.cumsum(p / p.sum(), 0)
    which = torch.searchsorted(cdf, torch.rand(n, generator=g, device=DEV, dtype=torch.float64)).clamp_(max=199)
    distinct = torch.randint(-(1 << 31), 1 << 31, (200,), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    k2 = torch.randn(n, generator=g, device=DEV, dtype=torch.float64) * 1e6
    u = torch.rand(n, generator=g, device=DEV)
    for value, lo, hi in ((-0.0, 0.0, 0.005), (0.0, 0.005, 0.01), (math.inf, 0.01, 0.015), (-math.inf, 0.015, 0.02),
                          (math.nan, 0.02, 0.03)):
        k2[(u >= lo) & (u < hi)] = value
    valid2 = torch.rand(n, generator=g, device=DEV) >= 0.05
    return distinct[which], k2, valid2, torch.randn(n, generator=g, device=DEV, dtype=torch.float64)


def _lengths(case):
    """The batch's array lengths: log-uniform, the same for every seed (a table's partitions keep their sizes)."""
    rng = np.random.default_rng(case["arrays"])
    return [int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(case["arrays"])]


def _strings(case, seed):
    import pyarrow as pa
    rng = np.random.default_rng(seed)
    n = case["rows"]
    lens = rng.integers(0, case["letters"] + 1, n, dtype=np.int32)
    offsets = np.zeros(n + 1, np.int32)
    np.cumsum(lens, out=offsets[1:])
    data = rng.integers(97, 123, int(offsets[-1]), dtype=np.uint8)
    bitmap, nulls = None, 0
    if case["nulls"]:
        valid = rng.random(n) >= case["nulls"]
        bitmap, nulls = pa.py_buffer(np.packbits(valid, bitorder="little")), int(n - valid.sum())
    return pa.Array.from_buffers(pa.utf8(), n, [bitmap, pa.py_buffer(offsets), pa.py_buffer(data)], null_count=nulls)


def _plan(cols, by, descending):
    exprs = [[c, '(col "%s")' % c] for c in cols]
    keys = [[k, d, {"nulls": "last"}] for k, d in zip(by, descending)]
    return json.dumps({"op": "select", "exprs": exprs, "input": {"op": "sort", "by": keys, "input": {"op": "scan", "source": "t"}}})


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op == "multikey":
        k1, k2, v2, pay = _multikey(case, seed)
        s["source"] = am.PlanSource("t", {"k1": _column(k1, "i"), "k2": _column(k2, "g", v2), "p": _column(pay, "g")})
        s["plan"] = _plan(["k1", "k2", "p"], ["k1", "k2"], [case["descending"], False])
    elif op == "batch":
        g = _gen(seed)
        cols = []
        for i, n in enumerate(_lengths(case)):
            if i % 2 == 0:
                cols.append(_column(_values(n, "int64", 64, g), "l"))
            else:
                cols.append(_column(_values(n, "float32", 32, g), "f", _valid(n, 0.02, g)))
        s["columns"] = cols
    elif op == "strings":
        s["key"] = am.MetalArray.from_arrow(_strings(case, seed))
        s["payload"] = _column(_values(case["rows"], "float64", 64, _gen(seed)), "g")
    else:
        t, valid, g = _key(case, seed)
        fmt = FORMAT[case["dtype"]]
        if op in ("order_by", "host_order_by"):
            p1, p2 = _payload(case["rows"], g)
            s["plan"] = _plan(["k", "p1", "p2"], ["k"], [case["descending"]])
            if op == "order_by":
                s["source"] = am.PlanSource("t", {"k": _column(t, fmt, valid), "p1": _column(p1, "g"), "p2": _column(p2, "i")})
            else:
                s["host"] = {"k": _host_column(t, valid), "p1": _host_column(p1), "p2": _host_column(p2)}
        else:
            s["key"] = _column(t, fmt, valid)
    torch.cuda.synchronize()
    return s


def _host_column(t, valid=None):
    """A pyarrow array over pinned host memory, as an engine's buffer pool hands it out."""
    import pyarrow as pa
    kind = {torch.int32: pa.int32(), torch.int64: pa.int64(), torch.float32: pa.float32(), torch.float64: pa.float64()}[t.dtype]
    host = t.cpu().pin_memory().numpy()
    bits, nulls = None, 0
    if valid is not None:
        b = _bitmap(valid).cpu().pin_memory().numpy()
        bits, nulls = pa.foreign_buffer(b.ctypes.data, b.nbytes, base=b), int((~valid).sum())
    return pa.Array.from_buffers(kind, host.size, [bits, pa.foreign_buffer(host.ctypes.data, host.nbytes, base=host)],
                                 null_count=nulls)


# ---- outputs

class _Exported:
    """One buffer of an exported CUDA array, as torch reads it; holds the export until the tensor goes."""

    def __init__(self, hold, ptr, count, typestr):
        self.hold = hold
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


class _Hold:
    def __init__(self, column):
        self.schema, self.array = am._ArrowSchema(), am._ArrowDeviceArray()
        am._ok(am._lib.am_export_device(column._h, ctypes.addressof(self.schema), ctypes.addressof(self.array)))

    def __del__(self):
        for s in (self.array.array, self.schema):
            if s.release:
                ctypes.CFUNCTYPE(None, ctypes.c_void_p)(s.release)(ctypes.addressof(s))


def _device(column):
    """A result's values as a CUDA tensor, and its validity bitmap's bytes when it has nulls."""
    hold = _Hold(column)
    n = hold.array.array.length
    bufs = ctypes.cast(hold.array.array.buffers, ctypes.POINTER(ctypes.c_void_p * 2)).contents
    values = torch.as_tensor(_Exported(hold, bufs[1], n, TYPESTR[hold.schema.format.decode()]), device=DEV)
    if not bufs[0]:
        return [values]
    return [values, torch.as_tensor(_Exported(hold, bufs[0], (n + 7) // 8, "|u1"), device=DEV)]


def _arrow(column):
    """A host result's buffers: its values, and its validity bitmap's bytes when it has nulls."""
    valid, values = column.buffers()
    n = len(column)
    out = [np.frombuffer(values, dtype=column.type.to_pandas_dtype(), count=n)]
    if column.null_count:
        out.append(np.frombuffer(valid, dtype=np.uint8, count=(n + 7) // 8))
    return out


def run(state):
    c = state["case"]
    op, desc = c["op"], c["descending"]
    if op == "argsort":
        key = state["key"]
        return _device(key.argsort64(descending=desc) if c["wide"] else key.argsort(descending=desc))
    if op == "sort":
        return _device(state["key"].sort(descending=desc))
    if op == "top_k":
        return _device(state["key"].top_k(c["k"], largest=desc))
    if op == "rank":
        return _device(state["key"].rank("descending" if desc else "ascending"))
    if op == "batch":
        return [_device(o) for o in am.argsort_batch(state["columns"], descending=desc)]
    if op == "strings":
        order = state["key"].argsort(descending=desc)
        return [_device(order), _device(state["payload"].take(order))]
    if op == "host_order_by":
        src = am.PlanSource("t", {k: am.MetalArray.from_arrow(v) for k, v in state["host"].items()})
        out = am.run_plan(state["plan"], [src])
        return {k: _arrow(v.to_arrow()) for k, v in out.items()}
    out = am.run_plan(state["plan"], [state["source"]])
    return {k: _device(v) for k, v in out.items()}


# ---- the compulsory work, and the results by plain torch

def _bits(n, nulls):
    return n / 8 if nulls else 0


def work(case):
    """Each input read once and each output written once."""
    op = case["op"]
    if op == "batch":
        lens = _lengths(case)
        return {"bytes": sum((8 + 4) * n if i % 2 == 0 else (4 + 4 + 1 / 8) * n for i, n in enumerate(lens)), "flops": 0}
    n = case["rows"]
    if op == "multikey":
        return {"bytes": 2 * n * (4 + 8 + 8 + 1 / 8), "flops": 0}
    if op == "strings":
        return {"bytes": n * (4 + case["letters"] / 2 + 4 + 8 + 8) + _bits(n, case["nulls"]), "flops": 0}
    key = n * WIDTH[case["dtype"]] + _bits(n, case["nulls"])
    if op == "argsort":
        return {"bytes": key + n * (8 if case["wide"] else 4), "flops": 0}
    if op == "rank":
        return {"bytes": key + n * 4, "flops": 0}
    if op == "top_k":
        return {"bytes": key + case["k"] * 4, "flops": 0}
    if op == "sort":
        return {"bytes": 2 * key, "flops": 0}
    return {"bytes": 2 * (key + n * 12), "flops": 0}


def _order(t, valid, descending):
    """The stable order of a column: values, NaN rows, null rows."""
    rows = torch.arange(t.numel(), device=DEV)
    null = torch.zeros_like(rows, dtype=torch.bool) if valid is None else ~valid
    nan = torch.isnan(t) & ~null if t.is_floating_point() else torch.zeros_like(null)
    vals = rows[~null & ~nan]
    k = t[vals]
    if k.is_floating_point():
        k = k + 0.0            # -0.0 ties 0.0
    return torch.cat([vals[torch.sort(k, stable=True, descending=descending).indices], rows[nan], rows[null]])


def _taken(t, valid, order):
    out = [t[order]]
    if valid is not None and not bool(valid.all()):
        out.append(_bitmap(valid[order]))
    return out


def exact(case, seed):
    """The results by stable sorts of plain torch (whole numbers compare with the start's own)."""
    op, desc = case["op"], case["descending"]
    if op == "order_by":
        t, valid, g = _key(case, seed)
        p1, p2 = _payload(case["rows"], g)
        order = _order(t, valid, desc)
        return {"k": [t[order] if t.is_floating_point() else None] + ([None] if valid is not None and not bool(valid.all()) else []),
                "p1": [p1[order]], "p2": [None]}
    if op == "sort":
        t, valid, _ = _key(case, seed)
        if not t.is_floating_point():
            return None
        return _taken(t, valid, _order(t, valid, desc))
    if op == "multikey":
        k1, k2, v2, pay = _multikey(case, seed)
        order = _order(k2, v2, False)
        order = order[torch.sort(k1[order], stable=True, descending=desc).indices]
        return {"k1": [None], "k2": [k2[order]] + ([None] if not bool(v2.all()) else []), "p": [pay[order]]}
    if op == "strings":
        return None
    return None
