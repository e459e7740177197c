"""The bucket sort of one key (bucket_sort.cu) where it can go wrong: the smallest columns, rows around a
tile and around the sample size (up to which one launch plans, counts and moves), one and two levels of bins, both key widths, keys spread
evenly (equal cuts) and unevenly (cells), buckets of one repeated key (the slow form, and the digit
passes when none can hold it), and null and NaN rows; each against the oracle's stable order, with and
without payload columns beside the key."""
import numpy as np
import pyarrow as pa
import pytest

pytestmark = pytest.mark.gpu

TILE = 512 * 7
CASES = [(1, "even"), (33, "normal"), (2003, "even"), (2048, "repeats"), (4097, "even"), (TILE * 2 - 1, "normal"), (TILE * 2 + 1, "normal32"), (65535, "even32"), (65536, "normal"),
         (65537, "repeats"), (200_003, "clusters"), (700_001, "even"), (1_500_000, "normal32"), (1_500_001, "repeats"),
         (3_000_017, "normal"), (3_000_017, "one_value"), (5_000_011, "even"), (2_000_003, "narrow"), (2_000_003, "exponential")]


def keys(kind, n, rng):
    if kind == "even":
        return rng.integers(0, 2**40, n, dtype=np.int64)
    if kind == "even32":
        return rng.integers(-2**31, 2**31, n).astype(np.int32)
    if kind in ("normal", "normal32"):
        v = rng.standard_normal(n).astype(np.float32 if kind == "normal32" else np.float64)
        v[rng.random(n) < 0.01] = np.nan
        v[rng.random(n) < 0.0005] = -0.0
        v[rng.random(n) < 0.0005] = 0.0
        return v
    if kind == "repeats":                       # 3,000 rows a value: more than the fast form takes
        return rng.integers(0, max(2, n // 3000), n).astype(np.int64) * 7919
    if kind == "clusters":                      # a few values repeated about a thousand times among others
        v = rng.integers(0, 2**50, n, dtype=np.int64)
        hit = rng.random(n) < 0.2
        v[hit] = rng.integers(0, 40, int(hit.sum())) * 2**43 + 5
        return v
    if kind == "one_value":                     # no bucket holds it: the digit passes
        v = rng.integers(0, 2**40, n, dtype=np.int64)
        v[rng.random(n) < 0.3] = 123_456_789_012
        return v
    if kind == "narrow":
        return rng.integers(-100, 100, n).astype(np.int16)
    return (rng.exponential(1e5, n)).astype(np.int64)


@pytest.mark.parametrize("n,kind", CASES)
def test_against_the_oracle(am, oracle, n, kind):
    rng = np.random.default_rng(n + len(kind))
    v = keys(kind, n, rng)
    for nulls, desc, place, order in ((0.0, False, "at_end", "ieee"), (0.1, True, "at_start", "nan_largest"),
                                      (0.3, False, "at_start", "ieee"), (0.02, True, "at_end", "total")):
        arr = pa.array(v, mask=rng.random(n) < nulls if nulls else None, from_pandas=False)
        want = oracle.argsort(arr, desc, place, order, threads=4)
        m = am.MetalArray.from_arrow(arr)
        assert np.array_equal(m.argsort(desc, place, order).to_arrow().to_numpy(), want)
        assert np.array_equal(m.argsort64(desc, place, order).to_arrow().to_numpy(), want)
        p1, p2 = rng.standard_normal(n), rng.integers(-2**31, 2**31, n).astype(np.int32)
        src = am.PlanSource("t", {"k": m, "a": pa.array(p1), "b": pa.array(p2)})
        by = [["k", desc, {"nulls": "first" if place == "at_start" else "last", "float_order": order}]]
        out = am.run_plan({"op": "sort", "by": by, "input": {"op": "scan", "source": "t"}}, [src])
        assert np.array_equal(out["a"].to_arrow().to_numpy(), p1[want])
        assert np.array_equal(out["b"].to_arrow().to_numpy(), p2[want])
        got, sorted_copy, exp = out["k"].to_arrow(), m.sort(desc, place, order).to_arrow(), arr.take(pa.array(want))
        valid = np.asarray(exp.is_valid())
        width = arr.type.bit_width // 8
        bits = [np.frombuffer(a.buffers()[1], np.uint8, n * width).reshape(n, width)[valid] for a in (got, sorted_copy, exp)]
        assert np.array_equal(np.asarray(got.is_valid()), valid) and np.array_equal(np.asarray(sorted_copy.is_valid()), valid)
        assert np.array_equal(bits[0], bits[2]) and np.array_equal(bits[1], bits[2])


@pytest.mark.parametrize("offset", [1, 32, 37])
def test_sliced_columns(am, oracle, offset):
    # A validity bitmap that starts inside a word, and values off their alignment.
    rng = np.random.default_rng(offset)
    base = pa.array(rng.integers(0, 2**40, 100_000), mask=rng.random(100_000) < 0.2)
    part = base.slice(offset, 90_001)
    m = am.MetalArray.from_arrow(base).slice(offset, 90_001)
    assert np.array_equal(m.argsort().to_arrow().to_numpy(), oracle.argsort(part))


@pytest.mark.parametrize("kind", ["normal", "one_value", "repeats"])
def test_concurrent_threads(am, oracle, kind):
    # Each thread sorts on its own stream, with its own scratch: by buckets, by the digit passes of one launch behind
    # them (with barriers over the grid), and by buckets of repeated keys.
    import threading
    rng = np.random.default_rng(3)
    arrays = [pa.array(keys(kind, 300_000 + 1000 * i, rng), from_pandas=False) for i in range(4)]
    want = [oracle.argsort(a) for a in arrays]
    bad = []

    def work(i):
        m = am.MetalArray.from_arrow(arrays[i])
        for _ in range(20):
            if not np.array_equal(m.argsort().to_arrow().to_numpy(), want[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def sampled_rows(n):
    """The rows that a sort of more than 65,536 looks at first: one of each 65,536th part, at a mixed offset."""
    j = np.arange(65_536, dtype=np.uint64)
    lo, hi = j * n // 65_536, (j + 1) * n // 65_536
    mask = np.uint64(0xFFFFFFFF)
    h = (j * 2654435761) & mask
    h ^= h >> np.uint64(15)
    h = (h * 2246822519) & mask
    h ^= h >> np.uint64(13)
    return (lo + ((h * (hi - lo)) >> np.uint64(32))).astype(np.int64)


@pytest.mark.parametrize("n", [70_001, 1_000_003, 5_000_011])
@pytest.mark.parametrize("kind", ["sorted", "reversed", "pipe", "stride", "sample_apart", "sample_below"])
def test_orders_that_mislead_the_sample(am, oracle, n, kind):
    # Columns already in order, periods of the sample's stride, and rows that lie outside the sampled keys' range
    # (all of them beside one key, or all above it).
    rng = np.random.default_rng(n)
    v = rng.integers(0, 2**40, n)
    if kind == "sorted":
        v = np.sort(v)
    elif kind == "reversed":
        v = np.sort(v)[::-1].copy()
    elif kind == "pipe":
        v = np.abs(np.arange(n) - n // 2) * 2**18
    elif kind == "stride":
        v = (np.arange(n) % max(2, n // 65_536)) * 2**30 + rng.integers(0, 2**20, n)
    elif kind == "sample_apart":
        v[sampled_rows(n)] = 2**39 + rng.integers(0, 50, 65_536)
    else:
        v += 2**41
        v[sampled_rows(n)] = rng.integers(0, 2**30, 65_536)
    arr = pa.array(v)
    m = am.MetalArray.from_arrow(arr)
    for desc in (False, True):
        want = oracle.argsort(arr, desc, threads=4)
        assert np.array_equal(m.argsort(desc).to_arrow().to_numpy(), want)
        assert np.array_equal(m.sort(desc).to_arrow().to_numpy(), v[want])


@pytest.mark.parametrize("n", [10_000_019, 62_914_560, 62_914_561])
def test_ranks_of_large_columns(am, oracle, n):
    # Both sides of the rows up to which ranks leave the buckets.
    rng = np.random.default_rng(n)
    v = rng.integers(0, 2**40, n) if n % 2 else rng.integers(0, n // 50, n) * 7919
    arr = pa.array(v)
    order = oracle.argsort(arr, threads=8)
    key = v[order]
    start = np.ones(n, bool)
    start[1:] = key[1:] != key[:-1]
    first = np.flatnonzero(start)[np.cumsum(start) - 1]
    ranks = np.empty(n, np.int64)
    ranks[order] = first + 1
    assert np.array_equal(am.MetalArray.from_arrow(arr).rank().to_arrow().to_numpy(), ranks)


@pytest.mark.parametrize("kind,order", [("normal", "ieee"), ("normal32", "nan_largest"), ("normal32", "ieee"), ("one_value", "ieee")])
@pytest.mark.parametrize("n", [3000, 300_007])
def test_rebuilt_float_keys_keep_their_bits(am, n, kind, order):
    # Zeros of both signs, NaN payloads and the bits under null rows come out as a take would copy them,
    # from the buckets and (a value too often repeated) from the digit passes.
    rng = np.random.default_rng(n)
    v = keys("normal" if kind == "one_value" else kind, n, rng)
    if kind == "one_value":
        v[rng.random(n) < 0.5] = -0.0
        v[rng.random(n) < 0.3] = 0.0
    bits = v.view(np.uint32 if v.dtype.itemsize == 4 else np.uint64)
    bits[np.isnan(v)] |= rng.integers(0, 1000, int(np.isnan(v).sum())).astype(bits.dtype)
    arr = pa.array(v, mask=rng.random(n) < 0.1, from_pandas=False)
    m = am.MetalArray.from_arrow(arr)
    p = am.MetalArray.from_arrow(pa.array(np.arange(n, dtype=np.int64)))
    for desc, place in ((False, "at_end"), (True, "at_start")):
        want = m.take(m.argsort(desc, place, order)).to_arrow()
        src = am.PlanSource("t", {"k": m, "p": p})
        by = [["k", desc, {"nulls": "first" if place == "at_start" else "last", "float_order": order}]]
        out = am.run_plan({"op": "sort", "by": by, "input": {"op": "scan", "source": "t"}}, [src])["k"].to_arrow()
        for got in (m.sort(desc, place, order).to_arrow(), out):
            assert got.null_count == want.null_count
            assert got.buffers()[1].to_pybytes()[:n * v.dtype.itemsize] == want.buffers()[1].to_pybytes()[:n * v.dtype.itemsize]
            assert np.array_equal(np.asarray(got.is_valid()), np.asarray(want.is_valid()))


@pytest.mark.parametrize("n,k,kind", [(2**19, 1, "even"), (600_011, 1000, "normal"), (2_000_003, 20_000, "even32"),
                                      (3_000_017, 500, "one_value"), (600_011, 30_000, "normal32"), (700_001, 5000, "narrow")])
def test_first_rows_are_the_sorts_first(am, n, k, kind):
    # The sampled limit and its fallbacks: few and many rows wanted, equal keys at the limit, nulls first.
    rng = np.random.default_rng(n + k)
    v = keys(kind, n, rng)
    if kind == "one_value":
        v[v == 123_456_789_012] = 0
    for nulls in (0.0, 0.3):
        m = am.MetalArray.from_arrow(pa.array(v, mask=rng.random(n) < nulls if nulls else None, from_pandas=False))
        for largest, place, order in ((True, "at_end", "ieee"), (False, "at_start", "nan_largest"), (False, "at_end", "total")):
            want = m.argsort(largest, place, order).to_arrow().to_numpy()[:k]
            got = m.top_k(k, largest, place, order).to_arrow().to_numpy()
            assert np.array_equal(got, want), (nulls, largest, place, order)


def repeated(kind, n, rng):
    """Keys that repeat: `kind` rows a value; two values side by side among distinct keys; sorted runs; a few
    values far apart on a logarithmic scale; floats with both zeros and NaN."""
    if isinstance(kind, int):
        m = max(1, n // kind)
        return rng.integers(0, 2**40, m)[rng.integers(0, m, n)]
    if kind == "two_close":
        v = rng.integers(0, 2**40, n)
        hit = rng.random(n) < 0.1
        v[hit] = rng.choice([2**39, 2**39 + 1], int(hit.sum()))
        return v
    if kind == "runs":
        return np.sort(rng.integers(0, max(1, n // 700), n)) * 2**33
    if kind == "log":
        v = np.exp2(rng.integers(0, 62, n)).astype(np.int64)
        return v + rng.integers(0, 3, n)
    if kind == "int32":
        m = max(1, n // 40)
        return rng.integers(-2**31, 2**31, m).astype(np.int32)[rng.integers(0, m, n)]
    v = rng.standard_normal(max(1, n // 100))[rng.integers(0, max(1, n // 100), n)]
    for value in (0.0, -0.0, np.nan, np.inf):
        v[rng.random(n) < 0.003] = value
    return v


@pytest.mark.parametrize("n", [33, 2003, 30_011, 65_537, 1_500_001])
@pytest.mark.parametrize("kind", [12, 30, 100, 700, 2500, 9000, "two_close", "runs", "log", "int32", "float"])
def test_keys_that_repeat(am, oracle, n, kind):
    # Bins of repeated keys, several of them in a bin, and buckets larger than a CTA orders at once: the order,
    # records, the sorted key column and the ranks.
    rng = np.random.default_rng(n + len(str(kind)))
    v = repeated(kind, n, rng)
    for nulls, desc, place in ((0.0, False, "at_end"), (0.1, True, "at_start")):
        arr = pa.array(v, mask=rng.random(n) < nulls if nulls else None, from_pandas=False)
        want = oracle.argsort(arr, desc, place, "ieee", threads=4)
        m = am.MetalArray.from_arrow(arr)
        assert np.array_equal(m.argsort(desc, place).to_arrow().to_numpy(), want)
        p1, p2 = rng.standard_normal(n), rng.integers(-2**31, 2**31, n).astype(np.int32)
        src = am.PlanSource("t", {"k": m, "a": pa.array(p1), "b": pa.array(p2)})
        by = [["k", desc, {"nulls": "first" if place == "at_start" else "last"}]]
        out = am.run_plan({"op": "sort", "by": by, "input": {"op": "scan", "source": "t"}}, [src])
        assert np.array_equal(out["a"].to_arrow().to_numpy(), p1[want])
        assert np.array_equal(out["b"].to_arrow().to_numpy(), p2[want])
        exp = arr.take(pa.array(want))
        valid = np.asarray(exp.is_valid())
        width = arr.type.bit_width // 8
        for got in (m.sort(desc, place).to_arrow(), out["k"].to_arrow()):
            bits = [np.frombuffer(a.buffers()[1], np.uint8, n * width).reshape(n, width)[valid] for a in (got, exp)]
            assert np.array_equal(np.asarray(got.is_valid()), valid) and np.array_equal(bits[0], bits[1])
        # Ranks: runs of equal rows in order (null and NaN rows are equals of one another).
        key, other = v[want], ~valid | (np.isnan(v[want]) if v.dtype.kind == "f" else False)
        start = np.ones(n, bool)
        start[1:] = (other[1:] != other[:-1]) | (~other[1:] & (key[1:] != key[:-1]))
        run, first = np.cumsum(start) - 1, np.flatnonzero(start)
        last = np.append(first[1:], n)
        for tiebreaker, pos in (("min", first[run] + 1), ("max", last[run]), ("first", np.arange(1, n + 1))):
            ranks = np.empty(n, np.int64)
            ranks[want] = pos
            got = m.rank("descending" if desc else "ascending", place, tiebreaker).to_arrow().to_numpy()
            assert np.array_equal(got, ranks), tiebreaker
