"""The splitting sort of long arrays and long rows (csrc/b2s_split.cuh) against NumPy's stable sort, bit for bit: one
input per mapping of keys to cells, per edge of its tables and per way out of it."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _values(how: str, n: int, dtype: np.dtype, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    if dtype.kind == "f":
        if how == "normal":
            a = rng.standard_normal(n)
        elif how == "nans":          # three values in a hundred, and one pattern of them
            a = rng.standard_normal(n)
            a[rng.integers(0, n, n // 33)] = np.nan
        elif how == "patterns":      # zeros of both signs, several NaN patterns: input order among equal images
            a = np.round(rng.standard_normal(n) * 4) / 4
            a = a.astype(dtype)
            u = a.view(f"u{dtype.itemsize}")
            at = rng.integers(0, n, n // 50)
            u[at] = np.array(np.nan, dtype).view(u.dtype) + (at % 5).astype(u.dtype)
            return a
        elif how == "wide":          # every magnitude, and infinities
            a = np.exp2(rng.uniform(-140 if dtype.itemsize == 4 else -1000, 120, n)) * rng.choice([-1.0, 1.0], n)
            a[rng.integers(0, n, 9)] = np.inf
            a[rng.integers(0, n, 9)] = -np.inf
        elif how == "spike":         # half of the keys are one value, the others around it
            a = np.where(rng.random(n) < 0.5, 0.75, rng.standard_normal(n))
        elif how == "few":           # values far apart, each with many copies
            a = rng.integers(0, 37, n) * 1.37e5
        elif how == "crowded":       # two clusters that a linear function does not take apart
            a = np.where(rng.random(n) < 0.5, 1.0, 1e30) * (1 + rng.random(n) * 1e-4)
        elif how == "equal":
            a = np.full(n, 2.5)
        else:
            a = np.full(n, np.nan)
        return a.astype(dtype)
    info = np.iinfo(dtype)
    if how == "normal":
        return rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True)
    if how == "nans":                # the ends of the range
        a = rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True)
        a[rng.integers(0, n, n // 30)] = info.max
        a[rng.integers(0, n, n // 30)] = info.min
        return a
    if how == "patterns":            # Zipf: crowded at the lower end, the largest value often
        return np.minimum(rng.zipf(1.2, n).astype(np.float64), min(info.max, 2**40 - 1)).astype(dtype)
    if how == "wide":
        return np.exp2(rng.uniform(0, 8 * dtype.itemsize - 2, n)).astype(dtype)
    if how == "spike":
        return np.where(rng.random(n) < 0.5, 12345, rng.integers(0, 2**31 - 1, n)).astype(dtype)
    if how == "few":
        return (rng.integers(0, 100, n) * (1 if seed % 2 else info.max // 128)).astype(dtype)
    if how == "crowded":             # almost in order
        a = np.arange(n).astype(dtype)
        i, j = rng.integers(0, n, n // 100), rng.integers(0, n, n // 100)
        a[i], a[j] = a[j], a[i]
        return a
    return np.full(n, 7 if how == "equal" else info.max, dtype)


OPEN, SPLIT, RADIX, LATE = range(4)   # who sorted: nobody tried, the splits, the passes since the sample, since later


def _device(a: np.ndarray) -> torch.Tensor:
    d = torch.from_numpy(a.view(f"i{a.dtype.itemsize}") if a.dtype.kind == "u" else a).cuda()
    return d.view({"u4": torch.uint32, "u8": torch.uint64}[a.dtype.str[1:]]) if a.dtype.kind == "u" else d


def _route() -> int:
    """Of the last sort of this thread: a word of the control block at the head of its workspace."""
    from cupynumeric_b200.runtime import runtime

    return int(runtime.workspace(1)[48:52].view(torch.int32).item())


def _check(a: np.ndarray, op: str) -> int:
    import cupynumeric_b200 as num

    d = _device(a)
    order = np.argsort(a, axis=-1, kind="stable")
    if op == "argsort":
        got = num.argsort(num.array(d), axis=-1, kind="stable").to_numpy()
        assert np.array_equal(got, order)
    else:
        got  = num.sort(num.array(d), axis=-1).to_numpy()
        want = np.take_along_axis(a, order, axis=-1)
        assert np.array_equal(got.view(f"u{a.dtype.itemsize}"), want.view(f"u{a.dtype.itemsize}"))
    return _route()


HOW = ["normal", "nans", "patterns", "wide", "spike", "few", "crowded", "equal", "last"]


@pytest.fixture
def split_all(monkeypatch):
    """1-D sorts of every length and of all keys are tried by the splitting kernels."""
    monkeypatch.setenv("B2S_SPLIT", "8193")


def _tried(route: int, how: str, dtype: np.dtype, op: str) -> None:
    """The splits were tried, spread keys stayed with them, and what needs the input order of equal images did not."""
    assert route != OPEN
    if how == "normal":
        assert route == SPLIT
    if how == "patterns" and dtype.kind == "f" and op == "sort":
        assert route in (RADIX, LATE)


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("op", ["sort", "argsort"])
@pytest.mark.parametrize("dtype", ["int32", "uint32", "float32", "int64", "uint64", "float64"])
def test_two_splits(split_all, dtype, op, how):
    # (more keys than one split takes apart, and of 4-byte argsorts so many that the tables fit)
    t = np.dtype(dtype)
    n = 5_000_011 if op == "argsort" and t.itemsize == 4 else 2_100_019
    _tried(_check(_values(how, n, t, 11), op), how, t, op)


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("op", ["sort", "argsort"])
@pytest.mark.parametrize("dtype", ["int32", "float32", "uint64", "float64"])
def test_one_split(split_all, dtype, op, how):
    _tried(_check(_values(how, 300_007, np.dtype(dtype), 13), op), how, np.dtype(dtype), op)


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("op", ["sort", "argsort"])
@pytest.mark.parametrize("dtype", ["int32", "float32", "uint64", "float64"])
def test_long_rows(dtype, op, how):
    t = np.dtype(dtype)
    n, rows = 20_011, 60   # (sorts of 4-byte keys: from 10^6 on)
    _tried(_check(_values(how, n * rows, t, 12).reshape(rows, n), op), how, t, op)


# around the lengths where the buckets' size, the number of splits and the tables change: 200 buckets of 2048, 4096, 6144
# (with positions) and 8192 keys
@pytest.mark.parametrize("n", [8193, 8704, 16384, 30011, 409_600, 409_601, 819_201, 1_100_003, 1_228_801, 1_638_401])
@pytest.mark.parametrize("dtype", ["int32", "float32", "int64", "float64"])
def test_lengths(split_all, dtype, n):
    t = np.dtype(dtype)
    for op in ("sort", "argsort"):
        route = _check(_values("nans", n, t, n), op)
        # (the tables of two splits of 4-byte pairs do not fit the look-back room of so few keys)
        assert (route == OPEN) == (t.itemsize == 4 and op == "argsort" and n > 1_228_800)
    if n < 100_000:
        # (nor those of few rows of up to 16384 4-byte pairs)
        route = _check(_values("nans", n * 3, t, n).reshape(3, n), "argsort")
        assert (route == OPEN) == (t.itemsize == 4 and n <= 16384)


@pytest.mark.parametrize("dtype,op,n", [("int32", "sort", 39_000_017), ("int32", "sort", 60_000_011), ("int64", "sort", 60_000_011), ("float64", "sort", 60_000_011),
                                        ("float32", "argsort", 39_000_017), ("int64", "argsort", 93_000_017), ("float64", "argsort", 93_000_017)])
def test_long_plans(dtype, op, n):
    """Plans of 8192 cells, and leaves of 8192, with positions 6144, keys after two splits, for each mapping; against torch's sort."""
    import cupynumeric_b200 as num

    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    t = getattr(torch, dtype)
    bits = 8 * t.itemsize
    if t.is_floating_point:
        draws = [torch.rand(n, dtype=t, device="cuda", generator=gen), torch.randn(n, dtype=t, device="cuda", generator=gen)]
        draws[1][7::1001] = float("nan")
    else:
        raw = torch.randint(0, 256, (n * t.itemsize,), dtype=torch.uint8, device="cuda", generator=gen).view(t)
        u = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
        draws = [raw, (1 - u).pow(-5.0).clamp(max=2.0 ** min(bits - 2, 40)).to(t)] if op == "sort" else [raw]   # (Zipf argsorts go back)
        if op == "sort":
            draws.append(torch.where(u < 0.5, torch.full((), 12345, dtype=t, device="cuda"), raw))     # a spike
    for k, a in enumerate(draws):
        want = torch.sort(a, stable=True)
        got = num.sort(num.array(a)) if op == "sort" else num.argsort(num.array(a), kind="stable")
        assert _route() == SPLIT, k
        if op == "argsort":
            assert torch.equal(got.torch(), want.indices)
        else:
            i = torch.int32 if bits == 32 else torch.int64
            assert torch.equal(got.torch().view(i), want.values.view(i))
        del want, got


@pytest.mark.parametrize("names", [("float64", "int32"), ("float32", "int64"), ("int64", "float64", "int8")], ids="-".join)
def test_first_keys_of_lexsort(split_all, names):
    """Positions as 32 bits straight out of the leaves, for the keys behind."""
    import cupynumeric_b200 as num

    rng, n = np.random.default_rng(6), 300_007
    cols = [_values("normal", n, np.dtype(d), 5) if i == 0 else rng.integers(0, 90, n).astype(d) for i, d in enumerate(names)]
    cols[0][1::2] = cols[0][: n // 2]     # (two copies of each)
    assert np.array_equal(num.lexsort(cols).to_numpy(), np.lexsort(cols))


@pytest.mark.parametrize("n", [300_007, 3_000_017])
def test_payloads_of_complex_argsorts(n):
    """The real parts are sorted behind the imaginary ones, whose order is the payload that the leaves look up."""
    import cupynumeric_b200 as num

    rng = np.random.default_rng(n)
    a = rng.permutation(np.repeat(rng.standard_normal(n // 2 + 1), 2)[:n]) + 1j * rng.permutation(np.repeat(rng.standard_normal(n // 3 + 1), 3)[:n])
    assert np.array_equal(num.argsort(a, kind="stable").to_numpy(), np.argsort(a, kind="stable"))


@pytest.mark.parametrize("dtype", ["float64", "uint64"])
def test_payloads_of_distributed_argsorts(split_all, dtype):
    """What a rank received carries positions of the whole array."""
    from tests.test_gpu_dist_threads import run_ranks

    t = np.dtype(dtype)
    a = _values("normal", 700_001, t, 9)
    a[1::2] = a[:350_000]
    shards = np.split(a, [250_000, 460_000])
    parts = [part for status, part, _, _ in run_ranks(shards, True) if status == 0]
    assert len(parts) == 3 and min(p.size for p in parts) > 200_000
    assert np.array_equal(np.concatenate(parts), np.argsort(a, kind="stable"))


@pytest.mark.parametrize("dtype,n", [("float32", 6_000_011), ("int64", 24_000_017)])
def test_as_it_is_dispatched(dtype, n):
    # (above the borders of the dispatch)
    for how in ("normal", "patterns"):
        a = _values(how, n, np.dtype(dtype), 3)
        for op in ("sort", "argsort"):
            _check(a, op)


@pytest.mark.parametrize("dtype,op,n", [("float32", "argsort", 700_001), ("float32", "argsort", 5_000_011), ("float64", "argsort", 250_007),
                                        ("int64", "argsort", 24_000_017), ("int64", "sort", 24_000_017)])
def test_sent_back_with_the_sample(dtype, op, n):
    """Keys that need few passes: alike as far as the sample sees, or, in a sort of int64, of two differing bytes."""
    if op == "argsort":
        a = np.full(n, 3, np.dtype(dtype))
        a[n // 2] = 4
    else:
        a = np.random.default_rng(5).integers(0, 65536, n).astype(dtype)
    assert _check(a, op) == RADIX


def _crowds(how: str, n: int, dtype: np.dtype) -> np.ndarray:
    rng, bits = np.random.default_rng(n), 8 * dtype.itemsize - 1
    if how in ("signed", "negative"):          # every magnitude, in both directions or downwards only
        a = np.exp2(rng.uniform(0, bits, n))
        return (a * np.where(rng.random(n) < 0.5, 1.0, -1.0) if how == "signed" else -a).astype(dtype)
    a = np.rint(rng.standard_normal(n) * 3)     # crowded around one place, or two, with outliers on both sides
    if how == "two":
        a += np.where(rng.random(n) < 0.5, 2.0**29, -(2.0**28))
    out = rng.random(n) < 0.01
    a[out] = rng.integers(-(2**20), 2**20, n)[out] if how == "one" else rng.integers(-(2**30), 2**30, n)[out]
    return a.astype(dtype)


@pytest.mark.parametrize("rows,n", [(1, 300_007), (1, 2_100_019), (3, 400_009), (37, 20_011)])
@pytest.mark.parametrize("dtype", ["int32", "int64"])
def test_crowds_inside_the_range(split_all, dtype, rows, n):
    """Integers whose crowd lies at neither end of their range: a second split fills in or takes apart what is crowded around a place;
    what it could not, or a leaf, goes back with the sample.  No block is left with most of the keys."""
    for how in ("signed", "negative", "one", "two"):
        a = _crowds(how, rows * n, np.dtype(dtype))
        got = _check(a.reshape(rows, n) if rows > 1 else a, "sort")
        if n > 2_000_000:
            assert got == SPLIT or how in ("signed", "negative"), how
        else:
            assert got in (SPLIT, RADIX), how


@pytest.mark.parametrize("width,count,split", [(2048, 45_000, True), (2048, 55_000, False), (4096, 45_000, False)])
def test_a_bucket_of_few_values(split_all, width, count, split):
    """A cell of a row with no more values and keys than one block counts, or with more of either."""
    rng, n = np.random.default_rng(width), 1_000_003
    rows = np.empty((2, n), np.int64)
    edge = width * 1000 - ((width * 1980 - 1) >> 6) % width     # of a cell: the range gets a 64th of itself as room
    for r in rows:
        r[:] = rng.integers(0, width * 1980, n)
        r[:2] = 0, width * 1980 - 1
        r[rng.permutation(n - 2)[:count] + 2] = edge + rng.integers(0, width, count)
    assert (_check(rows, "sort") == SPLIT) == split


@pytest.mark.parametrize("dtype", ["int32", "float32", "int64"])
def test_rows_of_one_value(dtype):
    """A cell of its own, filled in: no copies that crowd anything."""
    assert _check(np.full((200, 12_000), 3, np.dtype(dtype)), "sort") == SPLIT


@pytest.mark.parametrize("dtype", ["int32", "float32", "int64"])
def test_rows_of_two_leaves(dtype):
    """Sorts of 4-byte keys in rows below 10000 keep the passes, others do not."""
    for n in (9_999, 10_000):
        tried = _check(_values("normal", n * 200, np.dtype(dtype), 2).reshape(200, n), "sort")
        assert tried == (OPEN if n < 10_000 and dtype != "int64" else SPLIT)


@pytest.mark.parametrize("dtype,rows,n,copies", [("float64", 1, 250_007, 60), ("float32", 1, 700_001, 400), ("float32", 1, 5_000_011, 60),
                                                 ("int64", 1, 24_000_017, 60), ("float32", 1, 16_000_003, 40), ("float32", 60, 20_011, 80)])
def test_copies_send_argsorts_back(dtype, rows, n, copies):
    """Evenly used values: two copies of each stay with the splits, many go back with the sample, which draws more keys of long arrays."""
    rng = np.random.default_rng(n)
    for c in (2, copies):
        if c == 2 and n > 5_000_011:
            continue   # (test_as_it_is_dispatched)
        names = rng.standard_normal((rows, n // c)) * (2.0**40 if dtype == "int64" else 1.0)
        a = np.take_along_axis(names, rng.integers(0, n // c, (rows, n)), axis=1).astype(dtype)
        assert _check(a if rows > 1 else a[0], "argsort") == (SPLIT if c == 2 else RADIX)


@pytest.mark.parametrize("dtype,rows,n", [("float64", 1, 250_007), ("float32", 1, 5_000_011), ("float64", 37, 20_011), ("float32", 60, 20_011)])
def test_patterns_of_zeros_and_nans(dtype, rows, n):
    """A sort keeps the one pattern that its zeros have, and its NaNs; where there are several the passes take it, at once if
    the sample sees them."""
    t, bits = np.dtype(dtype), np.dtype(dtype).itemsize * 8
    rng = np.random.default_rng(n)
    base = (rng.standard_normal(rows * n) + 0.5).astype(t)
    odd = np.array((1 << (bits - 1)) - 1, f"u{t.itemsize}").view(t)       # what arithmetic on a GPU gives
    neg = np.array(((1 << bits) - 1) ^ 4, f"u{t.itemsize}").view(t)

    def case(*parts):
        a = base.copy()
        for value, places in parts:
            a[places] = value
        return _check(a.reshape((rows, n) if rows > 1 else n), "sort")

    some, more = (rng.integers(0, rows * n, rows * n // 50) for _ in range(2))
    few = rng.integers(0, rows * n, 500)     # (no more copies of a zero than a leaf holds)
    one = np.array([rows * n // 3])
    assert case() == SPLIT
    assert case((-0.0, few), (odd, more)) == SPLIT
    assert case((0.0, few), (neg, one)) == SPLIT
    assert case((-0.0, one)) == SPLIT
    assert case((odd, some), (np.nan, more)) == RADIX
    assert case((0.0, some), (-0.0, more)) == RADIX
    assert case((odd, one), (np.nan, one + 1)) in (RADIX, LATE)
    assert case((0.0, one), (-0.0, one + n // 3)) in (RADIX, LATE)


def test_in_place_and_other_streams(split_all):
    """The input stays whole until the last kernel writes; two sorts on two streams, which run at the same time, have a
    workspace each."""
    import cupynumeric_b200 as num
    from cupynumeric_b200.runtime import runtime

    a, b = (_values("normal", 2_500_001, np.dtype("int64"), k) for k in (5, 6))
    x = num.array(torch.from_numpy(a).cuda())
    z = num.array(torch.from_numpy(b).cuda())
    side = torch.cuda.Stream()
    own = runtime.workspace(1 << 16)
    with torch.cuda.stream(side):
        assert runtime.workspace(1 << 16).data_ptr() != own.data_ptr()
    del own
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        y = num.sort(z)
    x.sort()
    torch.cuda.synchronize()
    assert np.array_equal(x.to_numpy(), np.sort(a))
    assert np.array_equal(y.to_numpy(), np.sort(b))


def test_two_threads_on_one_stream(split_all):
    """Their kernels are enqueued in any order between each other."""
    import threading

    import cupynumeric_b200 as num

    inputs = [_values("normal", 300_007, np.dtype("float64"), k) for k in (1, 2)]
    dev = [num.array(torch.from_numpy(a).cuda()) for a in inputs]
    torch.cuda.synchronize()
    out = [[], []]
    threads = [threading.Thread(target=lambda i=i: out[i].extend(num.argsort(dev[i], kind="stable") for _ in range(20))) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        want = np.argsort(inputs[i], kind="stable")
        assert len(out[i]) == 20 and all(np.array_equal(o.to_numpy(), want) for o in out[i])


def test_under_capture(split_all):
    """The launches and their chaining can be captured and replayed on other keys."""
    import ctypes

    from cupynumeric_b200 import _lib

    n, lib, need = 700_001, _lib.lib(), ctypes.c_size_t()
    code = _lib.DTYPE_CODE[np.dtype("float64")]
    _lib.check(lib.b2s_workspace_bytes(code, n, n, 1, ctypes.byref(need)), "ws")
    keys = torch.empty(n, dtype=torch.float64, device="cuda")
    idx = torch.empty(n, dtype=torch.int64, device="cuda")
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _lib.check(lib.b2s_local_sort(code, keys.data_ptr(), None, idx.data_ptr(), n, n, 0, 1, 1, ws.data_ptr(), need.value,
                                      torch.cuda.current_stream().cuda_stream), "sort")
    for how in ("normal", "few", "wide"):
        a = _values(how, n, np.dtype("float64"), 8)
        keys.copy_(torch.from_numpy(a))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(idx.cpu().numpy(), np.argsort(a, kind="stable")), how
