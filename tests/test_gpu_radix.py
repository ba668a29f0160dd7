"""Bucket sort and what stands behind it (the default of device sorts from some size
on): tile edges, ragged ends, one and two partition levels, digits
with one, two and sixteen values, clustered, duplicated and outlying keys, both
result buffers, chunks, and the bounded waits. Integer work: the tolerance is
zero."""
import ctypes

import numpy as np
import pytest

import oracle as orc
import origami_gpu as og

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__ as g
    g.build()
    assert torch.cuda.is_available()


def keys(dist, n, seed):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 2**64, n, dtype=np.uint64)
    if dist == "equal":
        k[:] = k[0]
    elif dist == "two":  # every digit has two values
        k = np.where(k & np.uint64(1), np.uint64(0), ~np.uint64(0))
    elif dist == "sixteen":
        k = (k & np.uint64(15)) * np.uint64(0x9E3779B97F4A7C15)
    elif dist == "small":  # constant high digits
        k &= np.uint64(0xFFFFF)
    elif dist == "one_high":  # all but one key share the high digits
        k &= np.uint64(0xFFFF)
        k[n // 2] = ~np.uint64(0)
    elif dist == "sorted":
        k.sort()
    elif dist == "normal":  # slices of very different sizes
        k = (np.clip(rng.normal(0.5, 0.1, n), 0, 1) * (2.0**64 - 4096)).astype(np.uint64)
    elif dist == "repeated":  # every key some 200 times
        d = rng.integers(0, 2**64, max(1, n // 200), dtype=np.uint64)
        k = d[rng.integers(0, len(d), n)]
    elif dist == "clusters":  # 100 neighbouring keys around each of many centres
        d = rng.integers(0, 2**64, max(1, n // 1000), dtype=np.uint64) & ~np.uint64(0x7F00000000)
        k = d[rng.integers(0, len(d), n)] + (rng.integers(0, 100, n).astype(np.uint64) << np.uint64(32))
    elif dist == "zipf":  # a few heavy keys, spread over the range
        k = np.exp(rng.random(n) * np.log(2.0**20)).astype(np.uint64) * np.uint64(0x9E3779B97F4A7C15)
    elif dist == "log":  # clusters in clusters
        k >>= (k % np.uint64(48)).astype(np.uint64)
    elif dist == "outliers":  # a narrow range and a few keys far outside it
        k = (k >> np.uint64(22)) + (np.uint64(5) << np.uint64(60))
        k[:: max(1, n // 5)] = rng.integers(0, 2**64, len(k[:: max(1, n // 5)]), dtype=np.uint64)
    return k


def items(kind, dist, n, seed):
    k = keys(dist, n, seed)
    a = orc.empty(kind, n)
    if kind == og.U32:
        a[:] = (k if dist in ("equal", "two", "sixteen", "small", "one_high") else k >> np.uint64(32)).astype(np.uint32)
    elif a.dtype.names:
        a["key"] = k.view(a.dtype["key"])
        a["value"] = np.arange(n)
    else:
        a[:] = k.view(a.dtype)
    return a


def expected(a, sort_n=0):
    out = a.copy()
    for i in range(0, len(a), sort_n or len(a)):
        c = a[i:i + (sort_n or len(a))]
        out[i:i + len(c)] = c[np.argsort(orc.keys_of(c), kind="stable")]
    return out


def device_sort(a, kind, **kw):
    d = torch.from_numpy(a.view(np.uint8).copy()).cuda()
    t = torch.empty_like(d)
    r = og.sort(d, t, kind=kind, **kw)
    torch.cuda.synchronize()
    assert r.data_ptr() == (t if kw.get("result_in_tmp") else d).data_ptr()
    return r.cpu().numpy().view(a.dtype)


@pytest.mark.parametrize("in_tmp", [False, True])
@pytest.mark.parametrize("dist", ["uniform", "equal", "two", "sixteen", "small", "one_high", "sorted"])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.I64, og.KV64, og.KVU64])
@pytest.mark.parametrize("n", [1 << 17, 135_167, 1_310_721])
def test_radix_matches_stable_sort(kind, dist, n, in_tmp):
    a = items(kind, dist, n, seed=n + kind)
    assert np.array_equal(device_sort(a, kind, result_in_tmp=in_tmp), expected(a))


# one bucket (up to 6144 uint32 keys, 4096 wider items), and the sizes around it and
# around the smallest sort by several buckets
@pytest.mark.parametrize("in_tmp", [False, True])
@pytest.mark.parametrize("dist", ["uniform", "equal", "sixteen", "zipf", "clusters", "sorted"])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.I64, og.KV64, og.KVU64])
def test_one_bucket(kind, dist, in_tmp):
    for n in (2, 3, 31, 255, 1000, 4095, 4096, 4097, 6143, 6144, 6145, 16383, 16384, 32767, 32768):
        a = items(kind, dist, n, seed=n)
        assert np.array_equal(device_sort(a, kind, result_in_tmp=in_tmp), expected(a)), n


# the largest one-level sort and the smallest two-level one of each kind are
# 2^20 / 2^20 + 1 items (u32) and 2^19 / 2^19 + 1 (64-bit keys)
@pytest.mark.parametrize("dist", ["uniform", "normal", "repeated", "clusters", "zipf", "log", "outliers"])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.I64, og.KV64, og.KVU64])
@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1, 1 << 20, (1 << 20) + 1, (1 << 22) + 8191])
def test_buckets_match_stable_sort(kind, dist, n):
    a = items(kind, dist, n, seed=n + kind)
    assert np.array_equal(device_sort(a, kind, result_in_tmp=bool(n & 1)), expected(a))


@pytest.mark.parametrize("kind", [og.U32, og.I64, og.KV64])
@pytest.mark.parametrize("sort_n", [1 << 19, 1 << 20])
@pytest.mark.parametrize("second", ["small", "zipf", "log"])
def test_radix_chunks(kind, sort_n, second):
    n = (1 << 21) + 4099  # the last chunk is short
    a = items(kind, "uniform", n, seed=3)
    a[sort_n:2 * sort_n] = items(kind, second, sort_n, seed=4)  # one chunk of other keys
    assert np.array_equal(device_sort(a, kind, sort_n=sort_n), expected(a, sort_n))


def device_keys(dist, n, sort_n):
    """n uint32 keys (int32 storage): all of one distribution, or one chunk of it."""
    g = torch.Generator(device="cuda").manual_seed(n)
    k = torch.randint(-(2**31), 2**31, (n,), dtype=torch.int32, device="cuda", generator=g)
    u = torch.rand(n, device="cuda", dtype=torch.float64, generator=g)
    if dist == "zipf":
        return (torch.exp(u * np.log(2.0**20)).long() * 0x9E3779B1).to(torch.int32)
    if dist == "log":
        return torch.exp2(u * 30.99).to(torch.int32)
    if dist == "sixteen":
        return (k & 15) * 0x1E3779B1
    if dist == "one chunk":
        k[sort_n:2 * sort_n] = (torch.exp(u[:sort_n] * np.log(2.0**20)).long() * 0x9E3779B1).to(torch.int32)
    return k


def merged(src, sort_n):
    d, t = src.clone(), torch.empty_like(src)
    return og.sort(d, t, kind=og.U32, sort_n=sort_n, min_k=2)


# chunks of uint32 keys that the buckets give up: merges stand behind them up to chunks of
# 2^17 keys (sorts of 2^22 and more), levels up to 2^20 (2^25), radix passes elsewhere; the
# sizes on either side, a short last chunk
@pytest.mark.parametrize("n, sort_n", [(1 << 22, 1 << 16), ((1 << 22) - 1, 1 << 16), ((1 << 22) + 8191, 1 << 17),
                                       ((1 << 22) + 1, 1 << 18), ((1 << 25) + 77, 1 << 17), (1 << 25, 1 << 18),
                                       ((1 << 25) + 4099, 1 << 20), ((1 << 25) - 1, 1 << 20), ((1 << 25) + 1, 1 << 21)])
@pytest.mark.parametrize("dist", ["uniform", "zipf", "log", "sixteen", "one chunk"])
@pytest.mark.parametrize("in_tmp", [False, True])
def test_skewed_chunks(n, sort_n, dist, in_tmp):
    src = device_keys(dist, n, sort_n)
    d, t = src.clone(), torch.empty_like(src)
    got = og.sort(d, t, kind=og.U32, sort_n=sort_n, result_in_tmp=in_tmp)
    assert got.data_ptr() == (t if in_tmp else d).data_ptr()
    assert torch.equal(got, merged(src, sort_n))


@pytest.mark.parametrize("sort_n, dist, most", [(1 << 16, "zipf", 1.75), (1 << 17, "zipf", 1.6), (1 << 19, "sixteen", 1.2),
                                                (1 << 20, "zipf", 1.35)])
def test_skewed_chunks_keep_pace(sort_n, dist, most):
    # against merges, 1.41, 1.25, 0.75 and 1.18 times their time (radix passes 2.31, 1.93,
    # 1.57 and 1.41)
    src = device_keys(dist, 1 << 26, sort_n)
    d, t = torch.empty_like(src), torch.empty_like(src)

    def ms(min_k):
        best = 1e9
        for _ in range(6):
            d.copy_(src)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            og.sort(d, t, kind=og.U32, sort_n=sort_n, min_k=min_k)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert ms(0) < most * ms(2)


# five chunks, the last one short: their sorts leave signed keys in the internal order
@pytest.mark.parametrize("dist", ["uniform", "equal", "zipf", "log", "repeated"])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.I64, og.KV64, og.KVU64])
def test_host_chunks(kind, dist):
    n = (1 << 24) + (1 << 17) + 3
    a = items(kind, dist, n, seed=kind)
    b = a.copy()
    og.sort(b, np.empty_like(b))
    assert np.array_equal(b, expected(a))


def test_radix_long_segment():
    # 2^30 items and more: the counts of one segment need the wide words
    n = (1 << 30) + 5
    g = torch.Generator(device="cuda").manual_seed(9)
    src = torch.randint(-(2**31), 2**31, (n,), dtype=torch.int32, device="cuda", generator=g)
    want = int(src.sum(dtype=torch.int64))
    t = torch.empty_like(src)
    out = og.sort(src, t, kind="u32")
    del t
    assert int(out.sum(dtype=torch.int64)) == want
    for i in range(0, n, 1 << 28):
        x = out[i:i + (1 << 28) + 1] ^ torch.tensor(-(2**31), dtype=torch.int32, device="cuda")
        assert bool((x[1:] >= x[:-1]).all())


def mix(i):
    """A bijection of 64-bit words."""
    i = i * -0x61C8864680B583EB
    i = i ^ (i >> 32 & 0xFFFFFFFF)
    return i * -0x3B314601E57A13AD


def unmix(k):
    inv = lambda m: pow(m, -1, 2**64) - 2**64  # noqa: E731  (as a negative number)
    k = k * torch.tensor(inv(-0x3B314601E57A13AD & 2**64 - 1), device=k.device)
    k = k ^ (k >> 32 & 0xFFFFFFFF)
    return k * torch.tensor(inv(-0x61C8864680B583EB & 2**64 - 1), device=k.device)


# the longest sorts that buckets take and the shortest that they don't (levels alone), and
# those whose counts need 64 bits: pairs from 2^30 items, keys from 2^32
@pytest.mark.parametrize("kind, n", [("u64", (1 << 27) + 65535), ("u64", (1 << 27) + 65536), ("kvu64", (1 << 27) + 65535),
                                     ("kvu64", (1 << 27) + 65537), ("kvu64", (1 << 30) + 3), ("u64", (1 << 32) + 5)])
def test_long_sorts(kind, n):
    pairs = kind == "kvu64"
    piece = 1 << 27
    d = torch.empty((n, 2) if pairs else n, dtype=torch.int64, device="cuda")
    for i in range(0, n, piece):
        x = torch.arange(i, min(n, i + piece), device="cuda")
        if pairs:  # every key twice
            d[i:i + piece, 0] = mix(x >> 1)
            d[i:i + piece, 1] = x
        else:
            d[i:i + piece] = mix(x)
    t = torch.empty_like(d)
    out = og.sort(d.view(-1), t.view(-1), kind=kind).view(d.shape)
    del t
    for i in range(0, n, piece):
        x = out[i:i + piece + 1]
        k = (x[:, 0] if pairs else x) ^ -(2**63)
        v = x[:, 1] if pairs else unmix(x)
        # strictly ascending (key, value), of values that belong to them: a permutation
        assert bool((v >= 0).all()) and bool((v < n).all())
        if pairs:
            assert torch.equal(mix(v >> 1), x[:, 0])
            assert bool(((k[1:] > k[:-1]) | ((k[1:] == k[:-1]) & (v[1:] > v[:-1]))).all())
        else:
            assert bool((k[1:] > k[:-1]).all())


@pytest.mark.parametrize("n", [(1 << 28) + 65535, (1 << 28) + 65536])
def test_long_uint32_sorts(n):
    g = torch.Generator(device="cuda").manual_seed(4)
    src = torch.randint(-(2**31), 2**31, (n,), dtype=torch.int32, device="cuda", generator=g)
    out = og.sort(src.clone(), torch.empty_like(src), kind="u32")
    assert torch.equal(out ^ -(2**31), torch.sort(src ^ -(2**31)).values)


# (2^31 keys in chunks and more: merges, as the bucket sort does not take them)
def test_chunks_beyond_the_bucket_sort():
    n, sort_n = (1 << 31) + 9, 1 << 20
    g = torch.Generator(device="cuda").manual_seed(6)
    src = torch.randint(-(2**31), 2**31, (n,), dtype=torch.int32, device="cuda", generator=g)
    d, t = src.clone(), torch.empty_like(src)
    out = og.sort(d, t, kind="u32", sort_n=sort_n) ^ -(2**31)
    for i in range(0, n, 1 << 28):
        want = src[i:i + (1 << 28)] ^ -(2**31)
        whole = len(want) // sort_n * sort_n
        assert torch.equal(out[i:i + whole], torch.sort(want[:whole].view(-1, sort_n)).values.view(-1))
        assert torch.equal(out[i + whole:i + len(want)], torch.sort(want[whole:]).values)


@pytest.mark.parametrize("kind", [og.U32, og.KV64])
def test_radix_reports_expired_wait_then_recovers(kind):
    n = 1 << 20
    a = items(kind, "sixteen", n, seed=5)  # (buckets of keys wait for nothing)
    d = torch.from_numpy(a.view(np.uint8).copy()).cuda()
    t = torch.empty_like(d)
    res = ctypes.c_void_p()
    default = og.wait_limit()
    og.set_wait_limit(0)
    try:
        rc = og.lib().origami_sort_device(kind, d.data_ptr(), t.data_ptr(), n, 0, 0, og.FLAG_SYNC,
                                          ctypes.byref(res), None)
        assert rc == og.ERR_TIMEOUT
    finally:
        og.set_wait_limit(default)
    assert np.array_equal(device_sort(a, kind), expected(a))


def test_tuning_selects_radix_or_merges(tmp_path):
    # another shape selects merge passes, the built-in one restores the built-in
    # choice; both travel through a tuning file
    n = 1 << 20
    a = items(og.U32, "uniform", n, seed=6)
    prev = og.tuning_get(og.U32, n)

    def launched():
        og.profile_enable(True)
        assert np.array_equal(device_sort(a, og.U32), expected(a))
        names = set(og.profile_report())
        og.profile_enable(False)
        return any(k.startswith("radix") for k in names)

    try:
        assert launched()
        og.tuning_set(og.U32, n, 2, 1)
        assert not launched()
        og.tuning_save(tmp_path / "t")
        og.tuning_set(og.U32, n, *prev)
        assert launched()
        og.tuning_load(tmp_path / "t")
        assert not launched()
    finally:
        og.tuning_set(og.U32, n, *prev)


# the first kernel of the merge sorts: its tiles (4096 64-bit items), chunks of one tile,
# sorts of one tile, and the k-way passes that sample its runs
@pytest.mark.parametrize("dist", ["uniform", "equal", "zipf", "log", "sorted"])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.I64, og.KV64, og.KVU64])
@pytest.mark.parametrize("min_k", [2, 16])
def test_merge_tiles(kind, dist, min_k):
    for n, sort_n in ((1, 0), (17, 0), (4096, 0), (6145, 0), (8193, 0), (70_001, 0), (300_007, 0), (50_001, 256),
                      (50_001, 512), (50_001, 2048), (50_001, 4096), (50_001, 8192)):
        a = items(kind, dist, n, seed=n)
        assert np.array_equal(device_sort(a, kind, min_k=min_k, sort_n=sort_n), expected(a, sort_n)), (n, sort_n)


# host sorts of one bucket, and those that land in device memory: sizes around both
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("dist", ["uniform", "zipf", "equal", "log"])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.I64, og.KV64, og.KVU64])
def test_host_sizes(kind, dist, pinned):
    for n in (2, 1000, 4096, 4097, 6144, 6145, 16383, 16384, 32768, 70_001, (1 << 20) + 5):
        a = items(kind, dist, n, seed=n)
        d, out = og.empty_host(kind, n, pinned=pinned), og.empty_host(kind, n, pinned=pinned)
        d[:] = a
        assert og.sort(d, out, result_in_tmp=True) is out
        assert np.array_equal(out, expected(a)), n
        assert np.array_equal(d, a)  # (the input is only read)
        assert og.sort(d) is d
        assert np.array_equal(d, expected(a)), n
