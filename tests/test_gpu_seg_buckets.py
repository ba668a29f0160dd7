"""Segmented sort by buckets (the default): lengths around the bucket, the tiles and
the levels, segments that start at any item, heavy and clustered keys, samples that
mislead, more buckets than the sort's grid, and the merge path as the other side.
Integer work: the tolerance is zero."""
import numpy as np
import pytest

import oracle as orc
import origami_gpu as og

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
KINDS = [og.U32, og.U64, og.I64, og.KV64, og.KVU64]


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__ as g
    g.build()
    assert torch.cuda.is_available()


def items(kind, k):
    """Items with the 64-bit keys k (32-bit kinds: their upper halves)."""
    a = orc.empty(kind, len(k))
    if kind == og.U32:
        a[:] = (k >> np.uint64(32)).astype(np.uint32)
    elif a.dtype.names:
        a["key"] = k.view(a.dtype["key"])
        a["value"] = np.arange(len(k))
    else:
        a[:] = k.view(a.dtype)
    return a


def check(kind, a, lens):
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    d = torch.from_numpy(a.view(np.uint8).copy()).cuda()
    og.sort_segmented(d, torch.from_numpy(off).cuda(), kind=kind)
    got = d.cpu().numpy().view(a.dtype)
    want = a.copy()
    for s, e in zip(off[:-1], off[1:]):
        x = a[s:e]
        want[s:e] = x[np.argsort(x["key"], kind="stable")] if a.dtype.names else np.sort(x)
    assert np.array_equal(got, want)


def keys(dist, n, rng):
    k = rng.integers(0, 2**64, n, dtype=np.uint64)
    if dist == "equal":
        k[:] = k[:1]
    elif dist == "heavy":  # one key for half of the items, at one end of the order
        k[rng.random(n) < 0.5] = ~np.uint64(0)
    elif dist == "ids":  # a few thousand neighbouring keys
        k = (k % np.uint64(3000)) << np.uint64(32)
    elif dist == "zipf":
        r = np.exp(rng.random(n) * np.log(2.0**20)).astype(np.uint64)
        k = r * np.uint64(0x9E3779B97F4A7C15)
    elif dist == "pairs":  # crowded bins of two heavy keys each
        k = (k % np.uint64(40)) * np.uint64(1 << 58) + (k >> np.uint64(63) << np.uint64(33))
    elif dist == "log":  # clusters in clusters
        k >>= (k % np.uint64(32)).astype(np.uint64)
    elif dist == "sorted":
        k.sort()
    return k


# a bucket holds 6144 uint32 keys or 4096 wider items; tiles of the same size
EDGES = [1, 0, 2, 33, 4095, 4096, 4097, 6143, 6144, 6145, 8191, 8193, 12289, 3 * 6144 + 1, 65537, 262147, 1]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dist", ["uniform", "equal", "heavy", "ids", "zipf", "pairs", "log", "sorted"])
def test_lengths(kind, dist):
    rng = np.random.default_rng(kind * 31 + len(dist))
    check(kind, items(kind, np.concatenate([keys(dist, n, rng) for n in EDGES])), EDGES)


@pytest.mark.parametrize("kind", [og.U32, og.I64, og.KV64])
@pytest.mark.parametrize("dist", ["uniform", "zipf", "log"])
def test_two_levels(kind, dist):
    lens = [3, (1 << 21) + 77, 5000]
    rng = np.random.default_rng(kind + 5)
    check(kind, items(kind, np.concatenate([keys(dist, n, rng) for n in lens])), lens)


def sampled(n, samples=2048):
    j = np.arange(samples, dtype=np.uint64)
    a = np.uint64(n) * j // np.uint64(samples)
    gap = np.uint64(n) * (j + np.uint64(1)) // np.uint64(samples) - a
    h = (j * np.uint64(2654435761) + np.uint64(12345)) & np.uint64(0xFFFFFFFF)
    return (a + (h * gap >> np.uint64(32))).astype(np.int64)


@pytest.mark.parametrize("kind", [og.U32, og.U64, og.KV64])
def test_misleading_samples(kind):
    # the first level's samples are spread over all keys, the other items lie in one
    # of its slices and spread over their logarithms: the last level's slices are
    # too long for a bucket and are sorted in global memory
    n = 1200000 if kind == og.U32 else 800000
    rng = np.random.default_rng(9)
    k = np.exp(rng.random(n) * np.log(2.0**23)).astype(np.uint64) << np.uint64(32)
    k |= rng.integers(0, 2**32, n, dtype=np.uint64)
    p = sampled(n)
    k[p] = rng.integers(0, 2**64, len(p), dtype=np.uint64)
    check(kind, items(kind, k), [n])


@pytest.mark.parametrize("kind", [og.U32, og.U64, og.KV64])
def test_more_buckets_than_the_grid(kind):
    # slices just over half a bucket, each followed by a slice of one item: twice as
    # many buckets as half buckets in the segment
    half = (6144 if kind == og.U32 else 4096) // 2 + 20
    rng = np.random.default_rng(3)
    k = []
    for s in range(0, 256, 2):
        k.append((np.uint64(s) << np.uint64(56)) + (np.uint64(1) << np.uint64(55)) +
                 (rng.integers(0, 2**20, half, dtype=np.uint64) << np.uint64(32)))
        k.append(np.array([((s + 1) << 56) + (1 << 55)], np.uint64))
    k = np.concatenate(k)
    check(kind, items(kind, rng.permutation(k)), [len(k)])


def log_uniform(n, rng):
    return np.exp2(rng.random(n) * 63).astype(np.uint64) << np.uint64(1)


# short segments whose bins of equal width do not settle them: around the size from which
# they take splitters, the largest, equal keys of some and of many items among them, keys
# in their range's upper end, and splitters that mislead (256 spread keys at the sampled
# places, all others close together)
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dist", ["log", "equal", "high", "misled"])
def test_crowded_buckets(kind, dist):
    lens = [17, 34, 255, 256, 257, 300, 1000, 2049, 4095, 4096, 5000, 6143, 6144]
    rng = np.random.default_rng(kind + 3)
    parts = []
    for n in lens:
        k = log_uniform(n, rng)
        if dist == "equal":
            for i in range(4):
                k[rng.random(n) < 0.2] = k[i]
        elif dist == "high":
            k = ~k
        elif dist == "misled" and n > 256:
            k = (np.uint64(3) << np.uint64(62)) + (rng.integers(0, 2**20, n, dtype=np.uint64) << np.uint64(32))
            p = sampled(n, 256)
            k[p] = rng.integers(0, 2**62, len(p), dtype=np.uint64)
        parts.append(k)
    check(kind, items(kind, np.concatenate(parts)), lens)


def best_ms(kind, k, sort):
    """Best of some runs of sort(d, t) on items with the keys k."""
    src = torch.from_numpy(items(kind, k).view(np.uint8).copy()).cuda()
    d, t = torch.empty_like(src), torch.empty_like(src)
    best = 1e9
    for _ in range(6):
        d.copy_(src)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        sort(d, t)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("kind", [og.U32, og.U64, og.KV64])
def test_skewed_groups_keep_pace(kind):
    # groups of 200 log-uniform keys against uniform ones: the time differs by 2.5 to 3.5
    # (by byte passes it did by 9 to 23)
    n, group = 1 << 22, 200
    off = torch.from_numpy(np.append(np.arange(0, n, group), n)).cuda()
    rng = np.random.default_rng(1)
    uniform, log = (best_ms(kind, k, lambda d, t: og.sort_segmented(d, off, t, kind=kind, sync=False))
                    for k in (keys("uniform", n, rng), log_uniform(n, rng)))
    assert log < 6 * uniform


def nested(n, rng):
    """Uniform keys, 11.5 % of them in one 256th of the range, of these 11.5 % in one
    256th of that, and so on."""
    k = rng.integers(0, 2**64, n, dtype=np.uint64)
    u = rng.random(n)
    for d in range(1, 8):
        low = np.uint64((1 << (64 - 8 * d)) - 1)
        k = np.where(u < 0.115**d, (np.uint64(0x5A5A5A5A5A5A5A5A) & ~low) | (k & low), k)
    return k


# one level, two and three
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.KV64])
@pytest.mark.parametrize("n", [120_000, 838_000, 3_500_000])
def test_nested_clusters(kind, n):
    check(kind, items(kind, nested(n, np.random.default_rng(n))), [n])


@pytest.mark.parametrize("kind", [og.U64, og.KV64])
@pytest.mark.parametrize("n", [838_000, 1 << 24])
def test_nested_clusters_keep_pace(kind, n):
    # no slice is left too long for a bucket: 1.4 to 2.6 times uniform keys (where the last
    # level left such slices, 6 to 20 times)
    rng = np.random.default_rng(2)
    uniform, clusters = (best_ms(kind, k, lambda d, t: og.sort(d, t, kind=kind))
                         for k in (keys("uniform", n, rng), nested(n, rng)))
    assert clusters < 4 * uniform


@pytest.mark.parametrize("kind", [og.U32, og.U64, og.KV64])
def test_long_slices_beyond_the_grid(kind):
    # more buckets than the grid, and among those beyond it slices that are too long:
    # two segments of alternating slices (as above), then one whose first level's
    # samples mislead, so that the last level cuts 100 buckets' worth of items into 127
    # uneven slices. (By the slices' definition some 600 buckets, 444 of them in the
    # grid, about 20 too long, 10 of them beyond the grid.)
    cap = 6144 if kind == og.U32 else 4096
    rng = np.random.default_rng(11)

    def alternating():
        k = [np.array([(255 << 56) + (1 << 55)], np.uint64)]
        for s in range(0, 186, 2):
            k.append((np.uint64(s) << np.uint64(56)) + (np.uint64(1) << np.uint64(55)) +
                     (rng.integers(0, 2**20, cap // 2 + 20, dtype=np.uint64) << np.uint64(32)))
            k.append(np.array([((s + 1) << 56) + (1 << 55)], np.uint64))
        return rng.permutation(np.concatenate(k))

    n = 102 * cap
    k = (np.uint64(77) << np.uint64(56)) + (np.uint64(1) << np.uint64(54))
    k = k + (rng.random(n) ** 4 * 2.0**55).astype(np.uint64)
    p = sampled(n)
    k[p] = rng.integers(0, 2**64, len(p), dtype=np.uint64)
    segs = [alternating(), alternating(), k]
    check(kind, items(kind, np.concatenate(segs)), [len(s) for s in segs])


@pytest.mark.parametrize("kind", [og.U32, og.KV64])
def test_merges_when_tuned(kind, tmp_path):
    rng = np.random.default_rng(2)
    lens = rng.integers(1, 40000, 50)
    a = items(kind, keys("zipf", int(lens.sum()), rng))
    cls = int(lens.sum() // len(lens)).bit_length() - 1
    f = tmp_path / "tuning"

    def launched(on):
        f.write_text(f"segbuckets {kind} {cls} {on}\n")
        og.tuning_load(str(f))
        og.profile_enable(True)
        check(kind, a, lens)
        names = set(og.profile_report())
        og.profile_enable(False)
        return {n for n in names if n.startswith("segbucket")}

    try:
        assert not launched(0)
        og.tuning_save(str(f))
        assert f"segbuckets {kind} {cls} 0" in f.read_text()
    finally:
        assert launched(1)


@pytest.mark.parametrize("kind", [og.KV64])
def test_pairs_report_expired_wait(kind):
    # keys: test_gpu_timeout.py
    lens = [1 << 16, 3 << 15]
    a = items(kind, keys("uniform", sum(lens), np.random.default_rng(1)))
    old = og.wait_limit()
    og.set_wait_limit(0)
    try:
        with pytest.raises(og.OrigamiError) as e:
            check(kind, a, lens)
        assert e.value.code == og.ERR_TIMEOUT
    finally:
        og.set_wait_limit(old)
    check(kind, a, lens)


ORDER = """
import sys
import numpy as np, torch, oracle as orc, origami_gpu as og
kind = int(sys.argv[1])
def buf(n):
    a = orc.empty(kind, n)
    k = np.random.default_rng(9).integers(0, 1 << 31, n).astype(np.uint32)
    if a.dtype.names:
        a["key"], a["value"] = k, np.arange(n)
    else:
        a[:] = k
    return a
def segmented():
    a = buf(30000)
    d, off = torch.from_numpy(a.view(np.uint8).copy()).cuda(), torch.tensor([0, 7, 30000], device="cuda")
    og.SegmentedPlan(d, off, torch.empty_like(d), kind).launch(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return d, a, [(0, 7), (7, 30000)]
def plain(n, sort_n, min_k=0):
    a = buf(n)
    d = torch.from_numpy(a.view(np.uint8).copy()).cuda()
    o = og.sort(d, torch.empty_like(d), kind=kind, sort_n=sort_n, min_k=min_k)
    torch.cuda.synchronize()
    s = sort_n or n
    return o, a, [(i, min(i + s, n)) for i in range(0, n, s)]
calls = {"segmented": segmented, "levels": lambda: plain(1 << 25, 1 << 18 if kind == og.U32 else 0),
         "merges": lambda: plain(1 << 22, 0, 16), "chunks": lambda: plain(1 << 22, 1 << 17)}
for c in sys.argv[2:]:
    d, a, segs = calls[c]()
    got = d.cpu().numpy().view(a.dtype)
    for s, e in segs:
        x = a[s:e]
        want = x[np.argsort(x["key"], kind="stable")] if a.dtype.names else np.sort(x)
        assert np.array_equal(got[s:e], want), c
"""


@pytest.mark.parametrize("order", [("segmented", "levels"), ("levels", "segmented"), ("merges", "chunks"), ("chunks", "merges")])
@pytest.mark.parametrize("kind", [og.U32, og.U64, og.KV64])
def test_first_calls_in_either_order(kind, order):
    # what a process sets up once for the kernels of its first call is there for the second
    import os
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", ORDER, str(kind), *order], capture_output=True, text=True,
                       env={**os.environ, "PYTHONPATH": os.pathsep.join(p for p in sys.path if p)})
    assert r.returncode == 0, r.stderr[-800:]
