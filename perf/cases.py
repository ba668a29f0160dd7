"""The sorts that users of this package run, as measured cases.

Each case is a dict of plain values: `form` is the entry point, `kind` the item
kind, `n` the items, `dist` the keys. Sizes and key distributions are those of
the repository's benchmark, tests and workloads: single arrays from 1,024 items
(the smallest served request) to 1 GiB of keys, chunked sorts of 128K to 2M
keys, pairs up to 2^27, batches of uneven arrays of 32 to 1,048,576 keys, host
buffers, and a mix of served requests.

A device sort works in place, so a program that keeps its column copies it
first: run() copies the kept input into the working buffer and sorts that.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "origami-sort_gb300"))
import origami_gpu as og  # noqa: E402

WORDS = {"u32": 1, "u64": 2, "i64": 2, "kv64": 4, "kvu64": 4}  # 32-bit words per item
ZIPF_DISTINCT = 1 << 20


def listed():
    return [
        # the smallest served request: one launch, all latency
        {"name": "u32 1,000", "form": "sort", "kind": "u32", "n": 1000, "dist": "uniform", "sort_n": 0, "in_tmp": False},
        # the plain sort's small configuration: L2-resident, launches count
        {"name": "u32 1M", "form": "sort", "kind": "u32", "n": 1 << 20, "dist": "uniform", "sort_n": 0, "in_tmp": False},
        # the headline: 1 GiB of uniform 32-bit keys
        {"name": "u32 1GiB", "form": "sort", "kind": "u32", "n": 1 << 28, "dist": "uniform", "sort_n": 0, "in_tmp": False},
        # the same volume as 64-bit keys
        {"name": "u64 1GiB", "form": "sort", "kind": "u64", "n": 1 << 27, "dist": "uniform", "sort_n": 0, "in_tmp": False},
        # 2^27 pairs with unique-ish keys (an index build)
        {"name": "kvu64 2^27", "form": "sort", "kind": "kvu64", "n": 1 << 27, "dist": "uniform", "sort_n": 0, "in_tmp": False},
        # pairs with many equal keys (a group-by), ragged size, result wanted in the second buffer
        {"name": "kv64 zipf 1.5M", "form": "sort", "kind": "kv64", "n": 1_500_007, "dist": "zipf", "sort_n": 0, "in_tmp": True},
        # the chunk sweep's middle: 1 GiB sorted in independent chunks
        {"name": "u32 chunks 512K", "form": "sort", "kind": "u32", "n": 1 << 28, "dist": "uniform", "sort_n": 1 << 19, "in_tmp": False},
        # the reference's own call with its default merge fan-in, signed keys, ragged size
        {"name": "i64 multi_thread", "form": "multi", "kind": "i64", "n": (1 << 24) + 77, "dist": "uniform", "min_k": 2},
        # the batched form: uneven arrays, one graph replay
        {"name": "batch u32", "form": "plan", "kind": "u32", "nseg": 4096, "lo": 32, "hi": 1 << 20},
        # many short groups of pairs in one plain call
        {"name": "segments kvu64", "form": "segmented", "kind": "kvu64", "nseg": 6000, "lo": 32, "hi": 1 << 16},
        # the drop-in for the CPU sort: pinned host memory in and out
        {"name": "host u32 256MiB", "form": "host", "kind": "u32", "n": 1 << 26, "dist": "uniform", "pinned": True},
        # the serving loop: requests of mixed kinds and sizes from pinned memory, submitted together
        {"name": "serve mix", "form": "serve", "requests": 24, "lo": 1 << 10, "hi": 1 << 23},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    form = rng.choice(["sort", "sort", "sort", "sort", "multi", "plan", "segmented", "host", "serve"])
    kind = rng.choice(["u32", "u64", "i64", "kv64", "kvu64"])
    dist = rng.choice(["uniform", "uniform", "zipf", "runs8", "reverse", "small"])
    most = (1 << 28) // WORDS[kind]  # 1 GiB of items
    if form == "sort":
        n = _log_int(rng, 1024, most)
        chunk = rng.choice([0, 0, 0, 1 << rng.randint(17, 21)])
        return {"form": form, "kind": kind, "n": n, "dist": dist, "sort_n": chunk if chunk < n else 0,
                "in_tmp": rng.random() < 0.3}
    if form == "multi":
        return {"form": form, "kind": kind, "n": _log_int(rng, 1024, most // 4), "dist": dist,
                "min_k": rng.choice([2, 2, 4, 8, 16])}
    if form == "plan":
        return {"form": form, "kind": kind, "nseg": _log_int(rng, 16, 4096), "lo": 32,
                "hi": (1 << 20) // WORDS[kind]}
    if form == "segmented":
        return {"form": form, "kind": kind, "nseg": _log_int(rng, 16, 6000), "lo": 32, "hi": _log_int(rng, 1 << 9, 1 << 16)}
    if form == "host":
        return {"form": form, "kind": kind, "n": _log_int(rng, 1024, most // 4), "dist": dist,
                "pinned": rng.random() < 0.5}
    return {"form": form, "requests": rng.randint(6, 24), "lo": 1 << 10, "hi": _log_int(rng, 1 << 16, 1 << 23)}


# ------------------------------------------------------------------ inputs --
def _uniform64(n, gen):
    return torch.randint(-(2**31), 2**31, (2 * n,), dtype=torch.int32, device="cuda", generator=gen).view(torch.int64)


def _keys(kind, n, dist, gen):
    """n keys: int32 storage for u32, int64 storage for the other kinds."""
    wide = WORDS[kind] > 1
    if dist == "zipf":  # rank r of 2^20 with probability ~ 1/r, spread by an odd factor
        u = torch.rand(n, device="cuda", generator=gen, dtype=torch.float64)
        rank = torch.floor(torch.exp(u * math.log(ZIPF_DISTINCT + 1.0))).to(torch.int64).clamp_(1, ZIPF_DISTINCT)
        if wide:
            return rank * -0x61C8864680B583EB
        k = (rank * 0x9E3779B1) & 0xFFFFFFFF
        return torch.where(k >= 2**31, k - 2**32, k).to(torch.int32)
    if dist == "small":  # ids below 2^20
        return torch.randint(0, 1 << 20, (n,), dtype=torch.int64 if wide else torch.int32, device="cuda", generator=gen)
    k = _uniform64(n, gen) if wide else torch.randint(-(2**31), 2**31, (n,), dtype=torch.int32, device="cuda", generator=gen)
    if dist == "uniform":
        return k
    top = torch.tensor(0 if kind in ("i64", "kv64") else (-(2**63) if wide else -(2**31)), dtype=k.dtype, device="cuda")
    k = torch.sort(k ^ top).values ^ top  # ascending in the kind's order
    if dist == "reverse":
        return k.flip(0)
    return k[: n // 8 * 8].view(n // 8, 8).t().reshape(-1).contiguous() if n >= 8 else k  # 8 sorted runs


def _items(kind, n, dist, gen):
    """Items as int32 words (u32) or int64 words; pairs carry their index."""
    k = _keys(kind, n, dist, gen)
    if WORDS[kind] < 4:
        return k
    return torch.stack([k, torch.arange(k.numel(), device="cuda", dtype=torch.int64)], dim=1).reshape(-1)


def _lengths(nseg, lo, hi, seed):
    r = np.random.default_rng(seed)
    x = np.floor(np.exp(r.uniform(np.log(lo), np.log(hi + 1), nseg))).astype(np.int64)
    return np.clip(x, lo, hi)


def _host(x, pinned):
    h = torch.empty(x.numel(), dtype=x.dtype, pin_memory=pinned)
    h.copy_(x)
    return h


_NP = {"u32": np.uint32, "u64": np.uint64, "i64": np.int64, "kv64": og.KV_DTYPE, "kvu64": og.KVU_DTYPE}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    form = case["form"]
    s = {"case": case}
    if form in ("sort", "multi"):
        s["src"] = _items(case["kind"], case["n"], case["dist"], gen)
        s["d"], s["tmp"] = torch.empty_like(s["src"]), torch.empty_like(s["src"])
    elif form in ("plan", "segmented"):
        lens = _lengths(case["nseg"], case["lo"], case["hi"], 5)  # a batch slot: the arrays change, their shape stays
        off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
        s["src"] = _items(case["kind"], int(off[-1]), "uniform", gen)
        s["d"], s["tmp"] = torch.empty_like(s["src"]), torch.empty_like(s["src"])
        s["off"] = torch.from_numpy(off).cuda()
        if form == "plan":
            s["plan"] = og.SegmentedPlan(s["d"], s["off"], s["tmp"], kind=case["kind"])
    elif form == "host":
        x = _items(case["kind"], case["n"], case["dist"], gen)
        s["in"], s["out"] = _host(x, case["pinned"]), torch.empty(x.numel(), dtype=x.dtype, pin_memory=case["pinned"])
        s["out"].zero_()
        s["in_np"], s["out_np"] = (s[k].numpy().view(_NP[case["kind"]]) for k in ("in", "out"))
    else:
        r = np.random.default_rng(7)
        kinds = [("u32", "u64", "kvu64")[i] for i in r.choice(3, size=case["requests"], p=[0.5, 0.3, 0.2])]
        lens = _lengths(case["requests"], case["lo"], case["hi"], 11)
        s["requests"] = []
        for i, (k, n) in enumerate(zip(kinds, lens)):
            h = _host(_items(k, int(n), "zipf" if i % 2 else "uniform", gen), True)
            o = torch.empty(h.numel(), dtype=h.dtype, pin_memory=True)
            s["requests"].append((h.numpy().view(_NP[k]), o.numpy().view(_NP[k]), o))
        s["server"] = og.Server(hbm_budget_bytes=16 << 30)
    return s


def run(s):
    case = s["case"]
    form = case["form"]
    if form == "sort":
        s["d"].copy_(s["src"])
        return og.sort(s["d"], s["tmp"], sort_n=case["sort_n"], kind=case["kind"], result_in_tmp=case["in_tmp"])
    if form == "multi":
        s["d"].copy_(s["src"])
        return og.sort_multi_thread(s["d"], s["tmp"], 8, 8, case["min_k"], kind=case["kind"])
    if form == "plan":
        s["d"].copy_(s["src"])
        s["plan"].launch(torch.cuda.current_stream().cuda_stream)
        return s["d"]
    if form == "segmented":
        s["d"].copy_(s["src"])
        return og.sort_segmented(s["d"], s["off"], s["tmp"], kind=case["kind"], sync=False)
    if form == "host":
        og.sort(s["in_np"], s["out_np"], result_in_tmp=True)
        return s["out"]
    server = s["server"]
    ids = [server.submit(x, out=y) for x, y, _ in s["requests"]]
    for i in ids:
        server.wait(i)
    return [o for _, _, o in s["requests"]]


def work(case):
    """Every item read once and written once; a sort computes nothing."""
    form = case["form"]
    if form in ("sort", "multi", "host"):
        return {"bytes": 8 * WORDS[case["kind"]] * case["n"], "flops": 0}
    if form in ("plan", "segmented"):
        n = int(_lengths(case["nseg"], case["lo"], case["hi"], 5).sum())
        return {"bytes": 8 * WORDS[case["kind"]] * n + 8 * (case["nseg"] + 1), "flops": 0}
    r = np.random.default_rng(7)
    words = np.array([1, 2, 4])[r.choice(3, size=case["requests"], p=[0.5, 0.3, 0.2])]
    return {"bytes": int(8 * (words * _lengths(case["requests"], case["lo"], case["hi"], 11)).sum()), "flops": 0}


def exact(case, seed):
    return None  # whole numbers: the outputs stay equal
