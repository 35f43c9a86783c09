"""Measured cases: removals as programs make them, through the package's public entry points.

Each case names an entry point (``kind``) and its sizes. Payloads are 4, 8, 16 or 32-byte items;
removal lists are distinct positions in random order, drawn uniformly, as runs of 256 consecutive
positions (``clustered``) or from the last tenth of the list (``tail``) -- the distributions of the
benchmark's sweep. Every pass edits its list in place, so passes on one state follow one another
the way repeated removals from a program's list do.
"""
from __future__ import annotations

import math

import torch

import redzone_b200 as rz

DEVICE = "cuda"
RUN = 256  # length of a clustered run


def listed():
    return [
        # The smallest calls: a few hundred rows out of a short list (launch latency counts).
        {"name": "remove_small", "kind": "remove", "n": 65521, "k": 1000, "w": 8, "dist": "uniform", "validate": False},
        # The benchmark's headline: 2^16 rows out of 2^28 int32.
        {"name": "remove_headline", "kind": "remove", "n": 1 << 28, "k": 1 << 16, "w": 4, "dist": "uniform",
         "validate": False},
        # Records of 16 bytes deleted in runs (time ranges, sessions); sizes off every power of two.
        {"name": "remove_clustered_16B", "kind": "remove", "n": 33554393, "k": 400009, "w": 16, "dist": "clustered",
         "validate": False},
        # A large sweep of int32 rows: the upper part of the k range, where the hole writes count.
        {"name": "remove_bulk", "kind": "remove", "n": 1 << 28, "k": 1 << 24, "w": 4, "dist": "uniform",
         "validate": False},
        # Recent rows of a time-ordered table, from a list that is not trusted (checked first).
        {"name": "remove_tail_checked", "kind": "remove", "n": 50000017, "k": 2000003, "w": 8, "dist": "tail",
         "validate": True},
        # The reference's host call: index list in host memory, new length back.
        {"name": "host_index", "kind": "host", "n": 1 << 28, "k": 1 << 16, "w": 4, "dist": "uniform"},
        # Order-preserving compaction of a whole list.
        {"name": "partition", "kind": "partition", "n": 100000007, "k": 9999991, "w": 4, "dist": "uniform"},
        # The inverse form: keep a few of many 16-byte records, given by a sorted list.
        {"name": "keep", "kind": "keep", "n": 33554393, "k": 2097143, "w": 16, "sorted": True},
        # A filter kernel that decides on the GPU which rows go, and their removal.
        {"name": "produced", "kind": "produced", "n": 1 << 26, "k": 32749, "w": 8},
        # A keyed table: delete by key, add as many records, look keys up.
        {"name": "keyed", "kind": "keyed", "n": 4194301, "k": 65521, "w": 32},
        # Many uneven lists in one launch of a kept plan (n log-uniform in [2^8, 2^22], k/n to 0.5).
        {"name": "batched", "kind": "batched", "lists": 1024, "lo": 8.0, "hi": 22.0, "w": 8},
        # The delete service: a burst of host batches (1 to 2^20 rows) over the shards of a table.
        {"name": "service", "kind": "service", "shards": 16, "capacity": 1 << 22, "batches": 64, "hi": 20.0, "w": 32},
    ]


def _log_int(rng, lo, hi):
    """An integer whose logarithm is uniform in [lo, hi]; odd ones as often as even ones."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["remove"] * 6 + ["host", "partition", "keep", "produced", "keyed", "batched", "service"])
    w = rng.choice([4, 8, 16, 32])
    if kind in ("remove", "host", "partition"):
        n = _log_int(rng, 1 << 14, (1 << 30) // w if w > 4 else 1 << 28)
        dist = rng.choice(["uniform", "clustered", "tail"])
        top = n // 10 if dist == "tail" else n // 4
        k = _log_int(rng, 64, min(top, 1 << (24 if kind != "host" else 18)))
        c = {"kind": kind, "n": n, "k": k, "w": w, "dist": dist}
        if kind == "remove":
            c["validate"] = rng.random() < 0.25
        return c
    if kind == "keep":
        n = _log_int(rng, 1 << 16, (1 << 30) // w)
        return {"kind": kind, "n": n, "k": _log_int(rng, 1 << 10, min(n // 4, 1 << 23)), "w": w,
                "sorted": rng.random() < 0.7}
    if kind == "produced":
        n = _log_int(rng, 1 << 18, (1 << 30) // w if w > 8 else 1 << 27)
        return {"kind": kind, "n": n, "k": _log_int(rng, 1 << 6, min(n // 512, 1 << 17)), "w": w}
    if kind == "keyed":
        w = rng.choice([8, 16, 32])
        n = _log_int(rng, 1 << 14, 1 << 23)
        return {"kind": kind, "n": n, "k": _log_int(rng, 1 << 8, n // 16), "w": w}
    if kind == "batched":
        hi = rng.uniform(14.0, 21.0)
        return {"kind": kind, "lists": _log_int(rng, 32, 1024), "lo": rng.uniform(6.0, 10.0), "hi": hi, "w": w}
    return {"kind": kind, "shards": rng.choice([4, 8, 16]), "capacity": _log_int(rng, 1 << 17, 1 << 21),
            "batches": _log_int(rng, 8, 96), "hi": rng.uniform(10.0, 16.0), "w": w}


def _distinct(g, lo, hi, k):
    """k distinct positions of [lo, hi), uniform, in random order (int64)."""
    span = hi - lo
    if 4 * k > span:
        return torch.randperm(span, generator=g, device=DEVICE)[:k] + lo
    u = torch.unique(torch.randint(lo, hi, (k + k // 2 + 64,), generator=g, device=DEVICE))
    while u.numel() < k:
        u = torch.unique(torch.cat([u, torch.randint(lo, hi, (k,), generator=g, device=DEVICE)]))
    return u[torch.randperm(u.numel(), generator=g, device=DEVICE)[:k]]


def _positions(g, dist, n, k):
    if dist == "uniform":
        p = _distinct(g, 0, n, k)
    elif dist == "tail":
        p = _distinct(g, n - n // 10, n, k)
    else:  # runs of RUN positions that do not overlap; the last one is cut short at random places
        m = -(-k // RUN)
        if m * RUN > n:
            raise ValueError("runs do not fit")
        y = torch.sort(torch.randint(0, n - m * RUN + 1, (m,), generator=g, device=DEVICE)).values
        starts = y + RUN * torch.arange(m, device=DEVICE)
        p = (starts[:, None] + torch.arange(RUN, device=DEVICE)).reshape(-1)
        p = p[torch.randperm(p.numel(), generator=g, device=DEVICE)[:k]]
    return p.to(torch.int32)


def _items(g, n, w):
    shape = (n,) if w == 4 else (n, w // 4)
    return torch.randint(-(1 << 31), (1 << 31) - 1, shape, dtype=torch.int32, generator=g, device=DEVICE)


def _batched_sizes(case, seed):
    """Sizes of the lists; their total depends on the case alone, their order on the seed."""
    m, lo, hi = case["lists"], case["lo"], case["hi"]
    g = torch.Generator().manual_seed(seed)
    n = [max(2, round(2 ** (lo + (hi - lo) * (q + 0.5) / m))) for q in range(m)]
    f = [0.001 + 0.499 * ((q * 0.6180339887498949) % 1.0) for q in range(m)]
    k = [max(1, min(ni - 1, round(fi * ni))) for ni, fi in zip(n, f)]
    order = torch.randperm(m, generator=g).tolist()
    return [n[q] for q in order], [k[q] for q in order]


def _batch_rows(case):
    """Rows of the service's batches: log-uniform in [1, 2^hi], at most a quarter of a shard."""
    m = case["batches"]
    return [max(1, min(case["capacity"] // 4, round(2 ** (case["hi"] * ((q * 0.6180339887498949) % 1.0)))))
            for q in range(m)]


def prepare(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    kind, w = case["kind"], case["w"]
    ctx = rz.default_context()
    s = {"kind": kind, "ctx": ctx}
    if kind in ("remove", "host", "partition"):
        s["data"] = _items(g, case["n"], w)
        s["idx"] = _positions(g, case["dist"], case["n"], case["k"])
        # A checked list is one whose status the program wants before it goes on.
        s["flags"] = rz.RZ_VALIDATE | rz.RZ_SYNC if case.get("validate") else 0
        if kind == "host":
            s["idx"] = s["idx"].cpu().pin_memory()
    elif kind == "keep":
        s["data"] = _items(g, case["n"], w)
        p = _distinct(g, 0, case["n"], case["k"])
        s["keep"] = (torch.sort(p).values if case["sorted"] else p).to(torch.int32)
    elif kind == "produced":
        n, k = case["n"], case["k"]
        s["data"] = _items(g, n, w)
        keys = torch.randint(1 << 30, (1 << 31) - 1, (n,), dtype=torch.int32, generator=g, device=DEVICE)
        rows = _distinct(g, 0, n, k)
        keys[rows] = torch.randint(0, 1 << 30, (k,), dtype=torch.int32, generator=g, device=DEVICE)
        s["keys"], s["threshold"], s["n"] = keys, 1 << 30, n
        s["producer"] = rz.Producer(ctx, capacity=k + k // 4, cand_capacity=4096)
    elif kind == "keyed":
        n, k = case["n"], case["k"]
        table = _items(g, n, w)
        keys = (torch.arange(1, n + 1, dtype=torch.int64, device=DEVICE) + (seed << 24)) * 0x1E3779B97F4A7C15
        table[:, :2] = keys.view(torch.int32).view(n, 2)
        s["keys"] = keys[_distinct(g, 0, n, k)].contiguous()
        fresh = _items(g, k, w)  # the records that take the deleted ones' place: same keys, new payload
        fresh[:, :2] = s["keys"].view(torch.int32).view(k, 2)
        # Half of the keys looked up are in the table, half are not.
        probe = keys[torch.randint(0, n, (k,), generator=g, device=DEVICE)]
        s["probe"] = torch.where(torch.rand(k, generator=g, device=DEVICE) < 0.5, probe, probe ^ (1 << 62)).contiguous()
        s["index"] = rz.KeyIndex(ctx, 2 * n)
        s["index"].build(table)
        s["table"], s["fresh"], s["n"] = table, fresh, n
    elif kind == "batched":
        ns, ks = _batched_sizes(case, seed)
        s["data"] = _items(g, sum(ns), w)
        lists, at = [], 0
        for n, k in zip(ns, ks):
            idx = torch.randperm(n, generator=g, device=DEVICE)[:k].to(torch.int32)
            lists.append((s["data"][at: at + n], idx))
            at += n
        s["lists"] = lists
        s["plan"] = rz.BatchPlan(ctx, lists)
    else:
        cap, shards = case["capacity"], case["shards"]
        floor = cap // 2
        s["table"] = _items(g, cap * shards, w)
        # Rows below the floor are live whenever a batch runs: a shard is refilled before it
        # would fall below it.
        s["batches"] = [_distinct(g, 0, floor, k).to(torch.int32).cpu().pin_memory() for k in _batch_rows(case)]
        s["shards"] = shards
        s["service"] = rz.Service(ctx, s["table"], shards, cap, floor_rows=floor)
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "remove":
        return s["data"][:ctx.remove(s["data"], s["idx"], flags=s["flags"])]
    if kind == "host":
        return s["data"][:ctx.remove_host_idx(s["data"], s["idx"])]
    if kind == "partition":
        return s["data"][:ctx.partition(s["data"], s["idx"])]
    if kind == "keep":
        return s["data"][:ctx.keep(s["data"], s["keep"])]
    if kind == "produced":
        p = s["producer"]
        p.reset(s["n"])
        p.produce_where_less(s["keys"], s["threshold"])
        return s["data"][:p.remove(s["data"], flags=rz.RZ_SYNC)]
    if kind == "keyed":
        left = s["index"].remove_by_key(s["table"], s["n"], s["keys"])
        s["table"][left:] = s["fresh"]
        s["index"].insert(s["table"], left, s["n"] - left)
        return {"table": s["table"], "rows": s["index"].find(s["probe"])}
    if kind == "batched":
        s["plan"].launch()
        return s["data"]
    svc = s["service"]
    for q, idx in enumerate(s["batches"]):
        svc.submit(q % s["shards"], idx, borrow=True)
    svc.drain()
    return {"table": s["table"], "lengths": torch.tensor(svc.lengths()[0])}


def _removal_bytes(n, k, w, dist="uniform"):
    """Index list read, surviving tail items read, holes written."""
    zone = n // 10 if dist == "tail" else n
    red = k * min(1.0, k / zone)
    return 4 * k + 2 * w * (k - red)


def work(case):
    kind, w = case["kind"], case["w"]
    if kind in ("remove", "host"):
        b = _removal_bytes(case["n"], case["k"], w, case["dist"])
    elif kind == "partition":
        b = case["n"] * w + (case["n"] - case["k"]) * w + 4 * case["k"]
    elif kind == "keep":
        b = case["k"] * (4 + 2 * w)
    elif kind == "produced":
        b = 4 * case["n"] + 4 * case["k"] + _removal_bytes(case["n"], case["k"], w)
    elif kind == "keyed":
        # Removal of the rows; the list of keys, one index entry (key and row) each for the delete,
        # the insert and the lookup, and one for each row that moved; the new records; the answers.
        k = case["k"]
        b = _removal_bytes(case["n"], k, w) + 8 * k + 4 * 12 * k + 2 * w * k + (8 + 8) * k
    elif kind == "batched":
        b = sum(_removal_bytes(n, k, w) for n, k in zip(*_batched_sizes(case, 0)))
    else:
        b = sum(_removal_bytes(case["capacity"], k, w) for k in _batch_rows(case))
    return {"bytes": float(b), "flops": 0.0}
