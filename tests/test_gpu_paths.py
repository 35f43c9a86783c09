"""GPU tests of kernels at the edges of their tiles and dispatch rules, bit-exact against the
oracle or a plain numpy statement of the same result."""
import numpy as np
import pytest
import torch

import oracle
import redzone_b200 as rz

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.fixture(scope="module")
def ctx():
    c = rz.Context(0)
    yield c
    c.close()


def payload(n: int, words: int, seed: int) -> np.ndarray:
    return np.random.default_rng(seed).integers(0, 1 << 32, size=(n, words), dtype=np.uint64).astype(np.uint32)


def on_gpu(a: np.ndarray):
    return torch.from_numpy(a.view(np.int32).copy()).to(DEV)


@pytest.mark.parametrize("words", [1, 2, 4, 8])
@pytest.mark.parametrize("m", [1, 255, 1023, 1024, 1025, 5000])
def test_keep_in_two_kernels(ctx, words, m):
    """rz_keep around one 1024-item block: entries on both sides of m (items kept from [0, m) go
    through the scratch), the same row several times, one entry past the end."""
    n = 5001
    rng = np.random.default_rng(m * 8 + words)
    host = payload(n, words, seed=m)
    keep = rng.integers(0, n, size=m).astype(np.uint32)
    keep[:: 3] = rng.integers(0, m, size=keep[:: 3].size)
    d = on_gpu(host)
    assert ctx.keep(d, on_gpu(keep), flags=rz.RZ_SYNC) == m
    got = d.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[:m], host[keep]) and np.array_equal(got[m:], host[m:])
    keep[m // 2] = n
    d = on_gpu(host)
    with pytest.raises(rz.RedzoneError):
        ctx.keep(d, on_gpu(keep), flags=rz.RZ_SYNC)
    exp = host[np.minimum(keep, n - 1)]
    exp[m // 2] = host[m // 2]
    assert np.array_equal(d.cpu().numpy().view(np.uint32)[:m], exp)


@pytest.mark.parametrize("n,k,place", [(511, 40, "spread"), (512, 512, "spread"), (513, 1, "end"), (70001, 3000, "spread"),
                                       (1 << 20, 60000, "run"), ((1 << 20) + 77, 60000, "run"), (4099, 0, "spread")])
@pytest.mark.parametrize("shift", [0, 1])
def test_produced_rows_of_the_key_filter(ctx, n, k, place, shift):
    """rz_produce_where_less emits exactly the rows below the threshold: around one warp step (512
    keys), runs long enough that blocks collect more rows than their buffer holds, keys off the
    16-byte boundary (shift), and the removal agrees with rz_remove on the list it wrote."""
    rng = np.random.default_rng(n + k)
    rows = {"spread": lambda: rng.choice(n, size=k, replace=False), "run": lambda: np.arange(n // 3, n // 3 + k),
            "end": lambda: np.arange(n - k, n)}[place]()
    keys = np.full(n + shift, 900, np.uint32)
    keys[shift + rows] = 100
    d_keys = on_gpu(keys)[shift:]
    p = rz.Producer(ctx, capacity=max(1, k + 5))
    p.reset(n)
    p.produce_where_less(d_keys, 500)
    lst, kk, _ = p.download()
    assert kk == k and np.array_equal(np.sort(lst), np.sort(rows).astype(np.uint32))
    host = payload(n, 1, seed=n)
    a, b = on_gpu(host), on_gpu(host)
    assert p.remove(a, flags=rz.RZ_SYNC) == n - k
    if k:
        ctx.remove(b, on_gpu(lst), flags=rz.RZ_SYNC)
    assert torch.equal(a, b)


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 100003])
@pytest.mark.parametrize("share", [2, 255, 257, 4000])
def test_validation_both_ways(ctx, n, share):
    """RZ_VALIDATE with lists long and short for their n (map zeroed as a whole / entry by entry): a
    valid list passes, also after one with a duplicate or an entry past the end (or both), which is
    reported and moves nothing."""
    k = max(1, n // share)
    rng = np.random.default_rng(n + share)
    host = payload(n, 1, seed=n)
    good = rng.choice(n, size=k, replace=False).astype(np.uint32)
    bad = []
    if k > 1:
        dup = good.copy()
        dup[-1] = dup[0]
        bad.append((dup, 2))
    out = good.copy()
    out[k // 2] = n
    bad.append((out, 3))
    if k > 2:
        both = out.copy()
        both[0] = both[k - 1]
        bad.append((both, 3))
    for idx, code in bad:
        d = on_gpu(host)
        with pytest.raises(rz.RedzoneError) as e:
            ctx.remove(d, on_gpu(idx), flags=rz.RZ_VALIDATE | rz.RZ_SYNC)
        assert e.value.code == code
        assert np.array_equal(d.cpu().numpy().view(np.uint32), host)
        d = on_gpu(host)
        assert ctx.remove(d, on_gpu(good), flags=rz.RZ_VALIDATE | rz.RZ_SYNC) == n - k
        exp = host.copy()
        oracle.remove(exp, good)
        assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], exp[: n - k])


@pytest.mark.parametrize("words", [1, 8])
@pytest.mark.parametrize("n_tiles,extra", [(1, -3), (1, 0), (8, 0), (8, 1), (9, 0), (600, 17), (1191, 5)])
def test_partition_runs_of_tiles(ctx, words, n_tiles, extra):
    """The partition's tiles are counted in runs: sizes around one tile, one run (8 tiles, or 3 at
    about 1200) and a last run that is cut short; an aligned list (pipelined move) and, for 4-byte
    items, one that is not; validated and not; twice on the same context."""
    n = n_tiles * (32768 // (4 * words)) + extra
    k = n // 7
    rng = np.random.default_rng(n + words)
    host = payload(n, words, seed=n)
    idx = rng.choice(n, size=k, replace=False).astype(np.uint32)
    exp = np.delete(host, idx.astype(np.int64), axis=0)
    d_idx = on_gpu(idx)
    for flags in (rz.RZ_SYNC, rz.RZ_SYNC | rz.RZ_VALIDATE):
        d = on_gpu(host)
        assert ctx.partition(d, d_idx, flags=flags) == n - k
        assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], exp)
    if words == 1:
        room = torch.zeros((n + 1, 1), dtype=torch.int32, device=DEV)
        room[1:] = on_gpu(host)
        assert ctx.partition(room[1:], d_idx, flags=rz.RZ_SYNC) == n - k
        assert np.array_equal(room[1: n - k + 1].cpu().numpy().view(np.uint32), exp)


@pytest.mark.parametrize("words", [2, 4, 8])
@pytest.mark.parametrize("n,k", [(1, 1), (300, 300), (5000, 257), (70000, 20000)])
def test_remove_by_key_after_refused_calls(ctx, words, n, k):
    """rz_remove_by_key after calls that were refused (a key twice, a missing and a reserved key, on
    the same index): those change neither table nor index and let go of their slots, and the good
    call that follows gives the oracle's table and an index that is exact; erased keys can be
    inserted and deleted again."""
    rng = np.random.default_rng(n * 8 + words)
    host = payload(n, words, seed=k)
    keys = rng.permutation(np.arange(1, 2 * n + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15))[:n]
    host[:, :2] = keys.view(np.uint32).reshape(n, 2)
    table = on_gpu(host)
    ix = rz.KeyIndex(ctx, 2 * n)
    ix.build(table)
    pick = rng.choice(n, size=k, replace=False).astype(np.uint32)

    def dev(a):
        return torch.from_numpy(a.view(np.int64).copy()).to(DEV)

    wrong = [(np.concatenate([keys[pick[:-1]], np.array([7], np.uint64)]), 3),
             (np.concatenate([keys[pick[:-1]], np.array([2**64 - 1], np.uint64)]), 3)]
    if k > 1:
        wrong.append((np.concatenate([keys[pick[:-1]], keys[pick[:1]]]), 2))
    for bad, code in wrong:
        with pytest.raises(rz.RedzoneError) as e:
            ix.remove_by_key(table, n, dev(bad))
        assert e.value.code == code
    assert np.array_equal(table.cpu().numpy().view(np.uint32), host)
    assert np.array_equal(ix.find(dev(keys)).cpu().numpy(), np.arange(n))
    assert ix.remove_by_key(table, n, dev(keys[pick])) == n - k
    exp = host.copy()
    oracle.remove(exp, pick)
    got = table.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[: n - k], exp[: n - k])
    left = np.ascontiguousarray(exp[: n - k, :2]).view(np.uint64).reshape(-1)
    if n > k:
        assert np.array_equal(ix.find(dev(left)).cpu().numpy(), np.arange(n - k))
    assert (ix.find(dev(keys[pick])).cpu().numpy() == -1).all()
    table[n - k:] = on_gpu(host)[torch.from_numpy(pick.astype(np.int64)).to(DEV)]
    ix.insert(table, n - k, k)
    assert ix.remove_by_key(table, n, dev(keys[pick]), flags=rz.RZ_SYNC) == n - k
    assert np.array_equal(table.cpu().numpy().view(np.uint32)[: n - k], exp[: n - k])
    ix.close()


@pytest.mark.parametrize("k", [700, 20000])
def test_capture_after_copies_and_joins(ctx, k):
    """Removals that may start before the kernel ahead of them has ended, captured behind a copy
    (rz_append_remove), behind kernels that write their list, and behind a join with another stream;
    the graph is replayed with other lists and every result is the oracle's."""
    n, g = 100000, 300
    rng = np.random.default_rng(k)
    host, gain = payload(n + g, 2, seed=k), payload(g, 2, seed=k + 1)
    one = [rng.choice(n + g, size=k, replace=False).astype(np.uint32) for _ in range(3)]
    two = [rng.choice(n + g - k, size=k, replace=False).astype(np.uint32) for _ in range(3)]
    start, d, d_gain = on_gpu(host), on_gpu(host), on_gpu(gain)
    all_one, all_two = on_gpu(np.stack(one)), on_gpu(np.stack(two))
    idx_one, idx_two = torch.zeros((2, 1, k), dtype=torch.int32, device=DEV)
    pick = torch.zeros(1, dtype=torch.int64, device=DEV)
    ctx.append_remove(d, n, d_gain, all_one[0])  # the context's scratch grows outside the capture
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        here = torch.cuda.current_stream()
        d.copy_(start)
        torch.index_select(all_one, 0, pick, out=idx_one)
        ctx.append_remove(d, n, d_gain, idx_one)
        side.wait_stream(here)
        with torch.cuda.stream(side):
            torch.index_select(all_two, 0, pick, out=idx_two)
        here.wait_stream(side)
        ctx.remove(d[: n + g - k], idx_two)
    for q in (0, 2, 1):
        pick.fill_(q)
        graph.replay()
        assert ctx.sync_status() == 0
        exp = host.copy()
        exp[n:] = gain
        oracle.remove(exp, one[q])
        left = exp[: n + g - k].copy()
        oracle.remove(left, two[q])
        assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n + g - 2 * k], left[: n + g - 2 * k])


@pytest.mark.parametrize("k", [300, 4096, 9000, 60000])
def test_back_to_back_removals_on_one_list(ctx, k):
    """Each call reads what the one before it wrote, with nothing between them (and kernels of other
    shapes in between): 20 removals from one shrinking list."""
    n = 1 << 21
    rng = np.random.default_rng(k)
    host = payload(n, 1, seed=k)
    d, exp, m = on_gpu(host), host.copy(), n
    lists = []
    for _ in range(20):
        lists.append(rng.choice(m, size=k, replace=False).astype(np.uint32))
        m -= k
    d_lists = [on_gpu(x) for x in lists]
    torch.cuda.synchronize()
    m = n
    for q, x in enumerate(d_lists):
        ctx.remove(d[:m], x, flags=rz.RZ_FORCE_GRID if q % 7 == 3 else 0)
        m -= k
    assert ctx.sync_status() == 0
    m = n
    for x in lists:
        left = exp[:m].copy()
        oracle.remove(left, x)
        m -= k
        exp = left
    assert np.array_equal(d.cpu().numpy().view(np.uint32)[:m], exp[:m])


@pytest.mark.parametrize("words", [1, 4])
@pytest.mark.parametrize("k,red", [(4100, 0), (4100, 33), (8200, 300), (8200, 1024), (16385, 1025), (20001, 2100),
                                   (65536, 9000), (65535, 65000), (131072, 1500)])
def test_cluster_scan_over_red_counts(ctx, words, k, red):
    """Cluster scan with red entries in every amount its paths divide by (32, one block's threads, 256
    per slice, 1024 in all, more), spread over the list and crowded in its first slice; slices that
    end inside a warp's rounds."""
    n = 4 * k
    rng = np.random.default_rng(k + red)
    host = payload(n, words, seed=red)
    reds = rng.choice(k, size=red, replace=False) + (n - k)
    holes = rng.choice(n - k, size=k - red, replace=False)
    for crowded in (False, True):
        idx = np.concatenate([reds, holes]).astype(np.uint32)
        if not crowded:
            rng.shuffle(idx)
        d = on_gpu(host)
        assert ctx.remove(d, on_gpu(idx), flags=rz.RZ_SYNC) == n - k
        exp = host.copy()
        oracle.remove(exp, idx)
        assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], exp[: n - k]), crowded


BULK = rz.LaunchCfg(256, 4, 4, 0, 7)


@pytest.mark.parametrize("k,gap", [(1, 2), (33, 5), (4096, 40), (8191, 5), (8192, 64), (8193, 9), (100003, 6),
                                   (303105, 11), (1 << 20, 17)])
@pytest.mark.parametrize("dist", ["uniform", "runs", "tail", "most"])
def test_bulk_schedule(ctx, k, gap, dist):
    """The bulk schedule at the edges of its tiles and buckets: spread holes, runs of 256, holes in one
    part of the list (done by the grid kernel), nearly all entries red; index lists off 16 bytes; with
    validation, and twice in a row on one context."""
    n = k * gap + 7
    rng = np.random.default_rng(k + gap)
    if dist == "uniform":
        idx = rng.permutation(n)[:k]
    elif dist == "runs":
        starts = rng.permutation(n // 256 + 1)[: k // 256 + 1]
        idx = (starts[:, None] * 256 + np.arange(256)).ravel()
        idx = np.concatenate([idx[idx < n], np.setdiff1d(np.arange(n), idx)])[:k]
        rng.shuffle(idx)
    elif dist == "tail":
        idx = n - 1 - rng.permutation(min(n, 2 * k))[:k]
    else:
        idx = np.concatenate([np.arange(n - k, n - k // 8), rng.permutation(n - k)[: k // 8]])
        rng.shuffle(idx)
    idx = idx.astype(np.uint32)
    host = payload(n, 1, seed=k)
    exp = host.copy()
    oracle.remove(exp, idx)
    room = on_gpu(np.concatenate([np.zeros(1, np.uint32), idx]))
    for d_idx, flags in ((room[1:], 0), (on_gpu(idx), rz.RZ_VALIDATE)):
        d = on_gpu(host)
        ctx.remove_cfg(d, d_idx, BULK, flags=flags | rz.RZ_SYNC)
        assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], exp[: n - k]), flags


def test_bulk_schedule_refusals_limits_and_capture():
    """A list that fails validation changes nothing and the next call is exact; without its scratch
    memory, and in a capture that finds none, the grid schedule runs instead; a capture that finds
    the scratch replays the bulk schedule on other lists."""
    n, k = 400001, 20011
    rng = np.random.default_rng(3)
    host = payload(n, 1, seed=3)
    lists = [rng.permutation(n)[:k].astype(np.uint32) for _ in range(3)]
    exps = []
    for idx in lists:
        exps.append(host.copy())
        oracle.remove(exps[-1], idx)
    c = rz.Context(0)
    start, d, d_idx = on_gpu(host), on_gpu(host), on_gpu(lists[0])

    def check(q):
        assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], exps[q][: n - k])

    def capture():
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            d.copy_(start)
            c.remove_cfg(d, d_idx, BULK)
        return graph, c.last_launch()[0]

    c.remove_cfg(d, d_idx, rz.LaunchCfg(256, 4, 4, 0, 3), flags=rz.RZ_SYNC)
    check(0)
    c.set_scratch_limit(0)
    d.copy_(start)
    c.remove_cfg(d, d_idx, BULK, flags=rz.RZ_SYNC)
    assert c.last_launch()[0] == 1
    check(0)
    c.set_scratch_limit(None)
    assert capture()[1] == 1
    for at, val, code in ((5, None, 2), (k - 1, n + 9, 3)):
        bad = lists[0].copy()
        bad[at] = bad[at + 1] if val is None else val
        d.copy_(start)
        with pytest.raises(rz.RedzoneError) as e:
            c.remove_cfg(d, on_gpu(bad), BULK, flags=rz.RZ_VALIDATE | rz.RZ_SYNC)
        assert e.value.code == code
        assert torch.equal(d, start)
    graph, launches = capture()
    assert launches == 6
    for q in (1, 2, 0):
        d_idx.copy_(on_gpu(lists[q]))
        graph.replay()
        assert c.sync_status() == 0
        check(q)
    c.close()


def test_bulk_schedule_is_the_default_for_long_lists(ctx):
    """Default launch at the first size of the bulk schedule and one item below it, against the grid
    schedule: 3 * 2^22 of 2^27 int32."""
    n = 1 << 27
    g = torch.Generator(device=DEV).manual_seed(5)
    start = torch.arange(n, dtype=torch.int32, device=DEV).view(-1, 1)
    idx_all = torch.randperm(n, device=DEV, generator=g)[: 3 << 22].to(torch.int32)
    for k, bulk in ((3 << 22, True), ((3 << 22) - 1, False)):
        idx, out = idx_all[:k].contiguous(), []
        for cfg in (None, rz.LaunchCfg(896, 4, 2, 0, 3)):
            d = start.clone()
            if cfg is None:
                ctx.remove(d, idx, flags=rz.RZ_SYNC)
                assert (ctx.last_launch()[0] == 6) is bulk
            else:
                ctx.remove_cfg(d, idx, cfg, flags=rz.RZ_SYNC)
            out.append(d[: n - k])
        assert torch.equal(*out)
        del out, d
    torch.cuda.empty_cache()


@pytest.mark.parametrize("words", [1, 4])
@pytest.mark.parametrize("k,gap", [((1 << 17) + 1, 64), (163840, 64), (163841, 64), (163840, 63)])
def test_grid_shape_between_2e17_and_160k(ctx, words, k, gap):
    """Grid schedule with 512-thread CTAs: its first and last k and the next one, and a list too short for it."""
    n = k * gap
    host = payload(n, words, seed=k)
    idx = np.random.default_rng(gap).permutation(n)[:k].astype(np.uint32)
    d = on_gpu(host)
    assert ctx.remove(d, on_gpu(idx), flags=rz.RZ_SYNC) == n - k
    assert ctx.last_launch()[2] == (512 if k <= 163840 and gap == 64 else 896)
    oracle.remove(host, idx)
    assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], host[: n - k])


@pytest.mark.parametrize("k,cut", [(524289, 0), (524289, 1), (524300, 31), (600000, 32), (524321, 100003), (1048575, 3000017)])
def test_validation_marks_the_red_zone(ctx, k, cut):
    """Long validated lists take the red zone's marks from the validation's map: cuts on and off its
    words, everything removed, removals from the tail alone; also after a list that was refused, with
    one tile per CTA, and without validation right after."""
    n = k + cut
    rng = np.random.default_rng(k)
    host = payload(n, 2, seed=cut)
    for tail in (False, True):
        idx = rng.permutation(n)[:k] if not tail else n - 1 - rng.permutation(min(n, k + k // 3))[:k]
        idx = idx.astype(np.uint32)
        exp = host.copy()
        oracle.remove(exp, idx)
        for bad_val, code in ((idx[1], 2), (n + 5, 3)):
            bad = idx.copy()
            bad[0] = bad_val
            d = on_gpu(host)
            with pytest.raises(rz.RedzoneError) as e:
                ctx.remove(d, on_gpu(bad), flags=rz.RZ_VALIDATE | rz.RZ_SYNC)
            assert e.value.code == code
            assert np.array_equal(d.cpu().numpy().view(np.uint32), host)
        for cfg, flags in ((None, rz.RZ_VALIDATE), (rz.LaunchCfg(512, 8, 2, 0, 3), rz.RZ_VALIDATE), (None, 0)):
            d = on_gpu(host)
            if cfg is None:
                ctx.remove(d, on_gpu(idx), flags=flags | rz.RZ_SYNC)
            else:
                ctx.remove_cfg(d, on_gpu(idx), cfg, flags=flags | rz.RZ_SYNC)
            assert np.array_equal(d.cpu().numpy().view(np.uint32)[:cut], exp[:cut]), (tail, cfg, flags)


@pytest.mark.parametrize("order", ["sorted", "runs", "sorted in turn", "random"])
def test_default_route_of_long_lists_by_their_order(ctx, order):
    """3 * 2^22 of 2^27 int32: the default's result is the grid schedule's, and it takes no more than a fifth
    longer where a list's neighbours lie together (the grid kernel's stores share lines there; bulk takes
    1.5 to 2 times as long), and less where they do not."""
    n, k = 1 << 27, 3 << 22
    g = torch.Generator(device=DEV).manual_seed(9)
    if order == "runs":
        starts = torch.randperm(n // 256, device=DEV, generator=g)[: k // 256]
        idx = (starts[:, None] * 256 + torch.arange(256, device=DEV)).reshape(-1)
    else:
        idx = torch.randperm(n, device=DEV, generator=g)[:k]
        if order != "random":
            idx = idx.sort().values
        if order == "sorted in turn":
            idx = idx.view(4, -1).t().reshape(-1)
    idx = idx.to(torch.int32)
    start = torch.arange(n, dtype=torch.int32, device=DEV).view(-1, 1)
    out, us = [], []
    for cfg in (None, rz.LaunchCfg(1024, 4, 2, 0, 3)):
        def call():
            return ctx.remove(d, idx) if cfg is None else ctx.remove_cfg(d, idx, cfg)
        d = start.clone()
        call()
        assert ctx.sync_status() == 0
        out.append(d[: n - k].clone())
        best = 1e9
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        us.append(best)
    assert torch.equal(*out)
    assert us[0] < (1.2 if order != "random" else 0.85) * us[1], us
    del start, d, idx, out
    torch.cuda.empty_cache()


def test_bulk_scratch_grows_with_the_lists_only():
    """A context whose orphan lists have room for k removals takes the bulk schedule's scratch for k at its
    first bulk call: later calls up to k leave it where it is, so a captured call stays right."""
    c = rz.Context(0)
    n, k0, k1 = 3000001, 200003, 20011
    rng = np.random.default_rng(8)
    wide = torch.zeros((n, 2), dtype=torch.int32, device=DEV)
    c.remove_cfg(wide, on_gpu(rng.permutation(n)[:k0].astype(np.uint32)), rz.LaunchCfg(256, 4, 4, 0, 3), flags=rz.RZ_SYNC)
    host = payload(n, 1, seed=8)
    lists = {k: rng.permutation(n)[:k].astype(np.uint32) for k in (k1, k0)}
    exps = {}
    for k, idx in lists.items():
        exps[k] = host.copy()
        oracle.remove(exps[k], idx)
    start, d, d_idx = on_gpu(host), on_gpu(host), on_gpu(lists[k1])
    c.remove_cfg(d, d_idx, BULK, flags=rz.RZ_SYNC)
    held = c.scratch_bytes
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        d.copy_(start)
        c.remove_cfg(d, d_idx, BULK)
    assert c.last_launch()[0] == 6
    e = start.clone()
    c.remove_cfg(e, on_gpu(lists[k0]), BULK, flags=rz.RZ_SYNC)
    assert c.last_launch()[0] == 6 and c.scratch_bytes == held
    assert np.array_equal(e.cpu().numpy().view(np.uint32)[: n - k0], exps[k0][: n - k0])
    graph.replay()
    assert c.sync_status() == 0
    assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k1], exps[k1][: n - k1])
    c.close()


def test_bulk_schedule_without_memory_for_its_scratch():
    """With the GPU's memory taken, calls that would be bulk run the grid schedule and do not try the
    allocation each time (a failing one takes 0.5 to 1.5 ms, these calls 0.5)."""
    c = rz.Context(0)
    n, k = 1 << 26, 1 << 24
    d = torch.arange(n, dtype=torch.int32, device=DEV).view(-1, 1)
    idx = torch.randperm(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2))[:k].to(torch.int32)
    torch.cuda.empty_cache()
    want = d.clone()
    c.remove_cfg(want, idx, rz.LaunchCfg(1024, 4, 2, 0, 3), flags=rz.RZ_SYNC)
    torch.cuda.synchronize()
    taken = []
    size = torch.cuda.mem_get_info()[0] - (96 << 20)
    while size > 16 << 20 and torch.cuda.mem_get_info()[0] > 112 << 20:
        try:
            taken.append(torch.empty(min(size, torch.cuda.mem_get_info()[0] - (96 << 20)), dtype=torch.uint8, device=DEV))
        except torch.OutOfMemoryError:
            size //= 2
    try:
        cfg = rz.LaunchCfg(1024, 4, 2, 0, 7)
        c.remove_cfg(d, idx, cfg, flags=rz.RZ_SYNC)
        assert c.last_launch()[0] == 1 and torch.equal(d[: n - k], want[: n - k])
        ms = []
        for cf in (rz.LaunchCfg(1024, 4, 2, 0, 3), cfg):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                c.remove_cfg(d, idx, cf, flags=rz.RZ_SYNC)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        assert ms[1] < 1.5 * ms[0], ms
    finally:
        del taken, d, want, idx
        torch.cuda.empty_cache()
        c.close()


@pytest.mark.parametrize("k", [(1 << 18) - 1, 1 << 18, (1 << 21) + 5])
def test_partition_of_long_validated_lists(ctx, k):
    """The validated mark on both sides of 2^18 entries: the stable result twice in a row, a duplicate and
    an entry past the end reported, and the calls after them."""
    n = 2 * k + 77
    rng = np.random.default_rng(k)
    host = payload(n, 1, seed=k)
    idx = rng.permutation(n)[:k].astype(np.uint32)
    exp = np.delete(host, idx.astype(np.int64), axis=0)
    for bad_at in (None, idx[1], n, None):
        bad = idx.copy()
        if bad_at is not None:
            bad[0] = bad_at
        d = on_gpu(host)
        if bad_at is None:
            for _ in range(2):
                d = on_gpu(host)
                assert ctx.partition(d, on_gpu(bad), flags=rz.RZ_SYNC | rz.RZ_VALIDATE) == n - k
                assert np.array_equal(d.cpu().numpy().view(np.uint32)[: n - k], exp)
        else:
            with pytest.raises(rz.RedzoneError) as e:
                ctx.partition(d, on_gpu(bad), flags=rz.RZ_SYNC | rz.RZ_VALIDATE)
            assert e.value.code == (3 if bad_at == n else 2)


def test_partition_validation_of_half_a_list_costs_less_than_the_rest(ctx):
    """2^23 of 2^24 int32: validated partitions back to back take less than 1.65 times plain ones (1.35; 1.95
    when the mark runs in the shared memory split of the kernel ahead)."""
    n, k = 1 << 24, 1 << 23
    d = torch.zeros((n, 1), dtype=torch.int32, device=DEV)
    idx = torch.randperm(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4))[:k].to(torch.int32)
    best = {}
    for flags in (0, rz.RZ_VALIDATE) * 4:
        ctx.partition(d, idx, flags=flags)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            ctx.partition(d, idx, flags=flags)
        b.record()
        b.synchronize()
        best[flags] = min(best.get(flags, 1e9), a.elapsed_time(b))
    assert ctx.sync_status() == 0
    assert best[rz.RZ_VALIDATE] < 1.65 * best[0], best


@pytest.mark.parametrize("words,shift", [(1, 0), (2, 0), (4, 0), (8, 0), (8, 4)])
@pytest.mark.parametrize("share", ["wide", "sparse", "edge", "next", "half", "most", "all"])
def test_keep_of_long_lists(ctx, words, shift, share):
    """rz_keep in a list of 192 MiB, the first size with 64-byte loads, around 64 bytes per kept item where
    they end, at 2^20 items and a sixteenth (16-byte items: a 32nd) where they stay out of L1, and around
    seven eighths where all items are staged: any order, rows given twice, an entry past the end, 32-byte
    items on and off 32 bytes."""
    n = ((544 if share == "sparse" else 192) << 20) // (4 * words)
    m = {"wide": n // 1000, "sparse": n // (32 if words == 4 else 16), "edge": n * 4 * words // 64,
         "next": n * 4 * words // 64 + 1, "half": n // 2 + 1,
         "most": n - n // 8, "all": n - n // 8 + 1}[share]
    if m > n:
        pytest.skip("more than there are")
    g = torch.Generator(device=DEV).manual_seed(m)
    room = torch.randint(-(1 << 31), (1 << 31) - 1, (n * words + 8,), device=DEV, generator=g, dtype=torch.int64).to(torch.int32)
    d = room[shift: shift + n * words].view(n, words)
    keep = torch.randint(0, n, (m,), device=DEV, generator=g)
    keep[::3] = torch.randint(0, m, (keep[::3].numel(),), device=DEV, generator=g)
    exp = d[keep]
    rest = d[m:].clone()
    keep = keep.to(torch.int32)
    keep[m // 3] = -5  # 2^32 - 5: past the end, the slot keeps its own item
    exp[m // 3] = d[m // 3]
    with pytest.raises(rz.RedzoneError) as e:
        ctx.keep(d, keep, flags=rz.RZ_SYNC)
    assert e.value.code == 3
    assert torch.equal(d[:m], exp) and torch.equal(d[m:], rest)
    del room, d, keep, exp, rest
    torch.cuda.empty_cache()


def test_keep_of_all_items_without_order(ctx):
    """2^24 int32, all of them kept: in random order 1.8 times the time of sorted ones (2.8 with loads that
    ask for 64 bytes and leave nothing in L1)."""
    n = 1 << 24
    d = torch.arange(n, dtype=torch.int32, device=DEV).view(-1, 1)
    keep = torch.randperm(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(6)).to(torch.int32)
    us = []
    for k in (keep, torch.arange(n, dtype=torch.int32, device=DEV)):
        best = 1e9
        for _ in range(5):
            ctx.keep(d, k)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                ctx.keep(d, k)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        us.append(best)
    assert ctx.sync_status() == 0
    assert us[0] < 2.3 * us[1], us


def test_validation_of_a_tail_clears_a_big_map_by_entry(ctx):
    """2^20 validated removals from the last tenth of 255 * 2^20 int32 (a map of 32 MB, cleared entry by entry) and of
    127 * 2^20 (half the map, zeroed as a whole): the result of an unchecked call, a list with a duplicate refused
    in between, and the longer list takes 1.15 times as long (1.37 with its map zeroed)."""
    k, us = 1 << 20, []
    g = torch.Generator(device=DEV).manual_seed(3)
    for n in (255 << 20, 127 << 20, 1 << 27, (1 << 27) + 1):
        d = torch.arange(n, dtype=torch.int32, device=DEV).view(-1, 1)
        idx = (n - 1 - torch.randperm(n // 10, device=DEV, generator=g)[:k]).to(torch.int32)
        bad = idx.clone()
        bad[5] = bad[6]
        for _ in range(2):
            with pytest.raises(rz.RedzoneError) as e:
                ctx.remove(d, bad, flags=rz.RZ_VALIDATE | rz.RZ_SYNC)
            assert e.value.code == 2
        want = d.clone()
        ctx.remove_cfg(want, idx, rz.LaunchCfg(1024, 4, 2, 0, 3), flags=rz.RZ_SYNC)
        ctx.remove(d, idx, flags=rz.RZ_VALIDATE | rz.RZ_SYNC)
        assert torch.equal(d[: n - k], want[: n - k])
        best = 1e9
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                ctx.remove(d, idx, flags=rz.RZ_VALIDATE)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        us.append(best)
        del d, want, idx, bad
    torch.cuda.empty_cache()
    assert us[0] < 1.26 * us[1], us


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("n,k", [(40, 39), (5000, 300), (9001, 4000), (70000, 9000), (600001, 70000), (600001, 200003),
                                 (1600008, 200001), (1600007, 200001)])
def test_32_byte_items_on_and_off_whole_sectors(ctx, n, k, shift):
    """32-byte items in a list on 32 bytes (whole-sector stores, or halves in dense lists) and 16 bytes off (always
    two stores): every schedule, a validated call, keep, partition, a produced list and a batch; dense and
    sparse around n = 8 k."""
    rng = np.random.default_rng(n + k)
    host = payload(n, 8, seed=k)
    idx = rng.permutation(n)[:k].astype(np.uint32)
    exp = host.copy()
    oracle.remove(exp, idx)
    d_idx, start = on_gpu(idx), on_gpu(host).reshape(-1)
    room = torch.zeros(n * 8 + 8, dtype=torch.int32, device=DEV)
    d = room[shift: shift + n * 8].view(n, 8)

    def check(call, want=exp[: n - k]):
        room.fill_(7)
        d.copy_(start.view(n, 8))
        call()
        got = d[: want.shape[0]].cpu().numpy().view(np.uint32)
        assert np.array_equal(got, want)
        edge = torch.cat([room[:shift], room[shift + n * 8:]])
        assert (edge == 7).all()

    check(lambda: ctx.remove(d, d_idx, flags=rz.RZ_SYNC))
    check(lambda: ctx.remove(d, d_idx, flags=rz.RZ_SYNC | rz.RZ_VALIDATE))
    for sched in (1, 2, 3, 4, 5, 6, 7):
        if sched == 1 and k > 20000:
            continue
        for items in (1, 4):
            check(lambda: ctx.remove_cfg(d, d_idx, rz.LaunchCfg(256, items, 2, 0, sched), flags=rz.RZ_SYNC))
    check(lambda: ctx.partition(d, d_idx, flags=rz.RZ_SYNC), np.delete(host, idx.astype(np.int64), axis=0))
    check(lambda: ctx.keep(d, d_idx, flags=rz.RZ_SYNC), host[idx])
    if k <= 1 << 18:
        keys = np.full(n, 900, np.uint32)
        keys[idx] = 1
        p = rz.Producer(ctx, capacity=k)
        d_keys = on_gpu(keys)

        def produced():
            p.reset(n)
            p.produce_where_less(d_keys, 500)
            p.remove(d, flags=rz.RZ_SYNC)

        room.fill_(7)
        d.copy_(start.view(n, 8))
        produced()
        want = host.copy()
        oracle.remove(want, p.download()[0])
        assert np.array_equal(d[: n - k].cpu().numpy().view(np.uint32), want[: n - k])
    room.fill_(7)
    d.copy_(start.view(n, 8))
    plan = rz.BatchPlan(ctx, [(d, d_idx)])
    plan.launch()
    torch.cuda.synchronize()
    plan.close()
    assert np.array_equal(d[: n - k].cpu().numpy().view(np.uint32), exp[: n - k])


@pytest.mark.parametrize("n,k,dense", [(1 << 24, 1 << 21, 3), (50000017, 1 << 24, 0), (50000017, (1 << 24) - 5, 2)])
def test_bulk_schedule_beyond_one_tile(ctx, n, k, dense):
    """Buckets of several fill tiles (holes three times as dense in a 32nd of the list, which the sample does not
    call crowded) and blocks with more than one tile of orphans to pair (a third of the list removed), against
    the grid schedule."""
    g = torch.Generator(device=DEV).manual_seed(k)
    idx = torch.randperm(n, device=DEV, generator=g)
    if dense:
        lo, hi = n // 4, n // 4 + n // 32
        inside = (idx >= lo) & (idx < hi)
        share = min(dense * (k / n), 0.95)
        many = idx[inside][: int(share * (hi - lo))]
        idx = torch.cat([many, idx[~inside][: k - many.numel()]])
        idx = idx[torch.randperm(idx.numel(), device=DEV, generator=g)]
    idx = idx[:k].to(torch.int32)
    start = torch.arange(n, dtype=torch.int32, device=DEV).view(-1, 1)
    a, b = start.clone(), start
    ctx.remove_cfg(a, idx, BULK, flags=rz.RZ_SYNC)
    assert ctx.last_launch()[0] == 6
    ctx.remove_cfg(b, idx, rz.LaunchCfg(1024, 4, 2, 0, 3), flags=rz.RZ_SYNC)
    assert torch.equal(a[: n - k], b[: n - k])
    del idx, start, a, b
    torch.cuda.empty_cache()
