"""Calls issued from different torch streams get different libshmt contexts, so mini-batches,
relabels and scans that overlap on the GPU do not share look-back state, result words or the
relabel table.  Two host threads, one stream each, run mini-batches at the same time; every
result must be a legal sample with the oracle's relabel, exactly as when run alone."""
import threading

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _graph(rng, n, mean_deg):
    deg = np.minimum((rng.pareto(1.3, size=n) * mean_deg / 3).astype(np.int64), 400)
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    indices = np.concatenate([rng.choice(n, size=d, replace=False) for d in deg]).astype(np.int32)
    return indptr, indices


def test_one_context_per_stream():
    from shmtensor_b200 import capi
    dev = torch.device("cuda", 0)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        ca = capi._ctx(dev)
    with torch.cuda.stream(b):
        cb = capi._ctx(dev)
        capi.reserve_minibatch(512, [5, 10, 15])
        assert capi.context_scratch_bytes() >= 16 * (512 * 6 * 11 * 16) // 1024
    assert ca != cb and capi._ctx(dev) not in (ca, cb)
    with torch.cuda.stream(a):
        assert capi._ctx(dev) == ca


def test_minibatches_on_two_streams_at_once():
    from shmtensor_b200 import capi
    rng = np.random.default_rng(8)
    indptr_n, indices_n = _graph(rng, 30_000, 30)
    indptr, indices = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(indices_n).cuda()
    fan = [5, 10, 15]
    results, errors = {}, []

    def worker(tag, seed):
        try:
            stream = torch.cuda.Stream()
            r = np.random.default_rng(seed)
            out = []
            with torch.cuda.stream(stream):
                for _ in range(25):
                    seeds_n = r.integers(0, 30_000, size=700).astype(np.int32)
                    _, hops = capi.sample_minibatch(indptr, indices, torch.from_numpy(seeds_n).cuda(), fan, False)
                    scan = torch.ones(300_000, dtype=torch.int32, device="cuda")
                    capi.thrust_scan(scan)                       # same context, same stream, in between
                    uniq, (rel,) = capi.tensor_relabel([hops[-1][1]])
                    stream.synchronize()
                    out.append((seeds_n, [tuple(t.cpu().numpy() for t in h) for h in hops], scan[-1].item(),
                                uniq.cpu().numpy(), rel.cpu().numpy()))
            results[tag] = out
        except Exception as exc:  # noqa: BLE001
            errors.append((tag, exc))

    threads = [threading.Thread(target=worker, args=(t, 100 + t)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for tag in range(2):
        for seeds_n, hops, scan_last, uniq, rel in results[tag]:
            cur = seeds_n
            for (sp, sx, r, nxt), k in zip(hops, fan):
                oracle.check_sample_bulk(indptr_n, indices_n, cur, k, False, sp, sx, distinct_rows=True)
                wu, (_, wx) = oracle.tensor_relabel([cur, sx])
                assert np.array_equal(nxt, wu) and np.array_equal(r, wx)
                cur = wu
            assert scan_last == 300_000
            wu, (wr,) = oracle.tensor_relabel([hops[-1][1]])
            assert np.array_equal(uniq, wu) and np.array_equal(rel, wr)
    assert capi.device_fault() == 0


@pytest.mark.parametrize("n", [1, 600, 4096])
def test_one_context_goes_from_stream_to_stream(n):
    """A hop hands its result to the host before its kernel ends.  What follows on another stream with
    the same context (up to 512 tiles share look-back state that every kernel leaves at zero) finds
    that state clean: 300 hops on two streams in turn, scans and relabels in between."""
    import ctypes as C

    from shmtensor_b200 import _lib
    lib, check = _lib.lib, _lib.check
    torch.cuda.set_device(0)
    rng = np.random.default_rng(n)
    indptr_n, indices_n = _graph(rng, 20_000, 30)
    indptr, indices = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(indices_n).cuda()
    k, rounds = 10, 300
    seeds_n = rng.integers(0, 20_000, size=n)
    seeds = torch.from_numpy(seeds_n).cuda()
    want = np.concatenate([[0], np.cumsum(np.minimum(indptr_n[seeds_n + 1] - indptr_n[seeds_n], k))])
    sub_indptr = torch.empty(rounds, n + 1, dtype=torch.int64, device="cuda")
    sub_indices = torch.empty(rounds, n * k, dtype=torch.int32, device="cuda")
    unique, relabel = torch.empty(n, dtype=torch.int64, device="cuda"), torch.empty(n, dtype=torch.int64, device="cuda")
    ones = torch.ones(20_001, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    ctx, got = C.c_void_p(), C.c_int64()
    check(lib.shmt_ctx_create(0, C.byref(ctx)))
    try:
        for i in range(rounds):
            s = streams[i & 1].cuda_stream
            check(lib.shmt_sample_hop(ctx, indptr.data_ptr(), _lib.I64, indices.data_ptr(), _lib.I32, None, None, None,
                                      seeds.data_ptr(), _lib.I64, n, k, 0, 7, i, sub_indptr[i].data_ptr(),
                                      sub_indices[i].data_ptr(), C.byref(got), s))
            assert got.value == want[-1], i
            if i % 3 == 2:
                other = streams[~i & 1]
                check(lib.shmt_relabel(ctx, (C.c_void_p * 1)(seeds.data_ptr()), (C.c_int64 * 1)(n), 1, _lib.I64,
                                       unique.data_ptr(), relabel.data_ptr(), C.byref(got), other.cuda_stream))
                assert got.value == np.unique(seeds_n).size, i
                with torch.cuda.stream(other):
                    ones.fill_(1)
                check(lib.shmt_scan(ctx, ones.data_ptr(), _lib.I32, ones.numel(), 0, other.cuda_stream))
                check(lib.shmt_ctx_check(ctx, other.cuda_stream))
                assert ones[-1].item() == ones.numel(), i
        torch.cuda.synchronize()
    finally:
        lib.shmt_ctx_destroy(ctx)
    assert np.array_equal(sub_indptr.cpu().numpy(), np.broadcast_to(want, (rounds, n + 1)))
    for i in (0, 1, rounds - 1):
        oracle.check_sample_bulk(indptr_n, indices_n, seeds_n, k, False, sub_indptr[i].cpu().numpy(),
                                 sub_indices[i, :want[-1]].cpu().numpy(), distinct_rows=True)


def test_a_new_context_waits_for_no_stream():
    """The first call on a stream creates its context; that must not wait for what other streams, the
    default stream among them, still have queued."""
    import ctypes as C

    from shmtensor_b200 import _lib
    torch.cuda.set_device(0)
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(400_000_000)       # about 200 ms
    done.record()
    ctx = C.c_void_p()
    _lib.check(_lib.lib.shmt_ctx_create(0, C.byref(ctx)))
    busy = not done.query()
    torch.cuda.synchronize()
    _lib.check(_lib.lib.shmt_ctx_destroy(ctx))
    assert busy


@pytest.mark.parametrize("dim,dt", [(100, torch.float32), (301, torch.bfloat16), (33, torch.bfloat16)])
def test_lookups_fetches_and_scans_in_a_row_and_captured(dim, dt):
    """These kernels are scheduled while the one before them still runs: each reads what the one before it writes,
    called one after the other and replayed from a graph."""
    from shmtensor_b200 import capi
    g = torch.Generator(device="cuda").manual_seed(dim)
    rows, n = 50_000, 30_011
    hmap = capi.CUCOStaticHashmap(torch.arange(rows, device="cuda"), torch.arange(rows, dtype=torch.int32, device="cuda"), 0.5)
    table = torch.randn(rows, dim, generator=g, device="cuda").to(dt)
    ids = torch.randint(0, rows, (n,), generator=g, device="cuda")
    x = torch.ones(300_001, dtype=torch.int64, device="cuda")

    def step():
        at = (ids * 7 + 3) % rows
        mask = hmap.query(at)
        one = capi.cache_fetch_with_mask(None, table, at, mask)
        two = capi.cache_fetch(None, table, mask.long(), hmap)
        capi.thrust_scan(x)
        capi.thrust_scan(x)
        return at, one, two

    def check(got):
        at, one, two = got
        assert torch.equal(one, table[at]) and torch.equal(two, table[at])
        i = torch.arange(1, x.numel() + 1, device="cuda")
        assert torch.equal(x, i * (i + 1) // 2)

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(20):
            x.fill_(1)
            check(step())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = step()
    for _ in range(10):
        ids.random_(0, rows, generator=g)
        x.fill_(1)
        graph.replay()
        check(got)
