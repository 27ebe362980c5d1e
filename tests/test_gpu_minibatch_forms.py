"""The forms in which the ids of a mini-batch are relabelled, and the entry points that reach them: a word per node where
the row count is known, hashed slots for every id where it is not or where a sized context has no room for the
words.  All give the same result, bit for bit, and that of the oracle; so they do on graphs with popular neighbours, where many
lanes lower one word."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

CODE = {torch.int32: 0, torch.int64: 1}


@pytest.fixture(scope="module")
def capi():
    from shmtensor_b200 import capi as mod
    return mod


class _RowsNotKnown:
    """The library with a mini-batch's row count withheld: every id takes a slot."""

    def __init__(self, lib):
        self._lib = lib

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def shmt_minibatch_start(self, ctx, indptr, dtype, n_nodes, *rest):
        return self._lib.shmt_minibatch_start(ctx, indptr, dtype, 0, *rest)


def _by_slots(capi, monkeypatch, *args, **kw):
    with monkeypatch.context() as m:
        m.setattr(capi, "lib", _RowsNotKnown(capi.lib))
        return capi.sample_minibatch(*args, **kw)


def _older_entry(capi, indptr, indices, seeds, fanouts, replace, gpu=(None, None, None, None), eids=False, weights=None,
                 gpu_weights=None):
    """shmt_sample_minibatch, _eids or _weighted, with an output buffer for each piece of each hop."""
    from shmtensor_b200 import _lib
    gpu_indptr, gpu_indices, hmap, base = gpu
    n_hops, dev = len(fanouts), seeds.device
    caps = [seeds.numel()]
    for k in fanouts:
        caps.append(caps[-1] * (1 + k))
    new = lambda n, dt: torch.empty(n, dtype=dt, device=dev)
    sp = [new(caps[h] + 1, indptr.dtype) for h in range(n_hops)]
    sx = [new(caps[h] * fanouts[h], indices.dtype) for h in range(n_hops)]
    ee = [new(caps[h] * fanouts[h], indptr.dtype) for h in range(n_hops)]
    rel, front = ([new(caps[h + 1], indices.dtype) for h in range(n_hops)] for _ in range(2))
    at = lambda ts: (C.c_void_p * n_hops)(*[t.data_ptr() for t in ts])
    ptr = lambda t: None if t is None else t.data_ptr()
    sizes = (C.c_int64 * (3 * n_hops))()
    offset = capi._rng["calls"] + 1
    capi._rng["calls"] += n_hops
    head = (capi._ctx(dev), ptr(indptr), CODE[indptr.dtype], ptr(indices), CODE[indices.dtype])
    handle = hmap._handle if hmap is not None else None
    tail = (ptr(seeds), seeds.numel(), (C.c_int64 * n_hops)(*fanouts), n_hops, int(replace), capi._rng["seed"], offset)
    end = (at(rel), at(front), sizes, capi._stream(dev))
    if eids:
        rc = capi.lib.shmt_sample_minibatch_eids(*head, ptr(gpu_indptr), ptr(gpu_indices), ptr(base), handle, *tail, at(sp),
                                                 at(sx), at(ee), *end)
    elif weights is not None:
        rc = capi.lib.shmt_sample_minibatch_weighted(*head, ptr(weights), ptr(gpu_indptr), ptr(gpu_indices), ptr(gpu_weights),
                                                     handle, *tail, at(sp), at(sx), *end)
    else:
        rc = capi.lib.shmt_sample_minibatch(*head, ptr(gpu_indptr), ptr(gpu_indices), handle, *tail, at(sp), at(sx), *end)
    _lib.check(rc)
    hops = []
    for h in range(n_hops):
        n_in, nnz, n_out = sizes[3 * h:3 * h + 3]
        hop = (sp[h][:n_in + 1], sx[h][:nnz], rel[h][n_in:n_in + nnz], front[h][:n_out])
        hops.append(hop + (ee[h][:nnz],) if eids else hop)
    return hops[-1][3], hops


def _same(a, b):
    assert torch.equal(a[0], b[0]) and len(a[1]) == len(b[1])
    for x, y in zip(a[1], b[1]):
        assert len(x) == len(y) and all(torch.equal(s, t) for s, t in zip(x, y))


def _graph(rng, n, mean, kind, dt):
    deg = rng.integers(0, 2 * mean + 1, size=n)
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    m = int(indptr[-1])
    ids = rng.integers(0, n, size=m)
    if kind == "tenth":
        ids[rng.random(m) < 0.1] = 17
    elif kind == "star":
        ids = rng.integers(0, 3, size=m)
    elif kind == "rank":
        ids = np.minimum((1 + rng.random(m) * (float(n) ** -0.1 - 1)) ** -10.0, n).astype(np.int64) - 1
    elif kind == "beyond":  # half of the ids have no row, the popular one among them
        ids = np.where(rng.random(m) < 0.5, ids, n + ids % 7)
    return indptr, ids.astype(dt)


@pytest.mark.parametrize("dt", [torch.int32, torch.int64])
@pytest.mark.parametrize("kind,fanouts", [("even", (5, 10, 15)), ("tenth", (5, 10, 15)), ("star", (8, 9, 3)), ("rank", (16, 5)),
                                          ("rank", (40, 3)), ("tenth", (4, 33)), ("beyond", (12,)), ("beyond", (40,))])
@pytest.mark.parametrize("n_seeds", [1, 50, 700])
def test_words_slots_and_the_older_entries_agree(capi, monkeypatch, dt, kind, fanouts, n_seeds):
    rng = np.random.default_rng(n_seeds + len(kind))
    n = 5003
    indptr_n, indices_n = _graph(rng, n, 20, kind, np.int32 if dt == torch.int32 else np.int64)
    indptr, indices = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(indices_n).cuda()
    weights = torch.from_numpy(rng.random(indices_n.size).astype(np.float32)).cuda()
    hot = torch.from_numpy(rng.permutation(n)[:1000]).cuda()
    gp, gi = capi.create_subcsr(indptr, indices, hot)
    hmap = capi.CUCOStaticHashmap(hot, torch.arange(1000, device="cuda"), 0.5)
    base = capi.subcsr_edge_base(indptr, hot)
    pos = torch.repeat_interleave(base, gp[1:] - gp[:-1]) + torch.arange(gi.numel(), device="cuda") \
        - torch.repeat_interleave(gp[:-1], gp[1:] - gp[:-1])
    gw = weights[pos]
    assert torch.equal(indices[pos], gi)
    seeds_n = rng.integers(0, n, size=n_seeds).astype(indices_n.dtype)  # repeated ones among them
    seeds = torch.from_numpy(seeds_n).cuda()
    light = all(k <= 32 for k in fanouts)
    for replace in (False, True):
        for option in ("plain", "cached", "eids", "cached eids") + (("weighted", "cached weighted") if light or replace else ()):
            kw, older = {}, {}
            if "cached" in option:
                kw.update(gpu_indptr=gp, gpu_indices=gi, hashmap=hmap)
                older["gpu"] = (gp, gi, hmap, base)
            if "eids" in option:
                kw.update(return_eids=True, gpu_edge_base=base)
                older["eids"] = True
            if "weighted" in option:
                kw.update(weights=weights, gpu_weights=gw)
                older.update(weights=weights, gpu_weights=gw)
            capi.set_sampling_seed(9)
            words = capi.sample_minibatch(indptr, indices, seeds, fanouts, replace, **kw)
            capi.set_sampling_seed(9)
            _same(words, _by_slots(capi, monkeypatch, indptr, indices, seeds, fanouts, replace, **kw))
            capi.set_sampling_seed(9)
            _same(words, _older_entry(capi, indptr, indices, seeds, fanouts, replace, **older))
            cur = seeds_n
            for hop, k in zip(words[1], fanouts):
                sp, sx, rel, front = (t.cpu().numpy() for t in hop[:4])
                if "weighted" not in option:
                    oracle.check_sample_bulk(indptr_n, indices_n, cur, k, replace, sp, sx)
                if "eids" in option:
                    assert np.array_equal(indices_n[hop[4].cpu().numpy()], sx)
                wu, (_, wx) = oracle.tensor_relabel([cur, sx])
                assert np.array_equal(front, wu) and np.array_equal(rel, wx)
                cur = wu
                if kind == "beyond":
                    break  # its ids cannot be sampled from


def test_a_sized_context_without_room_for_the_words_works_by_slots(capi):
    """The words of the graph's nodes take more than all that the context holds, and it does not grow for them."""
    rng = np.random.default_rng(4)
    n = 4_000_000
    deg = np.zeros(n, np.int64)
    some = rng.permutation(n)[:2000]
    deg[some] = rng.integers(1, 9, size=2000)
    indptr_n = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    indices_n = some[rng.integers(0, 2000, size=int(indptr_n[-1]))].astype(np.int32)
    indptr, indices = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(indices_n).cuda()
    seeds_n = some[rng.integers(0, 2000, size=300)].astype(np.int32)
    results = []
    for n_nodes in (0, n):
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            capi.reserve_minibatch(300, [5, 5], n_nodes=n_nodes)
            held = capi.context_scratch_bytes()
            assert (4 * n > held) == (n_nodes == 0)
            capi.set_sampling_seed(3)
            results.append(capi.sample_minibatch(indptr, indices, torch.from_numpy(seeds_n).cuda(), [5, 5]))
            assert capi.context_scratch_bytes() == held
        torch.cuda.synchronize()
    _same(*results)
    cur = seeds_n
    for (sp, sx, rel, front) in results[0][1]:
        oracle.check_sample_bulk(indptr_n, indices_n, cur, 5, False, sp.cpu().numpy(), sx.cpu().numpy())
        wu, (_, wx) = oracle.tensor_relabel([cur, sx.cpu().numpy()])
        assert np.array_equal(front.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wx)
        cur = wu


def test_popular_neighbours_are_no_slower_by_words_than_by_slots(capi, monkeypatch):
    """A tenth of all edges leads to one node: its word must not be lowered once for every one of them.  By slots, which
    leave a smaller index alone, a batch takes 440 us; with a reduction for every edge it took 628 by words, 308 without."""
    n = 2_400_000
    g = torch.Generator(device="cuda").manual_seed(1)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.randint(5, 36, (n,), generator=g, device="cuda"), 0, out=indptr[1:])
    indices = torch.randint(0, n, (int(indptr[-1]),), generator=g, device="cuda")
    indices[torch.rand(indices.numel(), generator=g, device="cuda") < 0.1] = 17
    seeds = torch.randint(0, n, (8192,), generator=g, device="cuda")

    def us(call, reps=10):
        torch.cuda.synchronize()
        t = time.perf_counter()
        for _ in range(reps):
            call()
        torch.cuda.synchronize()
        return (time.perf_counter() - t) / reps * 1e6

    words = lambda: capi.sample_minibatch(indptr, indices, seeds, [5, 10, 15])
    slots = lambda: _by_slots(capi, monkeypatch, indptr, indices, seeds, [5, 10, 15])
    stream = torch.cuda.Stream()  # with a context that no test has sized
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        us(words), us(slots)
        best = [min(us(call) for _ in range(5)) for call in (words, slots)]
    assert best[0] < best[1], best


def test_a_minibatch_that_is_interrupted_is_over(capi, monkeypatch):
    """An exception between the hops leaves no mini-batch behind on the context, and the next one is right."""
    from shmtensor_b200 import _lib
    rng = np.random.default_rng(2)
    indptr_n, indices_n = _graph(rng, 3000, 9, "even", np.int64)
    indptr, indices = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(indices_n).cuda()
    seeds = torch.arange(200, device="cuda")
    capi.set_sampling_seed(5)
    want = capi.sample_minibatch(indptr, indices, seeds, [4, 4, 4])

    class Interrupted:
        def __init__(self, lib, at):
            self.lib, self.at = lib, at

        def __getattr__(self, name):
            return getattr(self.lib, name)

        def shmt_minibatch_hop(self, ctx, hop, sizes):
            if hop == self.at:
                self.at = None
                raise KeyboardInterrupt
            return self.lib.shmt_minibatch_hop(ctx, hop, sizes)

    for at in (0, 1):
        with monkeypatch.context() as m:
            m.setattr(capi, "lib", Interrupted(capi.lib, at))
            with pytest.raises(KeyboardInterrupt):
                capi.sample_minibatch(indptr, indices, seeds, [4, 4, 4])
        assert capi.lib.shmt_minibatch_hop(capi._ctx(seeds.device), 2, (C.c_int64 * 3)()) == _lib.ERR_INVALID
        capi.set_sampling_seed(5)
        _same(want, capi.sample_minibatch(indptr, indices, seeds, [4, 4, 4]))


def test_a_minibatch_is_refused_by_a_stream_that_is_being_captured(capi):
    """With the capture as it was: what else is captured replays, and the context's next mini-batch is right."""
    rng = np.random.default_rng(2)
    indptr_n, indices_n = _graph(rng, 3000, 9, "even", np.int64)
    indptr, indices = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(indices_n).cuda()
    seeds, x = torch.arange(200, device="cuda"), torch.zeros(8, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        capi.set_sampling_seed(5)
        want = capi.sample_minibatch(indptr, indices, seeds, [4, 4])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        x += 1
        with pytest.raises(RuntimeError, match="being captured"):
            capi.sample_minibatch(indptr, indices, seeds, [4, 4])
    graph.replay()
    graph.replay()
    assert (x == 2).all()
    with torch.cuda.stream(stream):
        capi.set_sampling_seed(5)
        _same(want, capi.sample_minibatch(indptr, indices, seeds, [4, 4]))
    torch.cuda.synchronize()
