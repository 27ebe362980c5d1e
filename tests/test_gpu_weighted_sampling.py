"""Weighted neighbour sampling (not in the reference, whose sampler is uniform): draws with
replacement follow the weights (chi-square, p > 0.01); draws without replacement have the
inclusion probabilities of sequential weighted sampling without replacement, computed exactly
by enumeration; rows with deg <= k are copied; cached rows behave like host rows."""
import itertools

import numpy as np
import pytest
import torch
from scipy import stats

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from shmtensor_b200 import capi
    capi.set_sampling_seed(4321)
    return capi


def _one_row(weights):
    deg = len(weights)
    indptr = torch.tensor([0, deg], dtype=torch.int64, device="cuda")
    indices = torch.arange(deg, dtype=torch.int32, device="cuda")
    return indptr, indices, torch.tensor(weights, dtype=torch.float32, device="cuda")


@pytest.mark.parametrize("k", [1, 7, 40])
def test_with_replacement_follows_the_weights(capi, k):
    rng = np.random.default_rng(k)
    w = rng.random(50) * 3 + 0.05
    w[7] = 25.0
    indptr, indices, weights = _one_row(w)
    reps = 200_000 // k
    p, x = capi.csr_weighted_sampling(indptr, indices, weights, torch.zeros(reps, dtype=torch.int64, device="cuda"),
                                      k, True)
    assert p[-1].item() == reps * k and x.numel() == reps * k
    counts = np.bincount(x.cpu().numpy(), minlength=50)
    assert stats.chisquare(counts, f_exp=w / w.sum() * counts.sum())[1] > 0.01


def test_a_single_pick_is_proportional_to_its_weight(capi):
    w = np.array([1.0, 2.0, 3.0, 4.0, 10.0, 0.5, 0.5, 1.0, 1.0, 7.0] * 5)   # deg 50 > 32: several chunks
    indptr, indices, weights = _one_row(w)
    reps = 150_000
    _, x = capi.csr_weighted_sampling(indptr, indices, weights, torch.zeros(reps, dtype=torch.int32, device="cuda"),
                                      1, False)
    counts = np.bincount(x.cpu().numpy(), minlength=50)
    assert stats.chisquare(counts, f_exp=w / w.sum() * reps)[1] > 0.01


def test_without_replacement_has_the_sequential_inclusion_probabilities(capi):
    w = np.array([5.0, 1.0, 1.0, 2.0, 0.5, 3.0, 1.0, 0.25, 4.0])
    k = 4
    # exact: P(set) summed over the orders in which sequential draws without replacement produce it
    incl = np.zeros(len(w))
    for seq in itertools.permutations(range(len(w)), k):
        prob, rest = 1.0, w.sum()
        for i in seq:
            prob *= w[i] / rest
            rest -= w[i]
        incl[list(seq)] += prob
    assert abs(incl.sum() - k) < 1e-9
    indptr, indices, weights = _one_row(w)
    reps = 200_000
    p, x = capi.csr_weighted_sampling(indptr, indices, weights, torch.zeros(reps, dtype=torch.int64, device="cuda"),
                                      k, False)
    x = x.cpu().numpy().reshape(reps, k)
    assert (np.sort(x, 1)[:, 1:] != np.sort(x, 1)[:, :-1]).all(), "an edge was picked twice"
    counts = np.bincount(x.reshape(-1), minlength=len(w))
    z = (counts - reps * incl) / np.sqrt(reps * incl * (1 - incl))
    assert (np.abs(z) < 4.5).all(), z


def test_weighted_hop_on_a_cached_graph_with_edge_ids(capi):
    rng = np.random.default_rng(5)
    deg = np.minimum((rng.pareto(1.2, size=3000) * 6).astype(np.int64), 500)
    indptr_n = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    indices_n = np.concatenate([rng.choice(3000, size=d, replace=False) for d in deg]).astype(np.int32)
    w_n = (rng.random(indices_n.size) + 0.01).astype(np.float32)
    indptr, indices, weights = (torch.from_numpy(a).cuda() for a in (indptr_n, indices_n, w_n))
    hot = torch.from_numpy(np.argsort(-deg)[:700].copy()).cuda()
    gp, gi = capi.create_subcsr(indptr, indices, hot)
    _, gw = capi.create_subcsr(indptr, weights.view(torch.int32), hot)
    gw = gw.view(torch.float32)
    base = capi.subcsr_edge_base(indptr, hot)
    hmap = capi.CUCOStaticHashmap(hot, torch.arange(700, device="cuda"), 0.5)
    seeds = torch.from_numpy(rng.integers(0, 3000, size=2500)).cuda()
    from oracle import oracle
    for k, replace in ((5, False), (32, False), (12, True), (48, True)):
        capi.set_sampling_seed(9)
        p, x, e = capi.csr_weighted_sampling(indptr, indices, weights, seeds, k, replace, gp, gi, gw, hmap, base,
                                             return_eids=True)
        capi.set_sampling_seed(9)
        p1, x1 = capi.csr_weighted_sampling(indptr, indices, weights, seeds, k, replace)   # uncached: same draws
        assert torch.equal(p, p1) and torch.equal(x, x1)
        oracle.check_sample_bulk(indptr_n, indices_n, seeds.cpu().numpy(), k, replace, p.cpu().numpy(),
                                 x.cpu().numpy(), distinct_rows=True)
        assert torch.equal(indices[e], x)
    from shmtensor_b200._lib import ShmtError
    with pytest.raises(ShmtError, match="limited to 32"):
        capi.csr_weighted_sampling(indptr, indices, weights, seeds, 33, False)
    with pytest.raises(RuntimeError, match="float32"):
        capi.csr_weighted_sampling(indptr, indices, weights.double(), seeds, 3, False)


def test_heavier_edges_win_more_often_on_long_rows(capi):
    """deg 2,000, fan-out 10: the 20 edges that carry half of the total weight take about half of
    the picks' first-order mass (a loose bound; the exact law is checked on the short row above)."""
    w = np.ones(2000)
    w[:20] = 99.0
    indptr, indices, weights = _one_row(w)
    reps = 20_000
    _, x = capi.csr_weighted_sampling(indptr, indices, weights, torch.zeros(reps, dtype=torch.int64, device="cuda"),
                                      10, False)
    x = x.cpu().numpy().reshape(reps, 10)
    assert (np.sort(x, 1)[:, 1:] != np.sort(x, 1)[:, :-1]).all()
    share = (x < 20).mean()
    assert 0.44 < share < 0.50, share   # sequential draws on the CPU give 0.471


@pytest.mark.parametrize("cached", [False, True])
def test_weighted_minibatch_equals_weighted_hops(capi, cached):
    """shmt_sample_minibatch_weighted: all hops in one native call, the same draws as one
    csr_weighted_sampling + tensor_relabel per hop."""
    rng = np.random.default_rng(11)
    n_nodes = 4000
    deg = np.minimum((rng.pareto(1.2, size=n_nodes) * 6).astype(np.int64), 400)
    indptr_n = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    indices_n = np.concatenate([rng.choice(n_nodes, size=d, replace=False) for d in deg]).astype(np.int32)
    w_n = (rng.random(indices_n.size) + 0.01).astype(np.float32)
    indptr, indices, weights = (torch.from_numpy(a).cuda() for a in (indptr_n, indices_n, w_n))
    gp = gi = gw = hmap = None
    if cached:
        hot = torch.from_numpy(np.argsort(-deg)[:900].copy()).cuda()
        gp, gi = capi.create_subcsr(indptr, indices, hot)
        gw = capi.create_subcsr(indptr, weights.view(torch.int32), hot)[1].view(torch.float32)
        hmap = capi.CUCOStaticHashmap(hot, torch.arange(900, device="cuda"), 0.5)
    for n_seeds, fanouts, replace in ((512, [4, 8, 3], False), (100, [32, 2], False), (300, [6, 40], True)):
        seeds = torch.from_numpy(rng.choice(n_nodes, size=n_seeds, replace=False)).int().cuda()
        capi.set_sampling_seed(31)
        want, cur = [], seeds
        for k in fanouts:
            p, x = capi.csr_weighted_sampling(indptr, indices, weights, cur, k, replace, gp, gi, gw, hmap)
            nxt, (_, rx) = capi.tensor_relabel([cur, x])
            want.append((p, x, rx, nxt))
            cur = nxt
        capi.set_sampling_seed(31)
        frontier, hops = capi.sample_minibatch(indptr, indices, seeds, fanouts, replace, gp, gi, hmap,
                                               weights=weights, gpu_weights=gw)
        assert torch.equal(frontier, cur) and len(hops) == len(fanouts)
        for (p, x, rx, nxt), (p2, x2, rx2, nxt2) in zip(want, hops):
            assert torch.equal(p, p2) and torch.equal(x, x2) and torch.equal(rx, rx2) and torch.equal(nxt, nxt2)
    from shmtensor_b200._lib import ShmtError
    with pytest.raises(ShmtError, match="at most 32"):
        capi.sample_minibatch(indptr, indices, seeds, [33], False, gp, gi, hmap, weights=weights, gpu_weights=gw)
    with pytest.raises(RuntimeError, match="cannot be combined"):
        capi.sample_minibatch(indptr, indices, seeds, [3], False, weights=weights, return_eids=True)
    capi.check_async()


@pytest.mark.parametrize("deg", [33, 127, 128, 129, 1023, 1024, 1025, 1153, 2049, 10_000])
@pytest.mark.parametrize("k", [1, 15, 32])
def test_rows_around_the_length_that_a_whole_cta_shares(capi, deg, k):
    """A row with k edges of overwhelming weight yields exactly those, wherever they lie; one whose
    weights are all zero still yields k different edges; rows of several lengths share a tile."""
    rng = np.random.default_rng(deg * 40 + k)
    degs = np.array([deg, 5, deg, 0, 40, deg + 1])
    indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(degs)])).cuda()
    indices = torch.arange(int(degs.sum()), dtype=torch.int32, device="cuda")
    w = rng.random(int(degs.sum())).astype(np.float32) + 0.01
    heavy = {}
    for row in (0, 5):
        heavy[row] = int(indptr[row]) + rng.choice(degs[row], size=k, replace=False)
        w[heavy[row]] = 1e25
    w[int(indptr[2]):int(indptr[3])] = 0.0
    for _ in range(3):
        p, x = capi.csr_weighted_sampling(indptr, indices, torch.from_numpy(w).cuda(),
                                          torch.arange(6, dtype=torch.int32, device="cuda"), k, False)
        p, x = p.cpu().numpy(), x.cpu().numpy()
        assert np.array_equal(np.diff(p), np.minimum(degs, k))
        for row in range(6):
            got = x[p[row]:p[row + 1]]
            assert np.unique(got).size == got.size
            assert ((got >= int(indptr[row])) & (got < int(indptr[row + 1]))).all()
            if row in heavy:
                assert set(got.tolist()) == set(heavy[row].tolist())
            if degs[row] <= k:
                assert np.array_equal(got, np.arange(int(indptr[row]), int(indptr[row + 1])))


@pytest.mark.parametrize("replace", [False, True])
def test_a_reserved_context_samples_weighted_batches_without_allocating(replace):
    """capi.reserve_minibatch covers weighted hops too, whose tiles hold at most 64 seeds where others
    hold up to 256: look-back state of 62,500 tiles for 4,000,000 seeds."""
    from shmtensor_b200 import capi
    n = 4_000_000
    indptr = torch.arange(1001, device="cuda") * 4
    indices = torch.arange(4000, device="cuda", dtype=torch.int32) % 1000
    weights = torch.rand(4000, device="cuda") + 0.1
    seeds = torch.arange(n, device="cuda", dtype=torch.int32) % 1000
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
        capi.reserve_minibatch(n, [2])
        reserved = capi.context_scratch_bytes()
        front, [(sp, sx, rel, _)] = capi.sample_minibatch(indptr, indices, seeds, [2], replace, weights=weights)
        assert capi.context_scratch_bytes() == reserved
        capi.sample_minibatch(indptr, indices, seeds, [2], replace)
        assert capi.context_scratch_bytes() == reserved
    torch.cuda.synchronize()
    assert sx.numel() == 2 * n and torch.equal(front[rel.long()], sx)


@pytest.mark.parametrize("deg", [1025, 1500, 5000, 10_000])
@pytest.mark.parametrize("k", [1, 7, 32])
def test_a_row_yields_the_same_picks_alone_and_shared(capi, deg, k):
    """Whether the warps of a CTA share a long row depends on the rows it shares a tile with; what is
    drawn for it does not: its place among the seeds decides.  Weights of which many are equal, or zero."""
    rng = np.random.default_rng(deg + k)
    degs = np.concatenate([np.full(8, deg), rng.integers(40, 200, size=8), [deg + 700, 3 * deg]])
    indptr_n = np.concatenate([[0], np.cumsum(degs)])
    indptr = torch.from_numpy(indptr_n).cuda()
    indices = torch.arange(int(indptr_n[-1]), dtype=torch.int32, device="cuda")
    w = torch.from_numpy((rng.integers(0, 4, size=int(indptr_n[-1])) ** 2).astype(np.float32)).cuda()

    def picks(seeds):
        capi.set_sampling_seed(77)
        p, x = capi.csr_weighted_sampling(indptr, indices, w, torch.tensor(seeds, dtype=torch.int32, device="cuda"), k, False)
        return [r.tolist() for r in torch.tensor_split(x.cpu(), p.cpu()[1:-1])]

    crowded = picks(list(range(8)))                              # eight rows of one length: none is shared
    for at in range(8):
        seeds = [8 + j for j in range(8)]
        seeds[at] = at
        assert picks(seeds)[at] == crowded[at]                   # one long row among short ones: shared
        seeds[(at + 3) % 8], seeds[(at + 6) % 8] = 16, 17
        assert picks(seeds)[at] == crowded[at]                   # among the longer ones of three
    assert picks([0])[0] == crowded[0]                           # and on its own
    assert len({tuple(r) for r in crowded}) == 8 and all(len(set(r)) == k for r in crowded)


@pytest.mark.parametrize("k", [1, 4, 5, 15, 31, 32])
def test_the_k_heavy_edges_win_wherever_they_lie(capi, k):
    """k edges outweigh the others by more than any two clocks differ (2^-24 to 17, against 10^30), so they
    are the picks exactly: candidates sorted 32 or 128 at a time, several sorts a row where the light edges
    grow heavier along it, rows shared by a CTA and not, and fan-outs small enough to be picked one by one."""
    rng = np.random.default_rng(k)
    deg = np.array([k + 1, 32, 33, 64, 127, 128, 129, 159, 161, 500, 1000, 1024, 1025, 3000, 9000])
    deg = np.maximum(deg, k + 1)
    indptr_n = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    w = np.empty(indptr_n[-1], np.float32)
    heavy = []
    for b, d in zip(indptr_n, deg):
        w[b:b + d] = 1e-20 * (1 + np.arange(d)) ** 2
        at = rng.choice(d, size=k, replace=False)
        if d > 40:
            at = np.concatenate([[d - 1], at[at != d - 1]])[:k] if d % 2 else at
        w[b + at] = np.float32(1e20) * (1 + rng.random(k)).astype(np.float32)
        heavy.append(np.sort(at))
    indptr, weights = torch.from_numpy(indptr_n).cuda(), torch.from_numpy(w).cuda()
    indices = torch.from_numpy(np.concatenate([np.arange(d) for d in deg]).astype(np.int32)).cuda()
    for n in (1, 15, 600):
        seeds_n = rng.integers(0, deg.size, size=n) if n != 15 else np.arange(deg.size)
        p, x = capi.csr_weighted_sampling(indptr, indices, weights, torch.from_numpy(seeds_n).cuda(), k, False)
        got = np.sort(x.cpu().numpy().reshape(n, k), 1)
        assert np.array_equal(got, np.stack([heavy[s] for s in seeds_n]))
        assert np.array_equal(p.cpu().numpy(), np.arange(n + 1) * k)
