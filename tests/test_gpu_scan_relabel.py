"""Decoupled look-back scan and first-occurrence relabel against the oracle (bit-exact)."""
import numpy as np
import pytest
import torch

from conftest import load_golden
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from shmtensor_b200 import capi
    return capi


@pytest.mark.parametrize("n", [1, 2, 255, 256, 2047, 2048, 2049, 100_003, 3_000_001])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_scan_matches_cumsum(capi, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randint(-1000, 1000, (n,), generator=g, device="cuda").to(dtype)
    inc, exc = a.clone(), a.clone()
    capi.thrust_scan(inc)
    capi.exclusive_scan_(exc)
    capi.check_async()          # the look-back's bounded waits all completed
    want = oracle.scan_inclusive(a.cpu().numpy())
    assert np.array_equal(inc.cpu().numpy(), want)
    assert np.array_equal(exc.cpu().numpy(), oracle.scan_exclusive(a.cpu().numpy()))


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_scan_tile_edges_views_and_many_tiles(capi, dtype):
    """Lengths around multiples of the 32 KB and 64 KB tiles, ragged tails shorter than 16 bytes,
    views that start off a 16-byte boundary, and enough tiles for every persistent CTA to loop."""
    item = 4 if dtype == torch.int32 else 8
    per32k = 32768 // item
    g = torch.Generator(device="cuda").manual_seed(77)
    big = torch.randint(-50, 50, (24_000_011,), generator=g, device="cuda").to(dtype)
    sizes = [4 * per32k - 1, 4 * per32k, 4 * per32k + 1, 5 * per32k + 3, 16 * per32k + per32k // 2 + 1,
             1000 * per32k + 7 if item == 4 else 700 * per32k + 1, big.numel()]
    for n in sizes:
        for off in (0, 1, 3, 4):
            src = big[off:off + n] if off + n <= big.numel() else big[off:]
            for fn, excl in ((capi.thrust_scan, False), (capi.exclusive_scan_, True)):
                work = big.clone()[off:off + src.numel()]      # a view: same alignment as src
                fn(work)
                want = torch.cumsum(src, 0, dtype=dtype)
                if excl:
                    want = want - src
                assert torch.equal(work, want), (n, off, excl)
    capi.check_async()
    assert capi.device_fault() == 0


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_small_scans_leave_their_state_clean_for_the_next(capi, dtype):
    """Scans of up to 512 tiles use look-back state that the CTA ending last puts back to zero: 400 scans
    queued in a row, from one tile to 512 and back, a tile more or less at a time, each against cumsum."""
    item = 4 if dtype == torch.int32 else 8
    per16k, per64k = 16384 // item, 65536 // item
    top = 512 * per64k if item == 4 else 511 * per64k
    g = torch.Generator(device="cuda").manual_seed(item)
    src = torch.randint(-1000, 1000, (top,), generator=g, device="cuda").to(dtype)
    want = torch.cumsum(src, 0, dtype=dtype)
    sizes = [top, 1, 2 * per16k, per16k, 296 * per16k, 296 * per16k + 1, 296 * 2 * per16k, 296 * 2 * per16k + 1]
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(400):
        n = sizes[i % len(sizes)] if i % 2 else 1 + i * per16k
        n = min(n, top)
        work = src[:n].clone()
        capi.thrust_scan(work)
        wrong += (work != want[:n]).sum()
    capi.check_async()
    assert wrong.item() == 0


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_scan_large_inputs_through_the_cluster_kernel(capi, dtype):
    """From 32 MB on, whole 256 KB super-tiles go through the persistent cluster kernel and the
    rest through the ticketed one, which carries on from the last super-tile's sum: lengths at and
    around super-tile multiples, more super-tiles than resident clusters (every cluster loops),
    inclusive and exclusive, values that wrap in int32."""
    item = 4 if dtype == torch.int32 else 8
    per_super = (256 << 10) // item
    g = torch.Generator(device="cuda").manual_seed(123)
    n_max = 700 * per_super + 12_345
    big = torch.randint(-(2 ** 20), 2 ** 20, (n_max,), generator=g, device="cuda").to(dtype)
    for n in (128 * per_super, 128 * per_super + 1, 129 * per_super - 1, 300 * per_super + 5 * 4096 + 3, n_max):
        for fn, excl in ((capi.thrust_scan, False), (capi.exclusive_scan_, True)):
            work = big[:n].clone()
            fn(work)
            capi.check_async()
            want = torch.cumsum(big[:n], 0, dtype=dtype)
            if excl:
                want = want - big[:n]
            assert torch.equal(work, want), (n, excl)
    assert capi.device_fault() == 0


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_small_scans_leave_their_state_clean_and_replay(capi, dtype):
    """Scans of up to 512 tiles use look-back state that every launch puts back: sizes around the
    16, 32 and 64 KB tiles and the grid sizes at which the tile grows, twice each; the same calls
    captured in a graph give the same result on every replay."""
    item = 4 if dtype == torch.int32 else 8
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [1, 16384 // item - 1, 16384 // item, 16384 // item + 1, 32768 // item + 3]
    sizes += [2 * sms * kb * 1024 // item + d for kb in (16, 32) for d in (-1, 0, 1)] + [512 * 65536 // item - 4]
    g = torch.Generator(device="cuda").manual_seed(5)
    big = torch.randint(-9, 9, (max(sizes) + 1,), generator=g, device="cuda").to(dtype)
    for n in sizes:
        for off in (0, 1):
            for _ in range(2):
                work = big.clone()[off:off + n]
                capi.thrust_scan(work)
                assert torch.equal(work, torch.cumsum(big[off:off + n], 0, dtype=dtype)), (n, off)
    n = 2 * sms * 16384 // item + 5
    work, start = big[:n].clone(), big[:n].clone()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        capi.exclusive_scan_(work)                 # the stream's context exists before the capture
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        work.copy_(start)
        capi.exclusive_scan_(work)
    for _ in range(3):
        work.zero_()
        graph.replay()
        assert torch.equal(work, torch.cumsum(start, 0, dtype=dtype) - start)
    capi.check_async()


def test_scan_int32_wraps_like_the_oracle(capi):
    a = torch.full((5000,), 2**30, dtype=torch.int32, device="cuda")
    want = oracle.scan_inclusive(a.cpu().numpy())
    capi.thrust_scan(a)
    assert np.array_equal(a.cpu().numpy(), want)
    e = torch.empty(0, dtype=torch.int32, device="cuda")
    capi.thrust_scan(e)  # empty input is a no-op
    with pytest.raises(RuntimeError, match="int32 or int64"):
        capi.thrust_scan(torch.zeros(4, device="cuda"))


def test_relabel_golden_vector(capi):
    g = load_golden("relabel.json")
    for dt in (torch.int64, torch.int32):
        ins = [torch.tensor(x, dtype=dt, device="cuda") for x in g["inputs"]]
        uniq, rel = capi.tensor_relabel(ins)
        assert uniq.dtype == dt and uniq.cpu().tolist() == g["unique"]
        assert [r.cpu().tolist() for r in rel] == g["relabel"]
        assert all(r.dtype == dt for r in rel)


@pytest.mark.parametrize("sizes,hi", [((1,), 5), ((1000, 3000), 500), ((5, 0, 7), 4),
                                      ((70_000, 1_200_000), 2_400_000), ((300_000,), 10),
                                      ((2000,) * 9, 3000)])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_relabel_random_matches_oracle(capi, sizes, hi, dtype):
    rng = np.random.default_rng(sum(sizes) + hi)
    ins_n = [rng.integers(0, hi, size=s).astype(np.int64) for s in sizes]
    if dtype == torch.int64:
        ins_n = [x + (1 << 35) for x in ins_n]  # ids beyond 32 bits
    ins = [torch.from_numpy(x).to(dtype).cuda() for x in ins_n]
    uniq, rel = capi.tensor_relabel(ins)
    wu, wr = oracle.tensor_relabel([x.cpu().numpy() for x in ins])
    assert np.array_equal(uniq.cpu().numpy(), wu)
    assert len(rel) == len(sizes)
    for a, b in zip(rel, wr):
        assert np.array_equal(a.cpu().numpy(), b)


def test_relabel_ids_as_slots_and_hashed_ids_share_one_table(capi):
    """Inputs whose table is larger than the cache use the ids themselves as slots when they all fit
    the table, and hash them when one does not (a larger or a negative id); calls of both kinds,
    one after the other on one context, all match the oracle."""
    n, top = 1_500_000, (1 << 22) - 1  # 2^22 slots serve 1,500,000 ids
    rng = np.random.default_rng(9)
    dense = rng.integers(0, 300_000, size=n).astype(np.int64)
    cases = []
    for extra in (top, top + 1, -5, None, 1 << 40, top):
        x = dense.copy()
        rng.shuffle(x)
        if extra is not None:
            x[rng.integers(0, n)] = extra
        cases.append(x)
    for x in cases:
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(x).cuda()])
        wu, (wr,) = oracle.tensor_relabel([x])
        assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    x32 = cases[0].astype(np.int32)
    uniq, rel = capi.tensor_relabel([torch.from_numpy(x32[:700_000]).cuda(), torch.from_numpy(x32[700_000:]).cuda()])
    wu, wr = oracle.tensor_relabel([x32[:700_000], x32[700_000:]])
    assert np.array_equal(uniq.cpu().numpy(), wu)
    assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip(rel, wr))
    # one int32 array of odd length (16-byte loads of the largest-id pass, then a tail), dense and not
    for extra in (None, -7):
        y = np.concatenate([x32, x32[:3]])
        if extra is not None:
            y[-2] = extra
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(y).cuda()])
        wu, (wr,) = oracle.tensor_relabel([y])
        assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    capi.check_async()


@pytest.mark.parametrize("spread", [1, 1_000_003])
def test_relabel_five_million_ids(capi, spread):
    """Inputs of 4 M ids and more take the compact kernel with 4,096-element tiles (and, like every
    input whose table exceeds the cache, the largest-id pass): dense ids (ids as slots) and ids
    spread beyond the table (hashed), with a ragged last tile."""
    rng = np.random.default_rng(77)
    x = rng.integers(0, 2_000_000, size=5_000_123).astype(np.int64) * spread
    uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(x).cuda()])
    wu, (wr,) = oracle.tensor_relabel([x])
    assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    # the table is clean afterwards: a small input right behind it
    y = x[:1000]
    uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(y).cuda()])
    wu, (wr,) = oracle.tensor_relabel([y])
    assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    capi.check_async()


def mix64(x):
    """The 64-bit finaliser of the survey's sample (csrc/common.cuh)."""
    x = x ^ (x >> np.uint64(33))
    x = x * np.uint64(0xff51afd7ed558ccd)
    x = x ^ (x >> np.uint64(33))
    x = x * np.uint64(0xc4ceb9fe1a85ec53)
    return x ^ (x >> np.uint64(33))


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1, (4 << 20) + 4095])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_relabel_around_the_survey_and_tile_limits(capi, n, dtype):
    """More than 2^20 ids are surveyed first (largest id, sampled distinct count) and use a part of
    the table; from 2^22 on tiles are larger.  Few, many and only distinct ids; parts of odd length,
    the second off a 16-byte boundary."""
    rng = np.random.default_rng(n)
    for distinct in (7, n // 5, n):
        ids = rng.permutation(distinct * 3)[:distinct] if distinct < n else rng.permutation(distinct)
        x = ids[rng.integers(0, distinct, size=n)] if distinct < n else ids
        x = x.astype(np.int32 if dtype == torch.int32 else np.int64)
        if dtype == torch.int64 and distinct < n:
            x = x * 0x100000001 + 5                              # hashed, not used as slots
        cut = n // 3 | 1
        whole = torch.from_numpy(x).cuda()
        uniq, rel = capi.tensor_relabel([whole[:cut].clone(), whole[cut:]])
        wu, (wr,) = oracle.tensor_relabel([x])
        assert np.array_equal(uniq.cpu().numpy(), wu)
        assert np.array_equal(torch.cat(rel).cpu().numpy(), wr)
    capi.check_async()


def test_relabel_when_the_survey_sees_far_too_few_ids(capi):
    """Ids picked so that none of them falls into the survey's sample: the part of the table meant
    for them holds almost none, and every id has to find its second home."""
    n = (1 << 20) + 300
    x = np.random.default_rng(3).integers(1 << 30, 1 << 40, size=2 * n).astype(np.int64)
    x = x[mix64(x.astype(np.uint64)) >> np.uint64(62) != 0][:n]   # one id in four is sampled at this size
    assert x.size == n
    for _ in range(2):                                            # the second call finds a clean table
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(x).cuda()])
        wu, (wr,) = oracle.tensor_relabel([x])
        assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    y = x[:5000]
    uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(y).cuda()])
    wu, (wr,) = oracle.tensor_relabel([y])
    assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)


@pytest.mark.parametrize("top_bits", [32, 43, 46, 47, 62])
def test_relabel_in_half_size_slots(capi, top_bits):
    """Two million distinct ids: up to 46 bits they are kept in half-size slots, beyond in ordinary ones;
    repeats near and far, every id twice, then ids on which the table must be found clean."""
    rng = np.random.default_rng(top_bits)
    ids = np.unique(rng.integers(0, 1 << top_bits, size=2_100_000).astype(np.int64))
    ids[-1] = (1 << top_bits) - 1
    rng.shuffle(ids)
    x = np.concatenate([ids, rng.permutation(ids)[:1_234_567], ids[:3]])
    for part in (x, x[::-1].copy(), x[:1_500_001]):
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(part).cuda()])
        wu, (wr,) = oracle.tensor_relabel([part])
        assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    capi.check_async()


def test_the_three_forms_of_the_table_follow_one_another(capi):
    """Ordinary slots, a word per id (dense ids) and half-size slots share one table: calls of every
    form after every other, on the same context, find it empty."""
    rng = np.random.default_rng(31)
    n = 2_000_000
    dense = rng.integers(0, 1_900_000, size=n).astype(np.int64)
    forms = [dense * 0x10000001 % (1 << 43), dense, dense * 0x3000000000001, rng.integers(0, 60_000, size=50_000) + (1 << 33)]
    want = [oracle.tensor_relabel([x]) for x in forms]
    for at in (0, 1, 2, 3, 1, 0, 3, 2, 1, 3, 0, 2, 0):
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(forms[at]).cuda()])
        assert np.array_equal(uniq.cpu().numpy(), want[at][0]) and np.array_equal(rel.cpu().numpy(), want[at][1][0]), at
    capi.check_async()


def test_relabel_when_half_size_slots_run_over(capi):
    """The survey sees less than half of the distinct ids (the others evade its sample), so the
    half-size slots are too few for all of them and some ids go to ordinary slots behind."""
    rng = np.random.default_rng(12)
    x = rng.integers(0, 1 << 42, size=16_000_000).astype(np.int64)
    evading = x[mix64(x.astype(np.uint64)) >> np.uint64(61) != 0][:2_400_000]     # one in 8 is sampled at this size
    x = np.concatenate([x[-1_400_000:], evading])
    rng.shuffle(x)
    x = np.concatenate([x, x[:1000]])
    for _ in range(2):
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(x).cuda()])
        wu, (wr,) = oracle.tensor_relabel([x])
        assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    capi.check_async()


@pytest.mark.parametrize("n", [4097, 300_001, (1 << 20) + 1, 3_000_000])
@pytest.mark.parametrize("share", [0.1, 0.5, 1.0])
def test_relabel_of_ids_that_many_elements_share(capi, n, share):
    """Lanes of a warp that are about to change the same slot, word or survey bit leave it to one of them:
    a few ids take a share of the elements, anywhere among them, in every form of the table (a word per
    id, ordinary slots, half-size slots) and width, the first elements among the shared ones or not."""
    rng = np.random.default_rng(n + int(10 * share))
    few = rng.integers(0, n, size=5)
    x = np.where(rng.random(n) < share, few[rng.integers(0, 5, size=n) // rng.integers(1, 6, size=n)], rng.permutation(n))
    for make in (lambda y: y.astype(np.int32), lambda y: y, lambda y: y * 0x100001, lambda y: y * 0x1000000000 - 7):
        for y in (make(x), make(x)[::-1].copy()):
            uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(y).cuda()])
            wu, (wr,) = oracle.tensor_relabel([y])
            assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)
    capi.check_async()


def unmix_bits(x, bits):
    """The inverse of the mix that gives half-size slots their homes (csrc/relabel.cu, mix_bits)."""
    mask, half = np.uint64((1 << bits) - 1), np.uint64((bits + 1) // 2)
    x = x ^ (x >> half)
    for factor in (0xc4ceb9fe1a85ec53, 0xff51afd7ed558ccd):
        x = (x * np.uint64(pow(factor, -1, 1 << bits))) & mask
        x = x ^ (x >> half)
    return x


def test_relabel_of_ids_made_against_the_half_size_slots(capi):
    """1.5 million distinct ids of 46 bits that all have the same home: 124 fill the places near it, every
    other one goes on to the ordinary slots behind, which hold as many ids as the call has."""
    rng = np.random.default_rng(5)
    low = np.unique(rng.integers(0, 1 << 26, size=1_600_000).astype(np.uint64))[:1_500_000]
    ids = unmix_bits((np.uint64(12_345) << np.uint64(26)) | low, 46).astype(np.int64)   # 2^20 homes
    assert ids.size == 1_500_000 and int(ids.max()).bit_length() == 46
    rng.shuffle(ids)
    x = np.concatenate([ids, ids[:30_000]])
    for part in (x, x[:1_400_000]):
        uniq, (rel,) = capi.tensor_relabel([torch.from_numpy(part).cuda()])
        wu, (wr,) = oracle.tensor_relabel([part])
        assert np.array_equal(uniq.cpu().numpy(), wu) and np.array_equal(rel.cpu().numpy(), wr)


def test_relabel_is_repeatable_and_idempotent(capi):
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randint(0, 100_000, (500_000,), generator=g, device="cuda")
    u1, (r1,) = capi.tensor_relabel([x])
    u2, (r2,) = capi.tensor_relabel([x])
    assert torch.equal(u1, u2) and torch.equal(r1, r2)
    assert torch.equal(u1[r1], x)                       # relabel inverts through unique
    u3, (r3,) = capi.tensor_relabel([u1])               # unique ids relabel to 0..n-1
    assert torch.equal(u3, u1) and torch.equal(r3, torch.arange(u1.numel(), device="cuda"))


def test_relabel_errors(capi):
    with pytest.raises(RuntimeError):
        capi.tensor_relabel([])
    # mixed integer widths are promoted, as the reference's torch::cat does
    u, (a, b) = capi.tensor_relabel([torch.tensor([5, 7], dtype=torch.int64, device="cuda"),
                                     torch.tensor([7, 9], dtype=torch.int32, device="cuda")])
    assert u.dtype == torch.int64 and u.cpu().tolist() == [5, 7, 9]
    assert a.cpu().tolist() == [0, 1] and b.cpu().tolist() == [1, 2]
    with pytest.raises(RuntimeError, match="int32 or int64"):
        capi.tensor_relabel([torch.zeros(2, device="cuda")])
    e = torch.empty(0, dtype=torch.int64, device="cuda")
    u, (r,) = capi.tensor_relabel([e])
    assert u.numel() == 0 and r.numel() == 0


@pytest.mark.parametrize("n, step", [(5000, 1), (1_200_000, 1), (1_200_000, 0x10000001)])
def test_lookback_wait_is_bounded_and_reported(capi, n, step):
    """A look-back whose predecessor never publishes gives up after its spin limit: the host gets
    SHMT_ERR_TIMEOUT, and the same context keeps working afterwards.  The relabel table, which the failed
    call leaves with an index in every slot, is empty again for the next call, whichever form of it that
    uses (ordinary slots, a word per id, slots of ids spread wide)."""
    from shmtensor_b200 import _lib
    x = np.random.default_rng(n).integers(0, n // 3, size=n).astype(np.int64) * step
    wu, (wr,) = oracle.tensor_relabel([x])
    ids = torch.from_numpy(x).cuda()
    capi.tensor_relabel([ids])                                                # the context has its table
    dev = torch.device("cuda", torch.cuda.current_device())
    ctx = capi._ctx(dev)
    rc = _lib.lib.shmt_debug_lookback_timeout(ctx, torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.ERR_TIMEOUT and "bounded look-back wait ran out" in _lib.last_error()
    a = torch.arange(1, 10_001, dtype=torch.int64, device="cuda")
    capi.thrust_scan(a)
    capi.check_async()
    assert a[-1].item() == 50_005_000
    u, (r,) = capi.tensor_relabel([torch.tensor([7, 7, 3], device="cuda")])   # in one CTA, without the table
    assert u.cpu().tolist() == [7, 3] and r.cpu().tolist() == [0, 0, 1]
    u, (r,) = capi.tensor_relabel([ids])                                      # table was re-cleaned
    assert np.array_equal(u.cpu().numpy(), wu) and np.array_equal(r.cpu().numpy(), wr)


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_relabel_in_one_cta_and_just_beyond(capi, n, dtype):
    """Up to 4,096 ids are relabelled by one CTA with 1, 2 or 4 ids per thread: the edges of each,
    all ids equal, all distinct and in between, ids that are negative or beyond 32 bits."""
    rng = np.random.default_rng(n)
    for hi in (1, max(1, n // 3), 1 << 30):
        x = rng.integers(0, hi, size=n).astype(np.int64)
        if hi > 1:
            x[rng.integers(0, n)] = -7
        if dtype == torch.int64:
            x = x * 0x300000001
        x = x.astype(np.int32 if dtype == torch.int32 else np.int64)
        cut = n // 3
        uniq, rel = capi.tensor_relabel([torch.from_numpy(x[:cut]).cuda(), torch.from_numpy(x[cut:]).cuda()])
        wu, (wr,) = oracle.tensor_relabel([x])
        assert uniq.dtype == dtype and np.array_equal(uniq.cpu().numpy(), wu)
        assert np.array_equal(torch.cat(rel).cpu().numpy(), wr)


@pytest.mark.parametrize("n", [4096, 4097, 1 << 20, (1 << 20) + 1, 8_000_001])
@pytest.mark.parametrize("sparse", [False, True])
def test_a_reserved_context_relabels_without_allocating(capi, n, sparse):
    """shmt_ctx_reserve(relabel_ids) covers all that a relabel of so many ids takes (table, look-back
    state and, above 2^20 ids, the survey and a flag bit per id), and of fewer."""
    import ctypes as C

    from shmtensor_b200 import _lib
    lib, check = _lib.lib, _lib.check
    stream = torch.cuda.current_stream().cuda_stream
    x = torch.randint(0, n // 2 + 1, (n,), device="cuda") * (0x10000001 if sparse else 1)
    unique, relabel = torch.empty_like(x), torch.empty_like(x)
    ctx, got = C.c_void_p(), C.c_int64()
    check(lib.shmt_ctx_create(0, C.byref(ctx)))
    try:
        check(lib.shmt_ctx_reserve(ctx, 0, n, stream))
        reserved = lib.shmt_ctx_scratch_bytes(ctx)
        for m in (n, n // 2 + 1, 1000, n):
            check(lib.shmt_relabel(ctx, (C.c_void_p * 1)(x.data_ptr()), (C.c_int64 * 1)(m), 1, _lib.I64,
                                   unique.data_ptr(), relabel.data_ptr(), C.byref(got), stream))
            assert lib.shmt_ctx_scratch_bytes(ctx) == reserved, m
            assert torch.equal(unique[:got.value][relabel[:m]], x[:m])
            assert got.value == torch.unique(x[:m]).numel()
    finally:
        lib.shmt_ctx_destroy(ctx)
