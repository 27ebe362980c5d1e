"""What the host does with the context of a mini-batch, on a runtime that runs nothing (fake_runtime.py): the memory
that a context keeps, a mini-batch that nobody waits for, and a stream that is being captured."""
import ctypes as C

import pytest

import fake_runtime
from shmtensor_b200 import _lib

N_IDS = 100_000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_runtime.load(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def ctx(lib):
    out = C.c_void_p()
    assert lib.shmt_ctx_create(0, C.byref(out)) == _lib.OK
    yield out.value
    lib.fake_capture(0)
    lib.shmt_ctx_destroy(out.value)


def _buffer(nbytes):
    return (C.c_char * (nbytes + 16))()


def _start(lib, ctx, n_nodes, n_seeds=100, k=5):
    edges = n_seeds * k
    pools = _buffer(64), _buffer(64), _buffer(64)  # nothing runs, so nothing is read or written
    layout = (C.c_int64 * 5)(0, 0, 0, edges, 2 * edges + n_seeds)
    some = C.addressof(pools[2])
    return lib.shmt_minibatch_start(ctx, some, _lib.I64, n_nodes, some, _lib.I64, None, None, None, None, None, None, some,
                                    n_seeds, (C.c_int64 * 1)(k), 1, 0, 1, 1, C.addressof(pools[0]), C.addressof(pools[1]),
                                    layout, 0, None)


def _relabel(lib, ctx, n=N_IDS):
    ids, unique, local = (_buffer(8 * n) for _ in range(3))
    return lib.shmt_relabel(ctx, (C.c_void_p * 1)(C.addressof(ids)), (C.c_int64 * 1)(n), 1, _lib.I64,
                            C.addressof(unique), C.addressof(local), None, None)


@pytest.mark.parametrize("n_nodes", [0, 3, 2_000_000, 1 << 25])
def test_a_minibatch_moves_no_memory_that_a_sized_context_holds(lib, ctx, n_nodes):
    """A relabel that was captured in a sized context keeps the addresses of its table: a mini-batch within that size may
    add memory for its words, and gives none back."""
    assert lib.shmt_ctx_reserve(ctx, 1 << 20, N_IDS, None) == _lib.OK
    assert _relabel(lib, ctx) == _lib.OK
    lib.fake_reset()
    for _ in range(3):
        assert _start(lib, ctx, n_nodes) == _lib.OK
        assert _relabel(lib, ctx) == _lib.OK
    assert lib.fake_frees() == 0


@pytest.mark.parametrize("reserved_for,sampled,slots", [(0, 900_000, False), (1000, 900_000, False), (1000, 3_000_000, True),
                                                        (3_000_000, 3_000_000, False), (1 << 26, 900_000, False)])
def test_a_context_sized_for_one_graph_has_words_for_another_that_is_not_much_larger(lib, ctx, reserved_for, sampled, slots):
    """At least as many as fit in what a small table's block is short of 4 MB."""
    fan = (C.c_int64 * 1)(5)
    assert lib.shmt_ctx_reserve_minibatch_nodes(ctx, 100, fan, 1, reserved_for, None) == _lib.OK
    held = lib.shmt_ctx_scratch_bytes(ctx)
    lib.fake_reset()
    assert _start(lib, ctx, 0) == _lib.OK
    by_slots = lib.fake_last_kernel()  # numbers the repeats, which are numbered otherwise where there are words
    assert _start(lib, ctx, sampled) == _lib.OK
    assert (lib.fake_last_kernel() == by_slots) == slots
    assert lib.shmt_ctx_scratch_bytes(ctx) == held and lib.fake_frees() == 0


def test_words_start_over_when_all_numbers_are_used(lib, ctx):
    """A hop takes as many numbers as it can have ids, here 2,020,000 of 2^32 - 1: 2,126 batches go by between two fills of
    the words, in the first lap and in the next."""
    lib.fake_reset()
    words, sizes = lib.fake_host_words(), (C.c_int64 * 3)()
    for batch in range(1, 2 * 2126 + 2):
        assert _start(lib, ctx, 1_000_000, 20_000, 100) == _lib.OK
        words[8], words[127] = 0, batch  # handed over, without an error
        assert lib.shmt_minibatch_hop(ctx, 0, sizes) == _lib.OK
        if batch % 2126 <= 1:
            table = lib.fake_fills(0xFF, 16_000_000)
            assert table == 1 and lib.fake_fills(0xFF, 4_000_000) - table == 1 + (batch - 1) // 2126


TIMEOUT = 2


@pytest.mark.parametrize("status,fails", [(0, False), (TIMEOUT, True), (1, True), (None, True)])
@pytest.mark.parametrize("between", [(), (1000,)])
def test_a_minibatch_that_nobody_waits_for_leaves_no_entries(lib, ctx, status, fails, between):
    """A mini-batch that failed may have left entries in the table.  If nobody asks for its sizes the next call that uses
    the table empties it: the status is read when the mini-batch is given up, before a small call's (`between`) results come
    over it, and a mini-batch that never handed it over counts as failed."""
    assert lib.shmt_ctx_reserve(ctx, 1 << 20, N_IDS, None) == _lib.OK
    assert _start(lib, ctx, 2_000_000) == _lib.OK
    if status is not None:
        words = lib.fake_host_words()
        words[1], words[3], words[8], words[127] = 500, 600, status, 1  # edges, distinct ids, status, the first post
    lib.fake_reset()
    for n in between:
        found = C.c_int64()
        ids, unique, local = (_buffer(8 * n) for _ in range(3))
        assert lib.shmt_relabel(ctx, (C.c_void_p * 1)(C.addressof(ids)), (C.c_int64 * 1)(n), 1, _lib.I64, C.addressof(unique),
                                C.addressof(local), C.byref(found), None) == _lib.OK
    assert _relabel(lib, ctx) == _lib.OK
    assert (lib.fake_largest_fill(0xFF) >= 16 * N_IDS) == fails
    sizes = (C.c_int64 * 3)()
    assert lib.shmt_minibatch_hop(ctx, 0, sizes) == _lib.ERR_INVALID  # it is over
    lib.fake_reset()
    assert _start(lib, ctx, 2_000_000) == _lib.OK
    assert (lib.fake_largest_fill(0xFF) >= 4 * 2_000_000) == fails    # and its words too


def test_a_minibatch_is_not_captured(lib, ctx):
    """Its words hold numbers that only this call has: a replay would find its own of the time before.  Refused before
    anything is queued, and the context works on."""
    assert _start(lib, ctx, 1000) == _lib.OK
    lib.fake_reset()
    for n_nodes in (0, 1000):
        lib.fake_capture(1)
        assert _start(lib, ctx, n_nodes) == _lib.ERR_INVALID
        assert b"being captured" in lib.shmt_last_error()
        assert lib.fake_launches() == 0 and lib.fake_largest_fill(0) == 0
        lib.fake_capture(0)
    assert _start(lib, ctx, 1000) == _lib.OK and lib.fake_launches() > 0


@pytest.mark.parametrize("n", [1000, 1_000_000, 9_000_000, 40_000_000])
def test_a_scan_whose_launch_fails_says_so_once(lib, ctx, n):
    """Scans of one tile, of a grid, and of clusters with a rest: the call reports the failure, and the caller's own next
    check of the runtime's last error does not find it again."""
    data = _buffer(8 * n)
    at = (C.addressof(data) + 15) & ~15
    assert lib.shmt_scan(ctx, at, _lib.I64, n, 0, None) == _lib.OK
    lib.fake_fail_launches(1)
    try:
        for where, m in ((at, n), (at + 8, n - 1)):
            assert lib.shmt_scan(ctx, where, _lib.I64, m, 0, None) == _lib.ERR_CUDA
            assert lib.fake_last_error() == 0
    finally:
        lib.fake_fail_launches(0)
    assert lib.shmt_scan(ctx, at, _lib.I64, n, 0, None) == _lib.OK


def test_lookups_fetches_and_relabels_report_a_failed_launch_once(lib, ctx):
    """The same of the other calls that are scheduled while the kernel before them runs."""
    ids, out, table = _buffer(8 * 64), _buffer(64 * 512), _buffer(64 * 512)
    at = [(C.addressof(b) + 15) & ~15 for b in (ids, out, table)]
    hmap = C.c_void_p()
    assert lib.shmt_map_create(0, 128, 64, _lib.I64, _lib.I32, None, None, C.byref(hmap)) == _lib.OK
    lib.fake_fail_launches(1)
    try:
        assert lib.shmt_map_query(hmap, at[0], _lib.I64, 64, at[1], None) == _lib.ERR_CUDA and lib.fake_last_error() == 0
        for row in (512, 602, 4):  # a ring of rows, of odd ones, and plain copies
            assert lib.shmt_fetch(hmap, None, 0, None, at[2], at[0], _lib.I64, 32, row, at[1], None) == _lib.ERR_CUDA
            assert lib.fake_last_error() == 0
        assert _relabel(lib, ctx, 100) == _lib.ERR_CUDA and lib.fake_last_error() == 0
    finally:
        lib.fake_fail_launches(0)
        lib.shmt_map_destroy(hmap)
