"""Symmetric gather rows of a pair list against numpy, at the edges of the
builder's routes: sorted and unsorted lists, lists off a 16-byte boundary, rows
of one to more than 65,536 entries, indices out of range."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SECOND = 1 << 31


def expected_rows(pairs, n):
    i = np.concatenate((pairs[:, 0], pairs[:, 1]))
    e = np.concatenate((pairs[:, 1], pairs[:, 0] | SECOND))
    ptr = np.zeros(n + 1, dtype=np.int64)
    np.add.at(ptr, i + 1, 1)
    return np.cumsum(ptr), e[np.lexsort((e, i))]


def check(pairs, n, dev, odd=False):
    from tensorsph_b200.droplet_impact import symmetric_rows
    t = torch.from_numpy(np.ascontiguousarray(pairs, dtype=np.int64).reshape(-1, 2)).to(dev)
    if odd:
        flat = torch.zeros(t.numel() + 1, dtype=torch.int64, device=dev)
        flat[1:] = t.reshape(-1)
        t = flat[1:].view(-1, 2)
    ptr, entries = symmetric_rows(t, n)
    want_ptr, want = expected_rows(pairs.reshape(-1, 2), n)
    assert np.array_equal(ptr.cpu().numpy(), want_ptr)
    assert np.array_equal(entries.cpu().numpy()[:want.size].view(np.uint32).astype(np.int64), want)


@pytest.mark.parametrize("n,count", [(1, 0), (5, 3), (300, 40), (2000, 30000), (50000, 900000), (700, 200000)])
def test_rows_of_random_lists(gpu, n, count):
    rng = np.random.default_rng(n)
    p = rng.integers(0, n, (count, 2))
    check(p, n, gpu)                                              # any order, both orientations, repeats
    lex = p[np.lexsort((p[:, 1], p[:, 0]))]
    check(lex, n, gpu)                                            # sorted, second index on either side
    q = np.sort(p, axis=1)
    check(q[np.lexsort((q[:, 1], q[:, 0]))], n, gpu, odd=True)    # sorted i <= j, off a 16-byte boundary


@pytest.mark.parametrize("count", [15, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 8192, 8193,
                                   65536, 65537])
def test_rows_at_the_sort_tiers(gpu, count):
    """One row with ``count`` second-element entries, one with as many first-element
    ones; the list sorted and reversed."""
    hub = np.stack((np.arange(count), np.full(count, count)), axis=1)
    fan = np.stack((np.zeros(count, dtype=np.int64), 1 + np.arange(count)), axis=1)
    for p in (hub, fan, hub[::-1], fan[::-1]):
        check(p, count + 1, gpu)


@pytest.mark.parametrize("bad", [[[0, 1], [2, 9]], [[0, 9], [1, 2]], [[-1, 2], [0, 1]], [[5, 1], [0, 99]]])
def test_rows_refuse_bad_indices(gpu, bad):
    from tensorsph_b200.droplet_impact import symmetric_rows
    with pytest.raises(ValueError):
        symmetric_rows(torch.tensor(bad, dtype=torch.int64, device=gpu), 9)


@pytest.mark.parametrize("per_row", [0, 1, 7, 19, 20, 10 ** 6])
@pytest.mark.parametrize("mixed", [False, True])
def test_rows_at_slot_counts(gpu, per_row, mixed):
    """Workspaces with room for no, few, almost enough, just enough and more slots than a
    row's second halves (at most 20 here) give the same rows."""
    from tensorsph_b200 import _lib
    rng = np.random.default_rng(per_row)
    n = 1003
    p = np.stack((np.repeat(np.arange(n), 20), (np.arange(n)[:, None] + 1 + np.arange(20)).reshape(-1)), axis=1)
    p = p[p[:, 1] < n]
    if mixed:
        p = np.sort(rng.permutation(n)[p], axis=1)
        p = p[np.lexsort((p[:, 1], p[:, 0]))]
    L = _lib.lib()
    t = torch.from_numpy(p).to(gpu)
    ptr = torch.empty(n + 1, dtype=torch.long, device=gpu)
    entries = torch.empty(2 * p.shape[0], dtype=torch.int32, device=gpu)
    least = L.tsph_csr_workspace_bytes(p.shape[0], n)
    room = min(4 * n * per_row, L.tsph_csr_slot_bytes(p.shape[0], n))
    ws = _lib.workspace(least + room, gpu)
    args = (t.data_ptr(), p.shape[0], n, ptr.data_ptr(), entries.data_ptr(), ws.data_ptr())
    _lib.check(L.tsph_csr_from_pairs(*args, least + room, _lib.stream(gpu)), "tsph_csr_from_pairs")
    want_ptr, want = expected_rows(p, n)
    assert np.array_equal(ptr.cpu().numpy(), want_ptr)
    assert np.array_equal(entries.cpu().numpy().view(np.uint32).astype(np.int64), want)
    assert L.tsph_csr_from_pairs(*args, least - 1, _lib.stream(gpu)) != 0


def test_rows_without_memory_for_slots(gpu, monkeypatch):
    from tensorsph_b200 import _lib
    plain, refused = _lib.workspace, []

    def tight(nbytes, device):
        if not refused:
            refused.append(nbytes)
            raise torch.OutOfMemoryError("no room")
        return plain(nbytes, device)

    monkeypatch.setattr(_lib, "workspace", tight)
    p = np.sort(np.random.default_rng(0).integers(0, 500, (9000, 2)), axis=1)
    check(p[np.lexsort((p[:, 1], p[:, 0]))], 500, gpu)
    assert refused


@pytest.mark.parametrize("count", [8191, 8192, 8193, 16383, 16384, 16385, 24577, 40000, 131073])
def test_rows_beyond_shared_memory(gpu, count):
    """Two rows sorted by stretches of 8192 entries, in arbitrary order and with repeats; the
    list sorted and shuffled."""
    rng = np.random.default_rng(count)
    n = count + 2
    p = np.concatenate((np.stack((rng.integers(0, n - 2, count), np.full(count, n - 1)), axis=1),
                        np.stack((rng.permutation(n - 2)[:count], np.full(count, n - 2)), axis=1)))
    check(rng.permutation(p), n, gpu)
    check(p[np.lexsort((p[:, 1], p[:, 0]))], n, gpu)


@pytest.mark.parametrize("count", [511, 131071, 131072, 131073, 300000])
def test_rows_where_degrees_are_counted_along(gpu, count):
    """Sorted and unsorted lists around the size up to which the first pass also counts the
    degrees, the order broken at the start, in the middle and by the last pair; an index out
    of range as the last thing in each."""
    from tensorsph_b200.droplet_impact import symmetric_rows
    rng = np.random.default_rng(count)
    n = count // 7
    p = rng.integers(0, n, (count, 2))
    p = p[np.lexsort((p[:, 1], p[:, 0]))]
    p[-1], p[-2] = (n - 1, n - 1), (n - 1, n - 2)
    for at in (None, 1, count // 2, count - 1):
        q = p.copy()
        if at is not None:
            q[[at - 1, at]] = [[n - 1, 3], [0, 5]]
        check(q, n, gpu)
        for bad in (n, -1):
            q[-1, 1] = bad
            with pytest.raises(ValueError):
                symmetric_rows(torch.from_numpy(q).to(gpu), n)
