"""The cell search against the oracle where its routes change: the number of
rows that switches lanes per row, three and four cells on a periodic axis,
particles outside the box, distances at the cutoff, a far-off origin, and the
list ends of a pruned search."""
import numpy as np
import pytest
import torch

from oracle import neighbors as on

pytestmark = pytest.mark.gpu


def lattice(counts, dx, dtype, jitter, seed=0):
    g = np.stack(np.meshgrid(*[np.arange(c) for c in counts], indexing="ij"), -1).reshape(-1, len(counts))
    rng = np.random.default_rng(seed)
    return ((g + 0.5 + jitter * rng.uniform(-1, 1, g.shape)) * dx).astype(dtype)


def search(pos, cutoff, dev, box=None):
    from tensorsph_b200.neighbor_search import cell_linked_pairs
    from tensorsph_b200.threed import periodic_pairs
    t = torch.from_numpy(pos).to(dev)
    return (cell_linked_pairs(t, cutoff) if box is None else periodic_pairs(t, box, cutoff)).cpu().numpy()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("cutoff", [1.0, 2.0, 2.6])
def test_lattice_shells_at_the_cutoff(gpu, dtype, cutoff):
    """Unjittered lattices: whole shells lie exactly at the cutoff, where the last bit decides."""
    for counts, scale in (((40, 31), 0.1), ((13, 11, 12), 0.013), ((900,), 0.37)):
        pos = lattice(counts, scale, dtype, 0.0)
        pos = pos[np.random.default_rng(1).permutation(pos.shape[0])]
        assert np.array_equal(search(pos, cutoff * scale, gpu), on.cell_linked_pairs(pos, cutoff * scale))


@pytest.mark.parametrize("n", [24575, 24576, 24577])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_lanes_per_row_switch(gpu, n, dtype):
    pos = lattice((160, 160), 0.01, dtype, 0.2)[:n]
    pos = pos[np.random.default_rng(2).permutation(n)]
    assert np.array_equal(search(pos, 0.027, gpu), on.cell_linked_pairs(pos, 0.027))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("cells", [1.5, 3.0, 3.9, 4.0, 4.5, 7.0])
def test_periodic_axes_of_few_cells(gpu, dtype, cells):
    rng = np.random.default_rng(5)
    for dim in (1, 2, 3):
        pos = rng.random((700, dim)).astype(dtype)
        pos[:50] += rng.integers(-3, 4, (50, dim))            # whole boxes away
        pos[50:60] = 0.0
        pos[60:70] = 1.0
        cutoff = 1.0 / cells
        assert np.array_equal(search(pos, cutoff, gpu, [1.0] * dim),
                              on.periodic_pairs(pos, [1.0] * dim, cutoff))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("offset", [0.0, -3.7, 900.0, 2.0e5])
def test_far_origin(gpu, dtype, offset):
    """FP32 records measured from the grid's corner; coordinates far from zero."""
    pos = (lattice((25, 24, 5), 0.1, np.float64, 0.2) + offset).astype(dtype)
    assert np.array_equal(search(pos, 0.27, gpu), on.cell_linked_pairs(pos, 0.27))


def test_long_thin_cloud(gpu):
    """A grid many thousand cutoffs long: the FP32 records no longer decide, the exact distances do."""
    rng = np.random.default_rng(8)
    pos = np.concatenate((rng.random((600, 2)) * [0.5, 0.2], rng.random((600, 2)) * [0.5, 0.2] + [8.0e5, 0.0]))
    assert np.array_equal(search(pos, 0.03, gpu), on.cell_linked_pairs(pos, 0.03))


def test_pruned_list_and_order(gpu):
    from tensorsph_b200.neighbor_search import cell_order, grid_pairs
    pos = lattice((60, 50), 0.01, np.float64, 0.2)
    t = torch.from_numpy(pos).to(gpu)
    full = on.cell_linked_pairs(pos, 0.027)
    for limit in (0, 1, 1234, 2999, 3000):
        pairs, total, order = grid_pairs(t, 0.027, row_limit=limit, with_order=True)
        assert total == full.shape[0]
        assert np.array_equal(pairs.cpu().numpy(), full[full[:, 0] < limit])
        assert torch.equal(order, cell_order(t, 0.027))


def rows_and_pairs(pos, cutoff, limit, dev):
    from tensorsph_b200.droplet_impact import symmetric_rows
    from tensorsph_b200.neighbor_search import grid_pairs, grid_rows
    t = torch.from_numpy(pos).to(dev)
    pairs, _, _ = grid_pairs(t, cutoff, row_limit=limit)
    return grid_rows(t, cutoff, row_limit=limit), symmetric_rows(pairs, pos.shape[0]), pairs


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("counts,cutoff", [((41, 30), 0.026), ((300, 301), 0.0293), ((17, 16, 15), 0.026),
                                           ((45, 44, 43), 0.0293), ((12, 13, 11), 0.055), ((400,), 0.03)])
def test_rows_without_the_list(gpu, dtype, counts, cutoff):
    """Gather rows straight from the cells equal those made of the pair list; the
    0.055 rows (about 700 neighbours) outgrow their slots."""
    pos = lattice(counts, 0.01, dtype, 0.2)
    n = pos.shape[0]
    for limit in (n, n // 2, 1, 0):
        (ptr, entries, count), (ptr2, entries2), pairs = rows_and_pairs(pos, cutoff, limit, gpu)
        assert count == 2 * pairs.shape[0]
        assert torch.equal(ptr, ptr2)
        assert torch.equal(entries[:count], entries2[:count])


@pytest.mark.parametrize("count", [15, 16, 17, 47, 48, 49, 50, 127, 128, 129, 130, 300])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_rows_at_their_slots(gpu, count, dim):
    """A cluster of ``count`` neighbours among spread-out particles, around the number of
    slots a row has in each dimension."""
    rng = np.random.default_rng(count)
    pos = np.concatenate((0.01 * rng.random((count, dim)), 1.0 + np.arange(2000)[:, None] * 0.1 + np.zeros(dim)))
    pos = pos[rng.permutation(pos.shape[0])]
    (ptr, entries, total), (ptr2, entries2), pairs = rows_and_pairs(pos, 0.02, pos.shape[0], gpu)
    assert np.array_equal(pairs.cpu().numpy(), on.cell_linked_pairs(pos, 0.02))
    assert torch.equal(ptr, ptr2) and torch.equal(entries[:total], entries2[:total])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("box,lattice_points,offset", [(None, False, 0.0), (None, True, 0.0), (None, False, 3.0e3),
                                                       (1.0, False, 0.0), (1.0, True, 0.0)])
def test_runs_of_any_length(gpu, dtype, box, lattice_points, offset):
    """The 3-D pass of a row per thread: runs of candidates from none to several words of
    32, starting anywhere in a block of four, with distances at the cutoff (the lattice) and
    with many candidates to decide exactly (the far origin)."""
    from oracle.neighbors import cell_linked_pairs_batched
    rng = np.random.default_rng(8)
    if lattice_points:
        pos = lattice((32, 32, 32), 1.0 / 32, dtype, 0.0)[:25000]
        cutoff = 2.0 / 32
    else:
        pos = rng.random((25000, 3)) ** [1.0, 1.0, 3.0]       # dense at one face, sparse at the other
        pos = (pos + offset).astype(dtype)
        cutoff = 0.052
    pos = pos[rng.permutation(pos.shape[0])]
    want = cell_linked_pairs_batched(pos, cutoff) if box is None else on.periodic_pairs(pos, [box] * 3, cutoff)
    assert np.array_equal(search(pos, cutoff, gpu, None if box is None else [box] * 3), want)
    if box is None:
        (ptr, entries, count), (ptr2, entries2), _ = rows_and_pairs(pos, cutoff, pos.shape[0] // 2, gpu)
        assert torch.equal(ptr, ptr2) and torch.equal(entries[:count], entries2[:count])


@pytest.mark.parametrize("dtype,scale", [(np.float64, 1e-100), (np.float64, 1e-25), (np.float64, 1e-12), (np.float64, 1e18),
                                         (np.float64, 1e20), (np.float64, 1e30), (np.float64, 1e45), (np.float64, 1e145),
                                         (np.float32, 1e-20), (np.float32, 1e-12), (np.float32, 1e14), (np.float32, 1e20)])
@pytest.mark.parametrize("counts", [(300,), (30000,), (24, 25), (160, 161), (8, 9, 10), (30, 30, 29)])
def test_any_unit_of_length(gpu, dtype, scale, counts):
    """Lengths whose squares leave the range of FP32, or of the positions' own dtype, on
    both sides of the row count that switches lanes per row: lists, periodic lists, rows."""
    pos = (lattice(counts, 1.0, np.float64, 0.2) * scale).astype(dtype)
    pos = pos[np.random.default_rng(3).permutation(pos.shape[0])]
    cutoff = 1.3 * scale
    with np.errstate(over="ignore", under="ignore"):
        want = on.cell_linked_pairs_batched(pos, cutoff)
        box = [c * scale for c in counts]
        periodic = on.periodic_pairs(pos, box, cutoff) if pos.shape[0] < 1000 else None
    assert np.array_equal(search(pos, cutoff, gpu), want)
    if periodic is not None:
        assert np.array_equal(search(pos, cutoff, gpu, box), periodic)
    (ptr, entries, count), (ptr2, entries2), _ = rows_and_pairs(pos, cutoff, pos.shape[0] // 2, gpu)
    assert torch.equal(ptr, ptr2) and torch.equal(entries[:count], entries2[:count])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [24576, 24577, 30001])
@pytest.mark.parametrize("dim", [2, 3])
def test_exact_grids_of_many_rows(gpu, dtype, n, dim):
    """Three periodic cells on an axis (every candidate takes the exact arithmetic) and a
    cloud with a far clump (the same, cells by bisection), on both sides of the row count
    that switches lanes per row elsewhere."""
    rng = np.random.default_rng(n)
    box = [1.0] * (dim - 1) + [n / 3.0 ** dim / 12]
    pos = (rng.random((n, dim)) * box).astype(dtype)
    assert np.array_equal(search(pos, 0.333, gpu, box), on.periodic_pairs(pos, box, 0.333))
    side = int(np.ceil(n ** (1.0 / dim)))
    pos = lattice((side,) * dim, 1.0, np.float64, 0.2)[:n]
    pos[-64:, 0] += 1.0e6
    pos = pos.astype(dtype)[rng.permutation(n)]
    assert np.array_equal(search(pos, 1.6, gpu), on.cell_linked_pairs_batched(pos, 1.6))


@pytest.mark.parametrize("counts,cutoff", [((200,), 2.6), ((40, 41), 2.6), ((40, 41), 6.0), ((12, 13, 11), 2.6),
                                           ((31, 30, 29), 2.6), ((12, 13, 11), 5.5)])
def test_emit_after_other_counts(gpu, counts, cutoff):
    """An emit gives the rows of its own count whatever was counted on the grid in between:
    the list and the rows share the slots (6.0 and 5.5: rows that outgrow them)."""
    import ctypes
    from tensorsph_b200 import _lib
    from tensorsph_b200.neighbor_search import _plan
    pos = lattice(counts, 1.0, np.float64, 0.2)
    pos = torch.from_numpy(pos[np.random.default_rng(6).permutation(pos.shape[0])]).to(gpu)
    n, L, s = pos.shape[0], _lib.lib(), _lib.stream(gpu)
    grid, ws = _plan(pos, cutoff)
    head = (pos.data_ptr(), ctypes.byref(grid))
    work = (ws.data_ptr(), ws.numel())

    def count_rows(limit):
        ptr, c = torch.empty(n + 1, dtype=torch.long, device=gpu), ctypes.c_int64(0)
        _lib.check(L.tsph_rows_count(*head, limit, *work, ptr.data_ptr(), ctypes.byref(c), s), "rows_count")
        return limit, ptr, c.value

    def emit_rows(limit, ptr, c):
        out = torch.empty(c, dtype=torch.int32, device=gpu)
        _lib.check(L.tsph_rows_emit(*head, limit, *work, ptr.data_ptr(), out.data_ptr(), c, s), "rows_emit")
        return out

    def count_pairs(limit):
        c, total = ctypes.c_int64(0), ctypes.c_int64(0)
        _lib.check(L.tsph_pairs_count(*head, limit, *work, ctypes.byref(c), ctypes.byref(total), s), "pairs_count")
        return limit, c.value

    def emit_pairs(limit, c):
        out = torch.empty((c, 2), dtype=torch.long, device=gpu)
        ews = _lib.workspace(L.tsph_pairs_emit_workspace_bytes(c, n), gpu)
        _lib.check(L.tsph_pairs_emit(*head, limit, *work, ews.data_ptr(), ews.numel(), out.data_ptr(), c, s),
                   "pairs_emit")
        return out

    _lib.check(L.tsph_grid_build(*head, *work, None, s), "tsph_grid_build")
    list_, half = count_pairs(n), n // 2
    want = emit_pairs(*list_)
    assert np.array_equal(want.cpu().numpy(), on.cell_linked_pairs(pos.cpu().numpy(), cutoff))
    whole = count_rows(n)
    rows = emit_rows(*whole)
    part = count_rows(half)
    part_rows = emit_rows(*part)
    assert torch.equal(emit_pairs(*list_), want)              # after the rows of another limit
    assert torch.equal(emit_rows(*whole), rows)
    assert torch.equal(emit_rows(*part), part_rows)
    short = count_pairs(half)                                 # the list's count between rows' count and emit
    assert torch.equal(emit_pairs(*short), want[want[:, 0] < half])
    assert torch.equal(emit_rows(*whole), rows)
    assert torch.equal(emit_rows(*part), part_rows)


@pytest.mark.parametrize("at", ["slots", "result"])
@pytest.mark.parametrize("counts,cutoff", [((40, 41), 2.6), ((12, 13, 11), 2.6), ((31, 30, 29), 2.6)])
def test_search_without_memory_for_slots(gpu, monkeypatch, at, counts, cutoff):
    """Where torch has no memory for the row slots, or for the result beside them, the
    search runs without them."""
    from tensorsph_b200 import _lib
    from tensorsph_b200 import neighbor_search as ns
    pos = lattice(counts, 1.0, np.float64, 0.2)
    n = pos.shape[0]
    t = torch.from_numpy(pos).to(gpu)
    want = on.cell_linked_pairs(pos, cutoff)
    rows = ns.grid_rows(t, cutoff, row_limit=n // 2)
    plain, empty, refused, sizes = _lib.workspace, torch.empty, [], []
    fewest = 4 * n * 48                                        # the slots of 48 (2-D) or 128 a row

    def tight(nbytes, device):
        sizes.append(nbytes)
        if at == "slots" and nbytes > fewest and not refused:
            refused.append(nbytes)
            raise torch.OutOfMemoryError("no room")
        return plain(nbytes, device)

    def no_result(*a, **k):
        result = k.get("dtype") in (torch.long, torch.int32) and (a[0] == (want.shape[0], 2) or a[0] == rows[2])
        if at == "result" and result and not refused:
            refused.append(a[0])
            raise torch.OutOfMemoryError("no room")
        return empty(*a, **k)

    monkeypatch.setattr(_lib, "workspace", tight)
    monkeypatch.setattr(torch, "empty", no_result)
    assert np.array_equal(ns.cell_linked_pairs(t, cutoff).cpu().numpy(), want)
    assert len(refused) == 1
    refused.clear()
    sizes.clear()
    got = ns.grid_rows(t, cutoff, row_limit=n // 2)
    assert len(refused) == 1 and got[2] == rows[2]
    assert torch.equal(got[0], rows[0]) and torch.equal(got[1], rows[1])
    big = [b for b in sizes if b > 1024]
    assert big[-1] <= big[0] - fewest                          # the second one has no slots
