"""Cell-list kernel against the brute-force oracle: the canonically sorted edge set must be bit-exact."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from tace_b200.neighbour_list import get_neighborhood, neighbor_list_batch

pytestmark = pytest.mark.gpu


def check(structure, cutoff):
    from oracle.neighbour_list import canonical_sort, neighbour_list

    ref_i, ref_s = neighbour_list(structure["positions"], structure["cell"], structure["pbc"], cutoff)
    ei, es, _, _ = get_neighborhood(structure["positions"], cutoff, structure["pbc"], structure["cell"])
    ei, es = canonical_sort(ei, es)
    assert ei.shape == ref_i.shape, (ei.shape, ref_i.shape)
    assert np.array_equal(ei, ref_i) and np.array_equal(es, ref_s)
    return ei


def test_cubic_fcc():
    ei = check(synth.fcc_supercell(3, 3.61, 0.05, seed=0), 5.0)
    assert ei.shape[1] > 0


def test_triclinic_small_cells_with_self_images():
    for s in synth.random_crystals(6, seed=7, nmin=2, nmax=10):
        check(s, 6.0)


def test_unwrapped_positions():
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=1)
    rng = np.random.default_rng(0)
    s["positions"] = s["positions"] + rng.integers(-2, 3, size=(s["positions"].shape[0], 3)) @ s["cell"]
    check(s, 4.5)


def test_mixed_and_open_boundaries():
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=2)
    for pbc in [(True, True, False), (False, False, False), (True, False, False)]:
        t = synth.Structure(s)
        t["pbc"] = pbc
        check(t, 4.5)


def test_single_atom_and_no_neighbours():
    one = synth.Structure(positions=np.zeros((1, 3)), atomic_numbers=np.array([1]), cell=np.eye(3) * 4.0, pbc=(True,) * 3)
    ei = check(one, 6.0)  # only self images
    assert ei.shape[1] > 0 and (ei[0] == ei[1]).all()
    far = synth.Structure(positions=np.array([[0.0, 0, 0], [10.0, 0, 0]]), atomic_numbers=np.array([1, 1]),
                          cell=np.eye(3) * 40.0, pbc=(False,) * 3)
    assert check(far, 3.0).shape[1] == 0


def test_batch_matches_per_structure():
    structs = synth.random_crystals(5, seed=3, nmin=3, nmax=20)
    b = synth.collate(structs)
    dev = torch.device("cuda:0")
    ei, es = neighbor_list_batch(torch.tensor(b["positions"], device=dev), torch.tensor(b["lattice"], device=dev),
                                 torch.tensor(b["pbc"], device=dev), torch.tensor(b["ptr"], dtype=torch.int32, device=dev), 6.0)
    from oracle.neighbour_list import canonical_sort, neighbour_list
    ref_i, ref_s = [], []
    for s, off in zip(structs, b["ptr"][:-1]):
        a, c = neighbour_list(s["positions"], s["cell"], s["pbc"], 6.0)
        ref_i.append(a + off)
        ref_s.append(c)
    ref_i, ref_s = canonical_sort(np.concatenate(ref_i, 1), np.concatenate(ref_s, 0))
    gi, gs = canonical_sort(ei.cpu().numpy(), es.cpu().numpy())
    assert np.array_equal(gi, ref_i) and np.array_equal(gs, ref_s)
    # grouped by target: row 1 is non-decreasing
    assert (np.diff(ei[1].cpu().numpy()) >= 0).all()


@pytest.mark.parametrize("n_mol,copies", [(1, 1), (5, 3), (900, 1), (2731, 1)])  # 3 atoms .. 8 193: one-block preparation and beyond it
def test_rows_entry_equals_the_count_and_fill_pair(n_mol, copies):
    """tace_nl_rows / tace_nl_fill_rows (device-side row pointers, reused preparation, real shifts) against tace_nl_count /
    tace_nl_fill with host-side row pointers: the same edges in the same order."""
    import ctypes
    from tace_b200 import lib as _lib, synth
    from tace_b200.neighbour_list import _list_on_device
    lib, dev = _lib.load(), torch.device("cuda:0")
    side = int(np.ceil(n_mol ** (1 / 3)))
    structs = [synth.water_box(n_side=side, box=max(3.2 * side, 4.0), seed=k, n_mol=n_mol) for k in range(copies)]
    b = synth.collate(structs)
    pbc = torch.as_tensor(b["pbc"], device=dev)
    pbc[0, 2] = 0  # one open axis
    pos, lat = torch.as_tensor(b["positions"], device=dev), torch.as_tensor(b["lattice"], device=dev)
    ptr = torch.as_tensor(b["ptr"], device=dev).to(torch.int32)
    n, g, rc = pos.shape[0], lat.shape[0], 5.0
    ei, es = _list_on_device(pos, lat, pbc, ptr, rc, -1, torch.float64)
    need = ctypes.c_size_t()
    assert lib.tace_nl_workspace_bytes(n, g, ctypes.byref(need)) == 0
    work = torch.empty(need.value, dtype=torch.uint8, device=dev)
    counts = torch.empty(n, dtype=torch.int32, device=dev)
    args = (pos.data_ptr(), lat.data_ptr(), pbc.data_ptr(), ptr.data_ptr(), g, n, rc)
    assert lib.tace_nl_count(*args, counts.data_ptr(), work.data_ptr(), work.numel(), 0) == 0
    rows = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    rows[1:] = torch.cumsum(counts, 0)
    E = int(rows[-1])
    ei2, es2 = torch.empty(2, E, dtype=torch.int64, device=dev), torch.empty(E, 3, dtype=torch.int32, device=dev)
    assert lib.tace_nl_fill(*args, rows.data_ptr(), E, ei2.data_ptr(), es2.data_ptr(), work.data_ptr(), work.numel(), 0) == 0
    assert E > 0 or n_mol == 1
    assert torch.equal(ei, ei2) and torch.equal(es, es2.double())


@pytest.mark.parametrize("n", [46500, 66000])  # row pointers in one block, by the device-wide scan (from 65 537 atoms)
def test_row_pointers_past_two_to_the_31_edges(n):
    """Every atom of a small open cluster sees every other one: n (n - 1) edges, 2.16e9 and 4.36e9 of them, counted but not stored."""
    import ctypes
    from tace_b200 import lib as _lib
    lib, dev = _lib.load(), torch.device("cuda:0")
    pos = torch.rand(n, 3, generator=torch.Generator().manual_seed(n), dtype=torch.float64).to(dev)
    lat = (4.0 * torch.eye(3, dtype=torch.float64, device=dev))[None].contiguous()
    pbc = torch.zeros(1, 3, dtype=torch.uint8, device=dev)
    ptr = torch.tensor([0, n], dtype=torch.int32, device=dev)
    need = ctypes.c_size_t()
    assert lib.tace_nl_workspace_bytes(n, 1, ctypes.byref(need)) == 0
    work = torch.empty(need.value, dtype=torch.uint8, device=dev)
    counts, rows = torch.empty(n, dtype=torch.int32, device=dev), torch.empty(n + 1, dtype=torch.int64, device=dev)
    assert lib.tace_nl_rows(pos.data_ptr(), lat.data_ptr(), pbc.data_ptr(), ptr.data_ptr(), 1, n, -1, 2.0, counts.data_ptr(), rows.data_ptr(),
                            work.data_ptr(), work.numel(), 0) == 0
    assert (counts == n - 1).all()
    assert torch.equal(rows, (n - 1) * torch.arange(n + 1, dtype=torch.int64, device=dev))
