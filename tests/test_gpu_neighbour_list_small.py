"""Small batches: the sources found by the count are kept for the fill (128 per target), and up to 2 048 atoms four warps share an atom.
Targets just below, at and above what is kept, batch sizes on both sides of the lines, and the pair of calls without anything kept."""
import ctypes

import numpy as np
import pytest
import torch

from tace_b200 import lib as _lib, synth
from test_gpu_neighbour_list import check

pytestmark = pytest.mark.gpu


def _gas(n, box, seed):
    rng = np.random.default_rng(seed)
    return synth.Structure(positions=rng.random((n, 3)) * box, atomic_numbers=np.ones(n, dtype=np.int64), cell=np.eye(3) * box, pbc=(True, True, False))


@pytest.mark.parametrize("n", [1, 128, 129, 130, 160])
def test_everybody_sees_everybody(n):
    """n atoms in a corner of a large cell: n - 1 sources each."""
    s = _gas(n, 2.0, n)
    s["cell"] = np.eye(3) * 20.0
    assert check(s, 4.0).shape[1] == n * (n - 1)


@pytest.mark.parametrize("n", [2047, 2048, 2049])
def test_both_sides_of_the_shared_search(n):
    check(_gas(n, 14.0, n), 3.0)


def test_a_workspace_without_room_for_the_sources():
    """What tace_nl_workspace_bytes reported before sources were kept is still enough, in either call of the pair."""
    lib, dev = _lib.load(), torch.device("cuda:0")
    n, rc = 300, 3.0
    s = _gas(n, 9.0, 5)
    pos, lat = torch.as_tensor(s["positions"], device=dev), torch.as_tensor(s["cell"], device=dev)[None].contiguous()
    pbc = torch.tensor([s["pbc"]], dtype=torch.uint8, device=dev)
    ptr = torch.tensor([0, n], dtype=torch.int32, device=dev)
    need = ctypes.c_size_t()
    assert lib.tace_nl_workspace_bytes(n, 1, ctypes.byref(need)) == 0
    work = torch.zeros(need.value + 256, dtype=torch.uint8, device=dev)
    counts, rows = torch.empty(n, dtype=torch.int32, device=dev), torch.empty(n + 1, dtype=torch.int64, device=dev)
    small = need.value - 16 * 128 * n
    args = (pos.data_ptr(), lat.data_ptr(), pbc.data_ptr(), ptr.data_ptr(), 1, n, -1, rc)
    lists = []
    for first, second in ((work.numel(), work.numel()), (small, small), (small, work.numel()), (work.numel(), small)):
        work.fill_(255)
        assert lib.tace_nl_rows(*args, counts.data_ptr(), rows.data_ptr(), work.data_ptr(), first, 0) == 0
        E = int(rows[-1])
        ei, es = torch.empty(2, E, dtype=torch.int64, device=dev), torch.empty(E, 3, dtype=torch.float32, device=dev)
        assert lib.tace_nl_fill_rows(*args, rows.data_ptr(), E, ei.data_ptr(), es.data_ptr(), _lib.TACE_F32, work.data_ptr(), second, 0) == 0
        lists.append((ei, es))
    assert lists[0][0].shape[1] > 0
    for ei, es in lists[1:]:
        assert torch.equal(ei, lists[0][0]) and torch.equal(es, lists[0][1])
