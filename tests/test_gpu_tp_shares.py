"""The general contraction kernels (fp64, weights in memory, channel counts other than 64 and 128) where the edges of a target are dealt
to several blocks or sets of threads: a target without edges, with one, with less, exactly and more than a batch of eight per share, and so
many targets that nothing is shared.  Against the oracle."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from tace_b200.graph import build_batch
from helpers import check_parity, make_models, oracle_batch, to_device
from test_gpu_tp_wide import _ring

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("L,Lmax,C,dtype", [(1, 1, 32, torch.float32), (2, 1, 96, torch.float32), (2, 2, 64, torch.float64), (3, 3, 32, torch.float64),
                                            (2, 2, 160, torch.float32)])
@pytest.mark.parametrize("degrees", [(1, 7, 8, 9, 33), (60, 64, 65), (63, 129)])
def test_shared_edges(L, Lmax, C, dtype, degrees):
    structs = [_ring(n) for n in degrees] + [synth.Structure(positions=np.zeros((1, 3)), atomic_numbers=np.array([29]), cell=np.eye(3) * 30.0,
                                                             pbc=(True, True, True))]
    model, oracle, _ = make_models(L, C, [13, 29], 4.0, 12.0, dtype, Lmax=Lmax)
    data = oracle_batch(structs, [13, 29], 4.0, dtype)
    check_parity(model(to_device(data, DEV)), oracle(data), data["ptr"], dtype, f"L{L} Lmax{Lmax} C{C}")


@pytest.mark.parametrize("C,dtype", [(96, torch.float32), (64, torch.float64)])
def test_few_and_many_targets_agree(C, dtype):
    """108 targets (shared edges) and 4 000 (none shared) of the same unperturbed crystal: the same energy per atom."""
    model, _, _ = make_models(2, C, [29], 5.0, 40.0, dtype)
    few, many = (model(build_batch(synth.collate([synth.fcc_supercell(n, 3.61, 0.0, seed=1)]), [29], 5.0, dtype, DEV))["energy"].item() / (4 * n ** 3)
                 for n in (3, 10))
    assert abs(many - few) <= (1e-5 if dtype is torch.float32 else 1e-8)


@pytest.mark.parametrize("C,dtype", [(96, torch.float64), (192, torch.float32)])
def test_first_interaction_with_48_kb_of_dynamic_shared_memory(C, dtype):
    """Rank 3 at these widths: (16 + 8 (4 + 2)) C values are 48 KB to the byte, and the kernel has static shared memory besides."""
    structs = [_ring(9)]
    model, oracle, _ = make_models(3, C, [13, 29], 4.0, 12.0, dtype)
    model.set_radial_table(False)
    data = oracle_batch(structs, [13, 29], 4.0, dtype)
    check_parity(model(to_device(data, DEV)), oracle(data), data["ptr"], dtype, f"C{C}")
