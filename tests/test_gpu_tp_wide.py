"""The contraction kernels with two channels per thread (fp32, tabulated radial weights, 64 or 128 channels) at the sizes where
their batches, shares and dispatch change: targets with one, fifteen to seventeen and many edges, a target without any, few
targets (edges of one target shared by several warps and blocks) against many."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from tace_b200.graph import build_batch
from helpers import check_parity, make_models, oracle_batch, to_device

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _ring(n, radius=2.2):
    """One atom in the middle of n others (degree n for the centre), all in a box too large for images."""
    rng = np.random.default_rng(n)
    v = rng.normal(size=(n, 3))
    pos = np.concatenate([np.zeros((1, 3)), radius * v / np.linalg.norm(v, axis=1, keepdims=True)]) + 20.0
    return synth.Structure(positions=pos, atomic_numbers=np.array([13, 29])[np.arange(n + 1) % 2], cell=np.eye(3) * 40.0, pbc=(True, True, True))


@pytest.mark.parametrize("L,Lmax,C", [(1, 1, 64), (2, 1, 128), (2, 2, 64), (3, 1, 64), (3, 2, 128), (3, 3, 64), (3, 3, 128)])
def test_edge_counts_around_the_batch(L, Lmax, C):
    structs = [_ring(n) for n in (1, 15, 16, 17)] + [synth.Structure(positions=np.zeros((1, 3)), atomic_numbers=np.array([29]), cell=np.eye(3) * 30.0,
                                                                    pbc=(True, True, True))]
    model, oracle, _ = make_models(L, C, [13, 29], 4.0, 12.0, torch.float32, Lmax=Lmax)
    data = oracle_batch(structs, [13, 29], 4.0, torch.float32)
    out = model(to_device(data, DEV))
    assert model.uses_radial_table
    check_parity(out, oracle(data), data["ptr"], torch.float32, f"L{L} Lmax{Lmax} C{C}")


@pytest.mark.parametrize("C", [64, 128])
def test_envelope_after_the_radial_mlp(C):
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=4, species=(13, 29), fractions=(0.5, 0.5))
    model, oracle, _ = make_models(3, C, [13, 29], 4.0, 20.0, torch.float32, radial={"apply_cutoff": False, "bias": True})
    data = oracle_batch([s], [13, 29], 4.0, torch.float32)
    check_parity(model(to_device(data, DEV)), oracle(data), data["ptr"], torch.float32, f"C{C}")


@pytest.mark.parametrize("L,C", [(2, 64), (3, 128)])
def test_few_and_many_targets_agree(L, C):
    """A cell of 32 atoms and its 5 x 5 x 5 repetition: the same energy per atom, forces and stress."""
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=6, species=(13, 29), fractions=(0.4, 0.6))
    shifts = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), axis=-1).reshape(-1, 1, 3) @ s["cell"]
    big = synth.Structure(positions=(s["positions"][None] + shifts).reshape(-1, 3), atomic_numbers=np.tile(s["atomic_numbers"], 125),
                          cell=5 * s["cell"], pbc=(True, True, True))
    model, _, _ = make_models(L, C, [13, 29], 5.0, 40.0, torch.float32)
    few, many = (model(build_batch(synth.collate([x]), [13, 29], 5.0, torch.float32, DEV)) for x in (s, big))
    assert model.device_error() == 0
    assert abs(many["energy"].item() / 4000 - few["energy"].item() / 32) <= 1e-5
    assert (many["forces"].reshape(125, 32, 3) - few["forces"]).abs().max().item() <= 1e-4
    assert (many["stress"] - few["stress"]).abs().max().item() <= 1e-4
