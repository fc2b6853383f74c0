"""A captured pass runs work that only its end needs beside its main line (last layers of the radial MLPs, attention weights and frame
gradients of the edge block).  Replays equal the pass that is launched kernel by kernel bit for bit, again and again on changing inputs: two
and three interactions, with and without the edge block, without gradients, fp32 without the radial table."""
import pytest
import torch

from tace_b200 import synth
from helpers import make_models, oracle_batch, to_device

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("layers,dtype,tece,targets", [
    (2, torch.float64, None, ("energy", "forces", "stress")),
    (3, torch.float64, None, ("energy", "forces", "stress")),
    (3, torch.float64, None, ("energy",)),
    (1, torch.float64, None, ("energy", "forces", "stress")),
    (2, torch.float32, None, ("energy", "forces", "stress")),
    (2, torch.float32, {"num_head": 4, "edge_ace_hidden": 16, "mmax": 2}, ("energy", "forces", "stress")),
    (3, torch.float32, {"num_head": 4, "edge_ace_hidden": 16, "mmax": 1}, ("energy", "forces", "stress")),
    (3, torch.float64, {"num_head": 3, "edge_ace_hidden": 8, "mmax": 2}, ("energy", "forces")),
    (2, torch.float64, {"num_head": 4, "edge_ace_hidden": 8, "mmax": 2}, ("energy",)),
])
def test_replays_equal_the_direct_pass(layers, dtype, tece, targets, monkeypatch):
    monkeypatch.setenv("TACE_B200_RADIAL_TABLE", "0")
    structs = [synth.fcc_supercell(3, 3.65, 0.05, seed=2, species=(13, 29), fractions=(0.5, 0.5))]
    model, _, _ = make_models(2, 96, [13, 29], 4.5, 20.0, dtype, num_layers=layers, targets=targets, tece=tece,
                              radial={"apply_cutoff": False} if tece else None)
    data = to_device(oracle_batch(structs, [13, 29], 4.5, dtype), DEV)
    inputs = [dict(data, positions=data["positions"] * f, lattice=data["lattice"] * f) for f in (1.0, 1.002, 0.999)]
    model.set_graph_mode(False)
    direct = [{k: v.clone() for k, v in model(d).items() if v is not None} for d in inputs]
    model.set_graph_mode(True)
    for _ in range(2):
        model(inputs[0])
    before = model.graph_replays()
    for n in range(30):
        out = model(inputs[n % 3])
        for k, v in direct[n % 3].items():
            assert torch.equal(out[k], v), (n, k)
    assert model.graph_replays() >= before + 30


@pytest.mark.parametrize("layers,Lmax,correlation", [(1, 2, 2), (2, 1, 2), (2, 2, 3), (3, 2, 3)])
def test_zeroed_gradients_of_other_products(layers, Lmax, correlation):
    """Buffers that a branch clears: a product with fewer ranks than the basis, third order, one to three interactions (radial table)."""
    structs = [synth.fcc_supercell(2, 3.65, 0.05, seed=2, species=(13, 29), fractions=(0.5, 0.5))]
    model, _, _ = make_models(2, 64, [13, 29], 4.5, 20.0, torch.float32, num_layers=layers, Lmax=Lmax, correlation=correlation)
    data = to_device(oracle_batch(structs, [13, 29], 4.5, torch.float32), DEV)
    direct = {k: v.clone() for k, v in model(data).items() if v is not None}
    for n in range(10):
        out = model(data)
        for k, v in direct.items():
            assert torch.equal(out[k], v), (n, k)
    assert model.graph_replays() >= 9
