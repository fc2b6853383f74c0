"""Edge views and replayed passes: edge lists in any order (one and several scan blocks, more and fewer atoms than the one-block
species sort takes), and edge counts that change from call to call under one captured graph."""
import pytest
import torch

from tace_b200 import synth
from tace_b200.graph import build_batch
from helpers import make_models

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("reps", [1, 3, 10, 13])  # 4, 108, 4 000 and 8 788 atoms
def test_shuffled_edges_give_the_same_result(reps):
    s = synth.fcc_supercell(reps, 3.61, 0.05, seed=reps, species=(13, 29), fractions=(0.3, 0.7))
    model, _, _ = make_models(1, 32, [13, 29], 3.0, 12.0, torch.float64, targets=("energy", "forces", "stress", "edge_forces"))
    data = build_batch(synth.collate([s]), [13, 29], 3.0, torch.float64, DEV)
    perm = torch.randperm(data["edge_index"].shape[1], device=DEV, generator=torch.Generator(DEV).manual_seed(1))
    shuffled = dict(data, edge_index=data["edge_index"][:, perm].contiguous(), edge_shifts=data["edge_shifts"][perm].contiguous())
    a, b = model(data), model(shuffled)
    assert (a["energy"] - b["energy"]).abs().max().item() <= 1e-9 * len(s["positions"])
    assert (a["forces"] - b["forces"]).abs().max().item() <= 1e-9
    assert (a["edge_forces"][perm] - b["edge_forces"]).abs().max().item() <= 1e-9


@pytest.mark.parametrize("kw", [{}, dict(radial={"apply_cutoff": False}, tece={"num_head": 4, "edge_ace_hidden": 8, "mmax": 2})])
def test_replay_with_changing_edge_counts(kw):
    """Frames of one structure whose lists differ by a few edges share a captured pass; every result equals the launch-by-launch
    one bit for bit."""
    torch.manual_seed(0)
    s = synth.fcc_supercell(3, 3.61, 0.05, seed=9, species=(13, 29), fractions=(0.5, 0.5))
    model, _, _ = make_models(2, 32, [13, 29], 4.0, 18.0, torch.float32, targets=("energy", "forces", "stress", "edge_forces"), **kw)
    data = build_batch(synth.collate([s]), [13, 29], 4.0, torch.float32, DEV)
    E = data["edge_index"].shape[1]
    frames = [dict(data, edge_index=data["edge_index"][:, :E - k].contiguous(), edge_shifts=data["edge_shifts"][:E - k].contiguous())
              for k in (0, 3, 1, 7, 0, 5)]
    replayed = [{k: v.clone() for k, v in model(f).items() if v is not None} for f in frames]
    assert model.graph_replays() >= 3
    model.set_graph_mode(False)
    for f, r in zip(frames, replayed):
        for k, v in model(f).items():
            if v is not None:
                assert torch.equal(v, r[k]), k
    assert model.device_error() == 0


@pytest.mark.parametrize("reps", [2, 13])  # species sorted by one block, by the device-wide sort
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_species_outside_the_element_list_give_nan_in_their_graph_only(reps, dtype):
    """An index that a caller puts on the device wrongly addresses nothing: its structure's energy is NaN, the other one's and the
    next evaluation's are what they were (the captured pass included)."""
    good = synth.fcc_supercell(reps, 3.61, 0.05, seed=4, species=(13, 29), fractions=(0.5, 0.5))
    other = synth.fcc_supercell(2, 3.61, 0.05, seed=5, species=(13, 29), fractions=(0.5, 0.5))
    model, _, _ = make_models(2, 64, [13, 29], 3.0, 12.0, dtype, targets=("energy", "forces"))
    data = build_batch(synth.collate([good, other]), [13, 29], 3.0, dtype, DEV)
    want = {k: v.clone() for k, v in model(data).items() if v is not None}
    n = len(good["positions"])
    wrong = data["species"].clone()
    wrong[n + 1], wrong[n + 4], wrong[n + 5], wrong[n + 9] = -1, 2, 1 << 20, -(1 << 31)
    tol = dict(rtol=0.0, atol=(1e-4 if dtype == torch.float32 else 1e-9) * n)
    for _ in range(3):
        out = model(dict(data, species=wrong))
        assert torch.isnan(out["energy"][1]) and torch.isnan(out["node_energy"][[n + 1, n + 4, n + 5, n + 9]]).all()
        assert torch.allclose(out["energy"][0], want["energy"][0], **tol)
        assert torch.isfinite(out["forces"][:n]).all() and torch.isfinite(out["node_energy"][:n]).all()
    for _ in range(2):
        out = model(data)
        assert torch.allclose(out["energy"], want["energy"], **tol) and torch.isfinite(out["forces"]).all()
    assert model.device_error() == 0
