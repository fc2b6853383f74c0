"""The SO(2) linears of the edge block on FP16 parts of scaled operands (fp32 models): one edge and several tiles of them, channel counts whose
linears are 64 and 128 columns wide, cluster expansions narrower than a warp, heads that a warp cannot reduce, steps in pairs and a
single last one; and operands that powers of two bring far from one."""
import pytest
import torch

from helpers import make_models, oracle_batch, to_device
from tace_b200 import synth
from test_gpu_parity import run_case

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n,nmax,channels,heads,hidden,mmax", [
    (1, 2, 64, 4, 32, 2),    # a few edges
    (3, 7, 64, 1, 48, 1),    # K = 192 of the way down: steps in pairs, widths that are no multiple of 128
    (4, 9, 96, 2, 40, 2),    # 48 channels per head; K = 160: a single last step, warps of the cluster expansion over two edges
    (6, 16, 128, 8, 32, 2),  # several row tiles, the widths of the example configuration
])
def test_linears_over_edges(n, nmax, channels, heads, hidden, mmax):
    run_case(synth.random_crystals(n, seed=7 + n, nmin=2, nmax=nmax, zmax=3), 3, channels, [1, 2, 3], 4.5, torch.float32, radial={"apply_cutoff": False},
             tece={"num_head": heads, "edge_ace_hidden": hidden, "mmax": mmax})


@pytest.mark.parametrize("power", [-24, 17, 30])
def test_powers_of_two_leave_no_trace(power):
    """Radial weights times 2^p and the linears that read the weighted features times 2^-p are the same function; every scale is a power of
    two, so not a bit of the results may move."""
    model, _, _ = make_models(3, 64, [1, 2, 3], 4.5, 20.0, torch.float32, seed=2, radial={"apply_cutoff": False},
                              tece={"num_head": 4, "edge_ace_hidden": 32, "mmax": 2})
    gpu = to_device(oracle_batch(synth.random_crystals(3, seed=9, nmin=4, nmax=12, zmax=3), [1, 2, 3], 4.5, torch.float32), DEV)
    before = {k: v.clone() for k, v in model(gpu).items() if v is not None}
    sd = model.state_dict()
    last = max(k for k in sd if ".interactions.1.edge_info.mlp." in k and k.endswith(".weight") and sd[k].dim() == 2)
    scaled = {k: v.clone() for k, v in sd.items()}
    scaled[last] *= 2.0 ** power
    for k in scaled:
        if ".interactions.1.rejector.linear_" in k and "linear_down" not in k and k.endswith(".weight"):
            scaled[k] *= 2.0 ** -power
    model.load_state_dict(scaled)
    after = model(gpu)
    assert torch.isfinite(before["forces"]).all()
    for k, v in before.items():
        assert torch.equal(after[k], v), k


def _rank_one(n_edges):
    """Edge block of rank 1 and order 1 at 64 channels: its key and query linears take exactly three K steps per result on average (K = 128 for
    order 0, two rows of K = 64 for order 1), the line between the two kernels."""
    model, _, _ = make_models(1, 64, [13, 29], 5.0, 40.0, torch.float32, radial={"apply_cutoff": False}, tece={"num_head": 4, "edge_ace_hidden": 64, "mmax": 1})
    data = to_device(oracle_batch([synth.fcc_supercell(3, 3.65, 0.05, seed=2, species=(13, 29), fractions=(0.5, 0.5))], [13, 29], 5.0, torch.float32), DEV)
    assert data["edge_index"].shape[1] > n_edges
    keep = torch.randperm(data["edge_index"].shape[1], generator=torch.Generator().manual_seed(0))[:n_edges].to(DEV)
    return model, dict(data, edge_index=data["edge_index"][:, keep].contiguous(), edge_shifts=data["edge_shifts"][keep].contiguous())


@pytest.mark.parametrize("n_edges", [1985, 2049])
def test_replays_take_the_kernels_of_the_direct_pass_on_the_line(n_edges):
    """2 049 edges fill 17 tiles of 128 and their pairs 33, the 2 176 of the capacity 17 and 34: a count of tiles puts the two on
    different sides of the line."""
    model, data = _rank_one(n_edges)
    direct = {k: v.clone() for k, v in model(data).items() if v is not None}
    assert model.graph_replays() == 0
    for n in range(3):
        out = model(data)
        for k, v in direct.items():
            assert torch.equal(out[k], v), (n, k)
    assert model.graph_replays() >= 2


def _launched(model, data, kernel):
    """Launches of kernels whose name holds `kernel` in one evaluation, kernel by kernel."""
    model.set_graph_mode(False)
    model(data)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        model(data)
        torch.cuda.synchronize()
    assert any("tc_gemm" in e.name for e in prof.events())
    return sum(kernel in e.name for e in prof.events())


def test_the_number_of_edges_does_not_choose_the_kernel():
    """The same shapes run the same kernels whatever the last tile holds (128 edges and none, one, half of them, ...)."""
    seen = {n: _launched(*_rank_one(n), "tc_gemm_fp16_kernel") for n in (2048, 2049, 2112, 2113, 2175)}
    assert len(set(seen.values())) == 1, seen
