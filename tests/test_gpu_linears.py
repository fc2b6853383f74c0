"""The linears at the sizes where their tiles end: the double-precision kernel (32 x 32 tiles, K steps of 16) with species that own
one atom, one tile less a row, exactly one tile and one row more; the tensor-core kernel where the products of several
correlation orders share one accumulator loop, mixed with widths it does not take.  Against the oracle."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from helpers import check_parity, make_models, oracle_batch, to_device
from test_gpu_parity import run_case

pytestmark = pytest.mark.gpu


def _cluster(counts, elements):
    """Atoms on a jittered grid (about 2.4 A apart), counts[i] of elements[i]."""
    z = np.repeat(elements, counts)
    rng = np.random.default_rng(int(sum(counts)))
    n = int(np.ceil(len(z) ** (1.0 / 3.0)))
    grid = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)[: len(z)] * 2.4
    return synth.Structure(positions=grid + rng.normal(0.0, 0.05, grid.shape), atomic_numbers=rng.permutation(z), cell=np.eye(3) * (2.4 * n),
                           pbc=(True, True, True))


@pytest.mark.parametrize("L,channels", [(1, 32), (2, 96), (3, 32)])
def test_double_precision_tiles(L, channels):
    run_case([_cluster((1, 31, 32, 33), (1, 6, 7, 8))], L, channels, [1, 6, 7, 8], 3.0, torch.float64)


@pytest.mark.parametrize("correlation", [1, 2, 3])
@pytest.mark.parametrize("channels", [64, 96, 128])
def test_products_of_several_orders_in_one_loop(channels, correlation):
    run_case([_cluster((1, 17, 43, 3), (1, 6, 7, 8))], 2, channels, [1, 6, 7, 8], 3.0, torch.float32, correlation=correlation)


# Multiply-adds of a call up to which its linears run on the CUDA cores (kSmallLinear in csrc/engine.cu)
SMALL = 32 << 20


def _edge_linear_work(model, calls):
    """Multiply-adds per edge of the SO(2) linears numbered in `calls` (two rows per order above 0)."""
    linears = model.readout_fn.plan.so2_linears()
    return sum((1 if m == 0 else 2) * n_in[m] * ci * n_out[m] * co
               for _, _, ci, co, n_in, n_out in (linears[k] for k in calls) for m in range(len(n_in)))


@pytest.mark.parametrize("calls", [None, (5,), (0, 1)])
def test_replays_take_the_kernels_of_the_direct_pass(calls, monkeypatch):
    """A captured pass holds more edges than the list (its capacity), a direct one exactly the list's: with the last edge count below
    a limit in the work of the linears over edges, and the capacity above it, both run the same kernels and agree bit for bit.  The
    hidden layers of the radial MLPs of three interactions, and the SO(2) linears of two launches in the edge block's backward pass."""
    monkeypatch.setenv("TACE_B200_RADIAL_TABLE", "0")
    tece = {"num_head": 4, "edge_ace_hidden": 64, "mmax": 2} if calls else None
    model, _, _ = make_models(2, 64, [13, 29], 5.0, 40.0, torch.float32, num_layers=2 if calls else 3, tece=tece,
                              radial={"apply_cutoff": False} if calls else None)
    n_edges = SMALL // (_edge_linear_work(model, calls) if calls else 3 * 64 * 64)
    assert 32 <= n_edges <= 4096 and n_edges % (64 if n_edges <= 2048 else 128) != 0
    data = to_device(oracle_batch([synth.fcc_supercell(3, 3.65, 0.05, seed=2, species=(13, 29), fractions=(0.5, 0.5))], [13, 29], 5.0, torch.float32),
                     torch.device("cuda:0"))
    assert data["edge_index"].shape[1] > n_edges
    keep = torch.randperm(data["edge_index"].shape[1], generator=torch.Generator().manual_seed(0))[:n_edges].to("cuda:0")
    data = dict(data, edge_index=data["edge_index"][:, keep].contiguous(), edge_shifts=data["edge_shifts"][keep].contiguous())
    direct = {k: v.clone() for k, v in model(data).items() if v is not None}
    assert model.graph_replays() == 0
    for n in range(3):
        out = model(data)
        for k, v in direct.items():
            assert torch.equal(out[k], v), (n, k)
    assert model.graph_replays() >= 2


@pytest.mark.parametrize("n_el", [16, 17])
@pytest.mark.parametrize("n_atoms", [24, 40])
def test_per_species_linears_of_few_tiles(n_el, n_atoms):
    """Per-species linears of little more than the limit in work, for a model with the largest number of elements for which they stay on the
    CUDA cores and for one with an element more."""
    elements = list(range(1, n_el + 1))
    structs = synth.random_crystals(1, seed=5, nmin=n_atoms, nmax=n_atoms, zmax=n_el)
    model, oracle, _ = make_models(3, 128, elements, 4.0, 20.0, torch.float32)
    plan = model.readout_fn.plan.layers[0]
    rows = [n_atoms * (2 * l + 1) for l in plan.out_ls]
    assert SMALL < sum(r * (1 + k) for r, k in zip(rows, plan.kp)) * 128 * 128 <= 4 * SMALL and sum((r + 127) // 128 for r in rows) <= 8
    data = oracle_batch(structs, elements, 4.0, torch.float32)
    check_parity(model(to_device(data, torch.device("cuda:0"))), oracle(data), data["ptr"], torch.float32, f"{n_el} elements {n_atoms} atoms")
