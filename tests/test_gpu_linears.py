"""The linears at the sizes where their tiles end: the double-precision kernel (32 x 32 tiles, K steps of 16) with species that own
one atom, one tile less a row, exactly one tile and one row more; the products of several correlation orders in one accumulator loop, on
the CUDA cores and, with more work, on the tensor cores, mixed with widths that those do not take.  The limit in work between the two: sizes on
both sides, and all linears of a pass above it.  Against the oracle."""
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


def _atom_linear_work(plan):
    """Multiply-adds per atom of the calls of a pass whose rows are atoms, by name (fp32, gated scalars, skip connections aware)."""
    C2, L, out = plan.C * plan.C, plan.L, {}
    for t, lp in enumerate(plan.layers):
        out[f"t{t}.down"] = sum((2 * l + 1) * lp.k[l] * (L + 2 if l == 0 else 1) for l in range(L + 1)) * C2
        out[f"t{t}.nl"] = (L + 1) ** 2 * C2
        orders = [1 + a + b + (1 if lp.has_res else 0) for a, b in zip(lp.kp if plan.correlation > 1 else [0] * len(lp.out_ls), lp.kp3)]
        out[f"t{t}.coef"] = sum((2 * l + 1) * k for l, k in zip(lp.out_ls, orders)) * C2
        if not lp.scalar_src:
            out[f"t{t}.up"] = sum(2 * l + 1 for l in lp.in_ls) * C2
    return out


@pytest.mark.parametrize("correlation", [1, 2, 3])
@pytest.mark.parametrize("channels", [64, 96, 128])
def test_products_of_several_orders_on_the_tensor_cores(channels, correlation):
    """The same on so many atoms that the coefficients of the lower interaction are above the limit (channels that are no multiple of 64
    leave all but the widest results to the CUDA cores)."""
    counts = (8, 136, 344, 536 if channels == 64 else 24)
    model, oracle, _ = make_models(2, channels, [1, 6, 7, 8], 3.0, 20.0, torch.float32, correlation=correlation)
    work = _atom_linear_work(model.readout_fn.plan)
    assert sum(counts) * min(work["t0.coef"], work["t0.down"]) > SMALL
    data = oracle_batch([_cluster(counts, (1, 6, 7, 8))], [1, 6, 7, 8], 3.0, torch.float32)
    check_parity(model(to_device(data, torch.device("cuda:0"))), oracle(data), data["ptr"], torch.float32, f"C{channels} correlation {correlation}")


@pytest.mark.parametrize("L,channels,cells", [(2, 64, 10), (3, 128, 6)])
def test_all_linears_on_the_tensor_cores(L, channels, cells):
    """Every linear of the lower interactions and of the radial MLP above the limit: FCC copper and aluminium with twelve neighbours per atom,
    path weights in memory."""
    struct = synth.fcc_supercell(cells, 3.61, 0.05, seed=9, species=(13, 29), fractions=(0.5, 0.5))
    n = len(struct["positions"])
    keep = np.arange(n) < (1024 if L == 2 else 512)  # a block with surfaces
    struct = synth.Structure(positions=struct["positions"][keep], atomic_numbers=struct["atomic_numbers"][keep], cell=struct["cell"] * 2.0, pbc=struct["pbc"])
    model, oracle, _ = make_models(L, channels, [13, 29], 3.0, 12.0, torch.float32)
    model.set_radial_table(False)
    data = oracle_batch([struct], [13, 29], 3.0, torch.float32)
    n, work = int(keep.sum()), _atom_linear_work(model.readout_fn.plan)
    assert n * min(work[k] for k in ("t0.down", "t0.nl", "t0.coef", "t1.up", "t1.down", "t1.nl")) > SMALL
    assert data["edge_index"].shape[1] * 2 * 64 * 64 > SMALL  # two interactions' hidden layers in one call
    check_parity(model(to_device(data, torch.device("cuda:0"))), oracle(data), data["ptr"], torch.float32, f"L{L} C{channels}")


@pytest.mark.parametrize("call,L,channels", [("t0.nl", 2, 64), ("t0.down", 3, 128), ("t0.nl", 3, 128)])
def test_both_sides_of_the_work_limit(call, L, channels):
    """The largest number of atoms with which a call is within the limit and one atom more: every four-atom crystal of the batch has the
    energy and the forces that it has alone, on both sides, and they are the oracle's."""
    model, oracle, _ = make_models(L, channels, [13, 29], 3.0, 12.0, torch.float32)
    n = SMALL // _atom_linear_work(model.readout_fn.plan)[call]
    crystal = synth.fcc_supercell(1, 3.61, 0.05, seed=4, species=(13, 29), fractions=(0.5, 0.5))
    lone = synth.Structure(positions=np.zeros((1, 3)), atomic_numbers=np.array([29]), cell=np.eye(3) * 30.0, pbc=(True, True, True))
    one = oracle_batch([crystal], [13, 29], 3.0, torch.float32)
    ref = oracle(one)
    for atoms in (n, n + 1):
        structs = [crystal] * (atoms // 4) + [lone] * (atoms % 4)
        data = oracle_batch(structs, [13, 29], 3.0, torch.float32)
        out = model(to_device(data, torch.device("cuda:0")))
        for g in (0, atoms // 4 - 1):
            part = {"energy": out["energy"][g:g + 1], "forces": out["forces"][4 * g:4 * g + 4], "stress": out["stress"][g:g + 1],
                    "virials": out["virials"][g:g + 1], "node_energy": out["node_energy"][4 * g:4 * g + 4]}
            check_parity(part, ref, one["ptr"], torch.float32, f"{call} {atoms} atoms")


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
