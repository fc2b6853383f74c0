"""The work a user of this framework has it do: energies, forces and stresses of the tensor atomic cluster expansion
potential through the public entry points, from one small cell in an ASE loop to a domain-decomposed MD block.

A case is a dictionary; ``kind`` names the entry point:

``calc``      ``TACEAseCalc.calculate`` on consecutive frames of one structure (relaxation or MD driven from Python): host
              arrays in, host arrays out, a neighbour list that changes with every frame.
``batch``     ``TensorModel.forward`` on a batch whose neighbour list is on the GPU already.
``e2e``       ``build_batch`` + ``TensorModel.forward`` from pinned host buffers (screening, data sets).
``torchsim``  ``TACETorchSimCalc.forward``: several systems that live on the GPU, neighbour list and evaluation.
``md``        one velocity-Verlet step of ``DomainMD`` (halo rows, skin list, exchange between the layers).

Weights are random (one fixed draw per architecture, as a program loads one checkpoint and evaluates many structures with
it); structures come from the generators of ``tace_b200.synth`` with the seed.
"""
from types import SimpleNamespace

import numpy as np
import torch

import tace_b200
from tace_b200 import synth
from tace_b200.graph import build_batch, z_to_index
from tace_b200.interface.ase_calculator import TACEAseCalc
from tace_b200.interface.torchsim import TACETorchSimCalc
from tace_b200.md import DomainMD, masses_for, maxwell_boltzmann
from tace_b200.pack import ModelPlan

# material: elements of the model, cutoff, mean number of neighbours, atoms per unit of "size"
MATERIALS = {
    "cu": dict(elements=[29], cutoff=5.0, degree=42.75),                            # FCC, size = cells per side
    "cual": dict(elements=[13, 29], cutoff=5.0, degree=42.1),                       # FCC alloy, size = cells per side
    "bcc": dict(elements=[23, 24, 26, 27, 28], cutoff=6.0, degree=64.2),            # five-component BCC, size = cells per side
    "water": dict(elements=[1, 8], cutoff=6.0, degree=86.7),                        # size = molecules
    "crystals": dict(elements=list(range(1, 90)), cutoff=6.0, degree=62.5),         # random triclinic cells of 8..64 atoms, size = cells
}
TARGETS = {"efs": ["energy", "forces", "stress"], "ef": ["energy", "forces"], "e": ["energy"]}


def listed():
    f32, f64 = "float32", "float64"
    return [
        # a 32-atom cell relaxed or propagated from Python: latency, launches and host work are everything
        dict(name="calc_cu32", kind="calc", material="cu", size=2, frames=6, systems=1, L=2, Lmax=2, C=64, dtype=f32, tece=False, targets="efs"),
        # the double-precision configuration (256-atom copper cell), same loop
        dict(name="calc_cu256_f64", kind="calc", material="cu", size=4, frames=2, systems=1, L=2, Lmax=2, C=64, dtype=f64, tece=False, targets="efs"),
        # the reference's default model shape (Lmax 2, lmax 3, 64 channels) on an alloy cell of 1 372 atoms
        dict(name="batch_cual1372", kind="batch", material="cual", size=7, frames=1, systems=1, L=3, Lmax=2, C=64, dtype=f32, tece=False, targets="efs"),
        # the headline batch: 64 random crystals, 89 elements, resident
        dict(name="batch_crystals64", kind="batch", material="crystals", size=64, frames=1, systems=1, L=3, Lmax=3, C=128, dtype=f32, tece=False, targets="efs"),
        # a small batch of the same, end to end from pinned host memory
        dict(name="e2e_crystals16", kind="e2e", material="crystals", size=16, frames=1, systems=1, L=3, Lmax=3, C=128, dtype=f32, tece=False, targets="efs"),
        # screening by energy only (forward pass), an odd number of crystals
        dict(name="e2e_crystals33_energy", kind="e2e", material="crystals", size=33, frames=1, systems=1, L=3, Lmax=3, C=128, dtype=f32, tece=False, targets="e"),
        # eight water boxes of 192 atoms propagated together on the GPU
        dict(name="torchsim_water8x192", kind="torchsim", material="water", size=64, frames=1, systems=8, L=3, Lmax=3, C=128, dtype=f32, tece=False, targets="efs"),
        # one large liquid box, energy and forces
        dict(name="batch_water32400", kind="batch", material="water", size=10800, frames=1, systems=1, L=3, Lmax=3, C=128, dtype=f32, tece=False, targets="ef"),
        # the edge-block model on a 128-atom alloy cell driven from Python
        dict(name="calc_tece128", kind="calc", material="bcc", size=4, frames=2, systems=1, L=3, Lmax=3, C=128, dtype=f32, tece=True, targets="efs"),
        # the edge-block model on 8 192 atoms
        dict(name="batch_tece8192", kind="batch", material="bcc", size=16, frames=1, systems=1, L=3, Lmax=3, C=128, dtype=f32, tece=True, targets="efs"),
        # one MD step of a 131 072-atom block (the share of one GPU in an 8-GPU run of the million-atom system)
        dict(name="md_cual131k", kind="md", material="cual", size=32, frames=1, systems=1, L=2, Lmax=2, C=64, dtype=f32, tece=False, targets="ef"),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["calc", "calc", "batch", "batch", "e2e", "torchsim", "md", "tece"])
    L, Lmax, C = rng.choice([(2, 2, 64), (3, 3, 128), (3, 2, 64), (1, 1, 32), (2, 1, 96), (2, 2, 128)])
    case = dict(kind=kind, material="cual", size=1, frames=1, systems=1, L=L, Lmax=Lmax, C=C, dtype="float32", tece=False, targets="efs")
    if kind == "calc":
        case.update(material=rng.choice(["cu", "cual"]), size=rng.randint(1, 5), frames=rng.randint(1, 6))
        if rng.random() < 0.3:
            case.update(dtype="float64", L=2, Lmax=2, C=64, frames=rng.randint(1, 2))
    elif kind == "batch":
        if rng.random() < 0.5:
            case.update(material="water", size=_log_int(rng, 20, 9000), targets=rng.choice(["efs", "ef", "e"]))
        else:
            case.update(material="cual", size=_log_int(rng, 3, 20), targets=rng.choice(["efs", "ef", "e"]))
    elif kind == "e2e":
        case.update(material="crystals", size=_log_int(rng, 1, 64), L=3, Lmax=3, C=128, targets=rng.choice(["efs", "e"]))
    elif kind == "torchsim":
        case.update(material="water", size=_log_int(rng, 20, 200), systems=_log_int(rng, 1, 24))
    elif kind == "md":
        case.update(material="cual", size=_log_int(rng, 6, 30), targets="ef")
        if rng.random() < 0.5:
            case.update(L=2, Lmax=2, C=64)
    else:
        size = _log_int(rng, 3, 14)
        case.update(kind="calc" if size < 6 else "batch", material="bcc", size=size, L=3, Lmax=3, C=128, tece=True)
    return case


# ---- structures -------------------------------------------------------------------------------------------------
def _water(n_mol, seed):
    side = 1
    while side ** 3 < n_mol:
        side += 1
    return synth.water_box(n_side=side, box=68.6 * (n_mol / 10800) ** (1.0 / 3.0), seed=seed, n_mol=n_mol)


def _structures(case, seed):
    m, size = case["material"], case["size"]
    if m == "crystals":
        # sizes spread over 8..64 atoms in the same way for every seed; cells, species and coordinates from the seed
        return [synth.random_crystals(1, seed=seed + 1000 * k, nmin=n, nmax=n)[0] for k, n in enumerate(8 + (37 * k + 28) % 57 for k in range(size))]
    if m == "water":
        return [_water(size, seed + 1000 * k) for k in range(case["systems"])]
    if m == "cu":
        return [synth.fcc_supercell(size, 3.61, 0.05, seed=seed)]
    if m == "cual":
        return [synth.fcc_supercell(size, 3.65, 0.05, seed=seed, species=(13, 29), fractions=(0.1, 0.9))]
    return [synth.bcc_supercell(size, 2.87, 0.08, seed=seed, species=MATERIALS["bcc"]["elements"])]


def _n_atoms(case):
    size = case["size"]
    return {"crystals": 36 * size, "water": 3 * size * case["systems"], "cu": 4 * size ** 3, "cual": 4 * size ** 3, "bcc": 2 * size ** 3}[case["material"]]


class _Atoms:
    """The four getters of ``ase.Atoms`` that a calculator reads."""

    def __init__(self, s, positions):
        self._s, self._positions = s, positions

    def get_positions(self):
        return self._positions

    def get_atomic_numbers(self):
        return self._s["atomic_numbers"]

    def get_cell(self):
        return self._s["cell"]

    def get_pbc(self):
        return np.array(self._s["pbc"])


# ---- models: one per architecture, as a program loads one checkpoint; the last one used is kept ------------------------
_loaded = {}


def _config(case):
    mat = MATERIALS[case["material"]]
    extra = synth.WORKLOADS["tece8192_fp32"]["model"] if case["tece"] else {}
    return synth.model_config(case["L"], case["C"], mat["cutoff"], mat["elements"], mat["degree"], Lmax=case["Lmax"], **extra)


def _model(case):
    key = (case["material"], case["L"], case["Lmax"], case["C"], case["dtype"], case["tece"], case["kind"] == "md")
    if key not in _loaded:
        _loaded.clear()
        torch.cuda.empty_cache()
        before = torch.get_default_dtype()
        torch.set_default_dtype(getattr(torch, case["dtype"]))
        try:
            torch.manual_seed(0)
            _loaded[key] = tace_b200.TensorModel(tace_b200.e3nnTACE(**_config(case)))
        finally:
            torch.set_default_dtype(before)
    model = _loaded[key]
    if case["kind"] != "md":
        model.reset_target_property(list(TARGETS[case["targets"]]))
    return model


def prepare(case, seed):
    device, dtype = torch.device("cuda"), getattr(torch, case["dtype"])
    mat, kind = MATERIALS[case["material"]], case["kind"]
    structures = _structures(case, seed % (1 << 30))
    model = _model(case)
    if kind == "calc":  # a trajectory: every frame moves the atoms a little further
        s, rng = structures[0], np.random.default_rng(seed + 7)
        frames, x = [], s["positions"]
        for _ in range(case["frames"]):
            frames.append(_Atoms(s, x))
            x = x + rng.normal(0.0, 0.02, size=x.shape)
        return {"kind": kind, "calc": TACEAseCalc(model, device="cuda"), "frames": frames}
    if kind == "torchsim":
        b = synth.collate(structures)
        state = SimpleNamespace(positions=torch.as_tensor(b["positions"], dtype=dtype, device=device),
                                row_vector_cell=torch.as_tensor(b["lattice"], dtype=dtype, device=device), pbc=(True, True, True),
                                atomic_numbers=torch.as_tensor(b["atomic_numbers"], device=device),
                                system_idx=torch.as_tensor(b["batch"], device=device))
        return {"kind": kind, "calc": TACETorchSimCalc(model, device=device, dtype=dtype), "state": state}
    if kind == "md":
        s = structures[0]
        masses = masses_for(s["atomic_numbers"])
        md = DomainMD(model, s["cell"], s["positions"], s["atomic_numbers"], velocities=maxwell_boltzmann(masses, 300.0, seed % (1 << 30)),
                      masses=masses, dt=1.0, skin=1.0, device=device, temperature=300.0, friction=0.01, seed=seed % (1 << 30))
        return {"kind": kind, "md": md}
    host = synth.collate(structures)
    host["species"] = z_to_index(host["atomic_numbers"], mat["elements"])
    if kind == "e2e":
        pinned = {k: torch.as_tensor(v).pin_memory() for k, v in host.items()}
        return {"kind": kind, "model": model, "host": pinned, "elements": mat["elements"], "cutoff": mat["cutoff"], "dtype": dtype, "device": device}
    return {"kind": kind, "model": model, "data": build_batch(host, mat["elements"], mat["cutoff"], dtype, device)}


def run(state):
    kind = state["kind"]
    if kind == "calc":
        out = []
        for atoms in state["frames"]:
            state["calc"].calculate(atoms)
            out.append(state["calc"].results)
        return out
    if kind == "torchsim":
        return state["calc"](state["state"])
    if kind == "md":
        md = state["md"]
        md.step(1)
        return {"positions": md.positions, "velocities": md.velocities, "forces": md.forces, "node_energy": md.node_energy}
    if kind == "e2e":
        data = build_batch(state["host"], state["elements"], state["cutoff"], state["dtype"], state["device"])
        return state["model"](data)
    return state["model"](state["data"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _tp_macs(paths):
    """Multiply-adds per (edge, channel) of one contraction: the coupling applied to the source feature, then the weight."""
    return sum((2 * l3 + 1) * (2 * l1 + 2) for l1, _, l3 in paths)


def work(case):
    n = _n_atoms(case)
    edges = n * MATERIALS[case["material"]]["degree"]
    frames, real = case["frames"], 8 if case["dtype"] == "float64" else 4
    L, Lmax, C, layers = case["L"], case["Lmax"], case["C"], 2
    grad = case["targets"] != "e"
    opts = dict(tece_layers=[1], mmax=2, num_head=8, edge_ace_hidden=32, gate_m0=False, element2=True, product_bilinear=True,
                resnet_type="identity", product_agnostic=True, apply_cutoff=False, mlp_bias=True, mlp_layers=2) if case["tece"] else {}
    plan = ModelPlan(L, layers, C, len(MATERIALS[case["material"]]["elements"]), 2, Lnode=Lmax, **opts)
    D = (L + 1) ** 2
    per_edge, per_atom, weights = 0.0, 0.0, 0.0
    for lp in plan.layers:
        if lp.tece:
            for _, _, ci, co, n_in, n_out in plan.so2_linears():
                terms = [(1 if m == 0 else 2, n_in[m] * ci * n_out[m] * co) for m in range(len(n_in))]
                per_edge += sum(rows * size for rows, size in terms)
                weights += sum(size for _, size in terms)
        else:
            per_edge += C * _tp_macs(lp.tp_paths)
        rows_in, rows_out = sum(2 * l + 1 for l in lp.in_ls), sum(2 * l + 1 for l in lp.out_ls)
        down = sum((2 * l + 1) * lp.k[l] for l in range(L + 1)) + lp.k[0] * (L + 1)
        coef = sum((2 * l + 1) * (1 + k) for l, k in zip(lp.out_ls, lp.kp))
        per_atom += C * C * (rows_in + down + D + coef + rows_out * (2 if lp.has_res else 1))
        species = 1.0 if case["tece"] else plan.n_el * (1.0 - (1.0 - 1.0 / plan.n_el) ** n)  # matrices of the elements present
        weights += C * C * (len(lp.in_ls) + sum(lp.k) + lp.k[0] * L + (L + 1) + species * (sum(lp.kp) + 2 * len(lp.out_ls)) + len(lp.out_ls))
    passes = 3 if grad else 1  # the backward pass has two contractions for each one of the forward pass
    flops = 2.0 * (passes * per_edge * edges + (2 if grad else 1) * per_atom * n)
    # edge list (index pair, shift), positions and species in, energies and forces out, weights once
    moved = edges * (16 + 3 * real) + n * (3 * real + 4 + real + (3 * real if grad else 0)) + real * weights
    return {"bytes": float(frames * moved), "flops": float(frames * flops)}


def tolerance(case):
    if case["dtype"] == "float64":
        return {"rel": 1e-10, "max": 1e-8}
    return {"rel": 2e-5, "max": 1e-3}
