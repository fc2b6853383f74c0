"""ASE calculator and LAMMPS ML-IAP entry points, driven with stand-in `atoms` / `data` objects."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from tace_b200.interface import TACEAseCalc, TACELammpsCalc
from tace_b200.interface.ase_calculator import export_tace
from helpers import make_models, oracle_batch, to_device

pytestmark = pytest.mark.gpu


class FakeAtoms:
    def __init__(self, s):
        self.s = s
        self.info = {}

    def get_positions(self): return self.s["positions"]
    def get_atomic_numbers(self): return self.s["atomic_numbers"]
    def get_cell(self): return self.s["cell"]
    def get_pbc(self): return np.array(self.s["pbc"])
    def __len__(self): return len(self.s["positions"])


def test_ase_calculator_matches_oracle_and_pt_roundtrip(tmp_path):
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=0, species=(13, 29), fractions=(0.5, 0.5))
    model, oracle, cfg = make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64)
    path = str(tmp_path / "model.pt")
    export_tace(model, path)
    calc = TACEAseCalc(path, device="cuda:0")
    calc.calculate(FakeAtoms(s))
    ref = oracle(oracle_batch([s], [13, 29], 4.0, torch.float64))
    assert abs(calc.results["energy"] - ref["energy"].item()) < 1e-8 * len(s["positions"])
    assert calc.results["free_energy"] == calc.results["energy"]
    assert np.abs(calc.results["forces"] - ref["forces"].numpy()).max() < 1e-7
    assert calc.results["stress"].shape == (3, 3)
    assert np.abs(calc.results["stress"] - ref["stress"][0].numpy()).max() < 1e-7
    assert set(calc.implemented_properties) >= {"energy", "free_energy", "forces", "stress"}


def test_ase_calculator_calls_the_model_as_a_module():
    """Forward hooks run, and an object put in the model's place is used through its call: here the mean of two models, whose
    results are separate tensors and whose energy has no dimension."""
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=0, species=(13, 29), fractions=(0.5, 0.5))
    models = [make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64, seed=k)[0] for k in (0, 5)]
    singles = []
    for model in models:
        calls = []
        handle = model.register_forward_hook(lambda *_: calls.append(1))
        calc = TACEAseCalc(model, device="cuda:0")
        calc.calculate(FakeAtoms(s))
        handle.remove()
        assert len(calls) == 1
        singles.append(calc.results)

    def mean(data):
        a, b = (m(data) for m in models)
        return {"energy": (0.5 * (a["energy"] + b["energy"]))[0], "forces": 0.5 * (a["forces"] + b["forces"]), "stress": None}

    calc.model = mean
    calc.calculate(FakeAtoms(s))
    assert set(calc.results) == {"energy", "free_energy", "forces"}
    assert abs(calc.results["energy"] - 0.5 * (singles[0]["energy"] + singles[1]["energy"])) < 1e-10
    assert np.abs(calc.results["forces"] - 0.5 * (singles[0]["forces"] + singles[1]["forces"])).max() < 1e-12


def _contract(model, seen):
    """An object in a model's place that works from the fields of the reference's ``forward(data)`` contract alone."""
    def call(data):
        fields = {k: data[k] for k in ("positions", "lattice", "node_attrs", "edge_index", "edge_shifts", "batch", "ptr")}
        n = fields["positions"].shape[0]
        assert fields["node_attrs"].dtype == fields["positions"].dtype and (fields["node_attrs"].sum(1) == 1).all()
        assert fields["batch"].dtype == fields["ptr"].dtype == torch.int64 and fields["batch"].shape == (n,)
        assert fields["edge_shifts"].dtype in (torch.int32, torch.float64)
        assert torch.equal(fields["ptr"], torch.cat([fields["ptr"][:1] * 0, torch.bincount(fields["batch"]).cumsum(0)]))
        assert torch.equal(fields["node_attrs"].argmax(1), data["species"].long())
        seen.append(set(data))
        return model(fields)
    return call


def test_ase_calculator_hands_others_the_whole_contract():
    """Whatever is called in the place of this package's own forward, or looks on, gets every field of the contract in its types: an
    object put there, a subclass, hooks of the model and of all modules, a forward set on the object."""
    from tace_b200 import TensorModel

    s = synth.fcc_supercell(2, 3.61, 0.05, seed=0, species=(13, 29), fractions=(0.5, 0.5))
    model = make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64)[0]
    calc = TACEAseCalc(model, device="cuda:0")
    atoms, seen = FakeAtoms(s), []
    calc.calculate(atoms)
    want = calc.results
    inner = make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64)[0]
    look = _contract(inner, seen)

    def check(count):
        calc.calculate(atoms)
        assert len(seen) == count
        assert calc.results["energy"] == want["energy"] and np.array_equal(calc.results["forces"], want["forces"])

    calc.model = look
    check(1)
    calc.model = model
    for n, register in enumerate((model.register_forward_pre_hook, model.register_forward_hook,
                                  torch.nn.modules.module.register_module_forward_pre_hook)):
        busy = []

        def hook(module, args, *_):
            if module is model and not busy:  # `look` calls a model itself
                busy.append(1)
                look(args[0])

        handle = register(hook)
        check(2 + n)
        handle.remove()

    class Sub(TensorModel):
        def forward(self, data):
            return look(data)

    model.__class__ = Sub
    check(5)
    model.__class__ = TensorModel
    model.forward = look
    check(6)
    del model.forward
    check(6)


class FakeLammpsData:
    """Single-rank stand-in for the Kokkos ML-IAP data object: local atoms plus periodic ghost copies."""

    def __init__(self, s, cutoff, elements, device):
        from oracle.neighbour_list import neighbour_list
        ei, es = neighbour_list(s["positions"], s["cell"], s["pbc"], cutoff)
        n = len(s["positions"])
        ghost_of = {}          # (owner, shift) -> ghost index
        owners = []
        pair_i, pair_j, rij = [], [], []
        for (src, dst), sh in zip(ei.T, es):
            # edge source -> target with vector r_dst - r_src + sh @ cell; LAMMPS pair (i = target, j = source or its ghost)
            key = (int(src), tuple(int(v) for v in -sh))
            if key[1] == (0, 0, 0):
                j = int(src)
            else:
                if key not in ghost_of:
                    ghost_of[key] = n + len(owners)
                    owners.append(int(src))
                j = ghost_of[key]
            pair_i.append(int(dst)); pair_j.append(j)
            rij.append(s["positions"][dst] - s["positions"][src] + sh @ s["cell"])
        zs = sorted(elements)
        species = [zs.index(int(z)) for z in s["atomic_numbers"]]
        self.nlocal, self.ntotal, self.npairs = n, n + len(owners), len(pair_i)
        self.owner = torch.tensor(owners, dtype=torch.int64, device=device)
        self.elems = torch.tensor(species + [species[o] for o in owners], dtype=torch.int32, device=device)
        self.rij = torch.tensor(np.array(rij), dtype=torch.float64, device=device)
        self.pair_i = torch.tensor(pair_i, dtype=torch.int32, device=device)
        self.pair_j = torch.tensor(pair_j, dtype=torch.int32, device=device)
        self.eatoms = torch.zeros(n, dtype=torch.float64, device=device)
        self.energy = None
        self.pair_forces = None
        self.exchanges = 0

    def forward_exchange(self, src, dst, vec_len):
        dst.copy_(src)
        dst[self.nlocal:] = src[self.owner]
        self.exchanges += 1

    def reverse_exchange(self, src, dst, vec_len):
        dst.copy_(src)
        dst[: self.nlocal].index_add_(0, self.owner, src[self.nlocal:])
        self.exchanges += 1

    def update_pair_forces(self, f):
        self.pair_forces = f.clone()


@pytest.mark.parametrize("num_layers", [1, 2, 3])
def test_lammps_mliap_with_ghost_exchange_matches_graph_mode(num_layers):
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=4, species=(13, 29), fractions=(0.5, 0.5))
    model, oracle, cfg = make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64, num_layers=num_layers)
    ref = oracle(oracle_batch([s], [13, 29], 4.0, torch.float64), compute_stress=False)
    dev = torch.device("cuda:0")
    data = FakeLammpsData(s, 4.0, [13, 29], dev)
    assert data.ntotal > data.nlocal
    calc = TACELammpsCalc(model)
    assert calc.element_types == ["Al", "Cu"] and abs(calc.rcutfac - 2.0) < 1e-12
    calc.compute_forces(data)
    n = data.nlocal
    assert abs(data.energy - ref["energy"].item()) < 1e-8 * n
    assert (data.eatoms.cpu() - ref["node_energy"]).abs().max().item() < 1e-8
    # forces as LAMMPS assembles them from pair forces (newton on): f_i -= f_ij, f_j += f_ij, ghosts folded back
    f = torch.zeros(data.ntotal, 3, dtype=torch.float64, device=dev)
    f.index_add_(0, data.pair_i.long(), -data.pair_forces)
    f.index_add_(0, data.pair_j.long(), data.pair_forces)
    f[:n].index_add_(0, data.owner, f[n:])
    assert (f[:n].cpu() - ref["forces"]).abs().max().item() < 1e-7
    assert data.exchanges == 2 * (num_layers - 1)


def test_lammps_requires_kokkos_exchange():
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=4)
    model, _, _ = make_models(2, 32, [29], 4.0, 20.0, torch.float64)
    data = FakeLammpsData(s, 4.0, [29], torch.device("cuda:0"))
    calc = TACELammpsCalc(model)

    class NoExchange:
        nlocal, ntotal, npairs, elems = data.nlocal, data.ntotal, data.npairs, data.elems
    with pytest.raises(RuntimeError, match="KOKKOS"):
        calc.compute_forces(NoExchange())


class FakeSimState:
    """The attributes of a torch_sim SimState that the model interface reads."""

    def __init__(self, structures, device):
        b = synth.collate(structures)
        self.positions = torch.as_tensor(b["positions"], device=device)
        self.row_vector_cell = torch.as_tensor(b["lattice"], device=device)
        self.pbc = torch.tensor([True, True, True], device=device)
        self.atomic_numbers = torch.as_tensor(b["atomic_numbers"], device=device)
        self.system_idx = torch.as_tensor(b["batch"], device=device)


def test_torchsim_model_matches_oracle_and_reuses_cached_setup():
    from tace_b200.interface import TACETorchSimCalc

    structs = synth.random_crystals(3, seed=12, nmin=4, nmax=10, zmax=3)
    model, oracle, cfg = make_models(2, 32, [1, 2, 3], 4.5, 20.0, torch.float64)
    ref = oracle(oracle_batch(structs, [1, 2, 3], 4.5, torch.float64))
    dev = torch.device("cuda:0")
    calc = TACETorchSimCalc(model, device=dev, dtype=torch.float64)
    state = FakeSimState(structs, dev)
    for _ in range(2):  # the second call reuses the cached species / pointers
        out = calc(state)
        n_per = torch.tensor([len(s["positions"]) for s in structs], dtype=torch.float64)
        assert ((out["energy"].cpu() - ref["energy"]).abs() / n_per).max() < 1e-8
        assert (out["forces"].cpu() - ref["forces"]).abs().max() < 1e-7
        assert (out["stress"].cpu() - ref["stress"]).abs().max() < 1e-7
    assert calc.compute_forces and calc.compute_stress and calc.device == dev and calc.dtype == torch.float64
    with pytest.raises(NotImplementedError):
        TACETorchSimCalc(model, device=dev, enable_cue=True)
    # an element outside the model's table is refused
    state.atomic_numbers = state.atomic_numbers.clone()
    state.atomic_numbers[0] = 7
    with pytest.raises(ValueError):
        calc(state)


def test_torchsim_model_hands_others_the_whole_contract():
    """The same for the TorchSim model, with this package's own list and with the systems' flags as a tensor."""
    from tace_b200.interface import TACETorchSimCalc

    structs = synth.random_crystals(3, seed=12, nmin=4, nmax=10, zmax=3)
    dev = torch.device("cuda:0")
    calc = TACETorchSimCalc(make_models(2, 32, [1, 2, 3], 4.5, 20.0, torch.float64)[0], device=dev, dtype=torch.float64)
    inner = make_models(2, 32, [1, 2, 3], 4.5, 20.0, torch.float64)[0]
    seen, state = [], FakeSimState(structs, dev)
    look = _contract(inner, seen)
    for pbc in ((True, True, True), state.pbc):
        state.pbc = pbc
        want = {k: v.clone() for k, v in calc(state).items()}
        shifts = []
        handle = calc.model.register_forward_pre_hook(lambda _, args: (look(args[0]), shifts.append(args[0]["edge_shifts"].dtype)) and None)
        out = calc(state)
        handle.remove()
        assert shifts == [torch.int32]  # what neighbour-list functions return
        for k, v in want.items():
            assert torch.equal(out[k], v), k
    assert len(seen) == 2


def test_lammps_mliap_with_the_tece_edge_block():
    """Edge-vector mode with ghost atoms for a model whose second interaction is the TECE edge block: ghost features arrive
    through the forward exchange, the gradients of ghost sources go back through the reverse exchange, and the gradient
    through the edge frames is part of the pair forces."""
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=6, species=(13, 29), fractions=(0.5, 0.5))
    model, oracle, cfg = make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64, radial={"apply_cutoff": False},
                                     tece={"num_head": 4, "edge_ace_hidden": 8, "mmax": 2})
    ref = oracle(oracle_batch([s], [13, 29], 4.0, torch.float64), compute_stress=False)
    dev = torch.device("cuda:0")
    data = FakeLammpsData(s, 4.0, [13, 29], dev)
    calc = TACELammpsCalc(model)
    calc.compute_forces(data)
    n = data.nlocal
    assert abs(data.energy - ref["energy"].item()) < 1e-8 * n
    f = torch.zeros(data.ntotal, 3, dtype=torch.float64, device=dev)
    f.index_add_(0, data.pair_i.long(), -data.pair_forces)
    f.index_add_(0, data.pair_j.long(), data.pair_forces)
    f[:n].index_add_(0, data.owner, f[n:])
    assert (f[:n].cpu() - ref["forces"]).abs().max().item() < 1e-7


@pytest.mark.parametrize("kw", [
    dict(zbl={"enable": True, "covalent_radii": {13: 1.5, 29: 1.6}}, scatter_norm="density"),
    dict(edge_update="element2", radial={"apply_cutoff": False, "bias": True, "hidden": [64, 64]}, gate_m0=False, use_alllayer=True),
    dict(product_nonlinear="silu_bilineargate", product_agnostic=True, resnet_linear_type="identity", correlation=2),
])
def test_lammps_mliap_with_model_options(kw):
    """Edge-vector mode with ghost atoms for the model options beyond the default: pair repulsion and learned edge density
    (sums over the edges into local atoms, species of ghost sources), element-dependent edge update with LayerNorm, gated
    bilinear product with identity skip."""
    s = synth.fcc_supercell(2, 3.61, 0.05, seed=10, species=(13, 29), fractions=(0.5, 0.5))
    model, oracle, cfg = make_models(2, 32, [13, 29], 4.0, 20.0, torch.float64, **kw)
    ref = oracle(oracle_batch([s], [13, 29], 4.0, torch.float64), compute_stress=False)
    dev = torch.device("cuda:0")
    data = FakeLammpsData(s, 4.0, [13, 29], dev)
    calc = TACELammpsCalc(model)
    calc.compute_forces(data)
    n = data.nlocal
    assert abs(data.energy - ref["energy"].item()) < 1e-8 * n
    assert (data.eatoms.cpu() - ref["node_energy"]).abs().max().item() < 1e-8
    f = torch.zeros(data.ntotal, 3, dtype=torch.float64, device=dev)
    f.index_add_(0, data.pair_i.long(), -data.pair_forces)
    f.index_add_(0, data.pair_j.long(), data.pair_forces)
    f[:n].index_add_(0, data.owner, f[n:])
    assert (f[:n].cpu() - ref["forces"]).abs().max().item() < 1e-7
