"""The node linears on FP16 parts of scaled operands (fp32 models without the edge block): calls beyond the limit of the CUDA cores, one to four
warps per atom in the kernels that note the largest elements, ranks whose tiles are 126 rows, species with one row, a few and several
tiles, with and without a skip connection, and the backward pass alone (two elements)."""
import numpy as np
import pytest
import torch

from helpers import make_models, oracle_batch, to_device
from tace_b200 import synth
from tace_b200.md import DomainMD
from tace_b200.pack import LayerPlan
from test_gpu_parity import run_case

pytestmark = pytest.mark.gpu
MANY = list(range(1, 21))


@pytest.mark.parametrize("L,Lmax,channels,structs,zs,cutoff", [
    (3, 3, 128, lambda: synth.random_crystals(4, seed=31, nmin=9, nmax=23, zmax=20), MANY, 4.5),
    (3, 2, 64, lambda: synth.random_crystals(5, seed=32, nmin=20, nmax=40, zmax=20), MANY, 4.0),
    (3, 1, 32, lambda: synth.random_crystals(9, seed=33, nmin=38, nmax=44, zmax=20), MANY, 3.5),
    (2, 2, 128, lambda: [synth.fcc_supercell(4, 3.65, 0.05, seed=5, species=(13, 29), fractions=(0.02, 0.98))], [13, 29], 4.0),
])
@pytest.mark.parametrize("skip", ["aware", "identity"])
def test_species_linears(L, Lmax, channels, structs, zs, cutoff, skip):
    run_case(structs(), L, channels, zs, cutoff, torch.float32, Lmax=Lmax, resnet_linear_type=skip)


def _blocks(sd, key, ls, power):
    """Multiplies the blocks of the ranks `ls` of a linear of ranks 0..3 (equal blocks, one after the other) by 2^power."""
    w = sd[key]
    n = w.shape[-1] // 4
    for l in ls:
        w[..., l * n:(l + 1) * n] *= 2.0 ** power


@pytest.mark.parametrize("power", [-24, 20])
@pytest.mark.parametrize("where", ["gated", "output"])
def test_ranks_of_every_magnitude(power, where):
    """Rank 2 times 2^p between two linears is the same function: of the gated features, and of the features that a layer hands to the next one and to
    its skip connection.  Every scale is a power of two and belongs to one rank, so not a bit of the results may move."""
    structs = synth.random_crystals(4, seed=31, nmin=9, nmax=23, zmax=20)
    model, _, _ = make_models(3, 128, MANY, 4.5, 20.0, torch.float32, seed=4)
    gpu = to_device(oracle_batch(structs, MANY, 4.5, torch.float32), torch.device("cuda:0"))
    before = {k: v.clone() for k, v in model(gpu).items() if v is not None}
    sd = {k: v.clone() for k, v in model.state_dict().items()}
    pre = "readout_fn.representation."
    if where == "gated":
        down = sd[pre + "interactions.1.linear_down.weight"]
        n2, n3 = (LayerPlan(1, 2, 3).k[l] * 128 * 128 for l in (2, 3))
        down[down.numel() - n3 - n2:down.numel() - n3] *= 2.0 ** power
        _blocks(sd, pre + "interactions.1.linear_nonlinearity.weight", [2], -power)
    else:
        _blocks(sd, pre + "products.0.linear.weight", [2], power)
        _blocks(sd, pre + "interactions.1.linear_up.weight", [2], -power)
    model.load_state_dict(sd)
    after = model(gpu)
    assert torch.isfinite(before["forces"]).all()
    for k, v in before.items():
        assert torch.equal(after[k], v), k


def _launched(model, data):
    """Names of the kernels of one evaluation."""
    model.set_graph_mode(False)
    model(data)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        model(data)
        torch.cuda.synchronize()
    return [e.name for e in prof.events()]


@pytest.mark.parametrize("channels,structs,cutoff,zs,forward,backward", [
    (128, lambda: synth.random_crystals(4, seed=31, nmin=9, nmax=23, zmax=20), 4.5, MANY, True, True),
    (64, lambda: synth.random_crystals(5, seed=32, nmin=20, nmax=40, zmax=20), 4.0, MANY, True, False),
    (32, lambda: synth.random_crystals(9, seed=33, nmin=38, nmax=44, zmax=20), 3.5, MANY, False, False),
    (128, lambda: [synth.fcc_supercell(4, 3.65, 0.05, seed=5, species=(13, 29), fractions=(0.02, 0.98))], 4.0, [13, 29], False, True),
])
def test_largest_elements_are_noted_where_a_linear_reads_them(channels, structs, cutoff, zs, forward, backward):
    """The kernel on FP16 parts runs in both directions with 128 channels and many elements, forward only with 64 channels, backward only with two
    elements, and not with 32 channels (whose linears are too narrow); without it no row gather looks for largest elements."""
    model, _, _ = make_models(3, channels, zs, cutoff, 20.0, torch.float32, num_layers=3)  # (the second of three has all ranks and a skip connection)
    names = _launched(model, to_device(oracle_batch(structs(), zs, cutoff, torch.float32), torch.device("cuda:0")))
    middle = next(i for i, n in enumerate(names) if "tp_bwd" in n)  # (the readout and the last products lie before it in both directions)
    first = next(i for i, n in enumerate(names) if "readout_kernel" in n)
    assert first < middle
    assert any("tc_gemm_fp16_kernel" in n for n in names[:first]) == forward
    assert any("tc_gemm_fp16_kernel" in n for n in names[first:]) == backward
    assert any("gather_rows_top_kernel" in n for n in names[:first]) <= forward and any("gather_rows_top_kernel" in n for n in names[first:]) == backward


@pytest.mark.parametrize("channels,zs,tece,packed", [
    (64, [13, 29], None, 0),     # no linear takes FP16 parts
    (128, [13, 29], None, 19),   # those of the backward pass: 4 + 4 of linear_down; 4 + 1 of either order of the coefficients, which are folded; 1 skip connection
    (64, [13, 29], {"num_head": 4, "edge_ace_hidden": 64, "mmax": 1}, 22),  # the edge block: key, query, up, glu and down of two orders, the coefficients of one, both ways
])
def test_packed_copies_are_made_of_what_can_be_read(channels, zs, tece, packed):
    kw = dict(radial={"apply_cutoff": False}, tece=tece) if tece else {}
    model, _, _ = make_models(3, channels, zs, 4.0, 20.0, torch.float32, **kw)
    data = to_device(oracle_batch([synth.fcc_supercell(2, 3.65, 0.05, seed=5, species=(13, 29), fractions=(0.5, 0.5))], zs, 4.0, torch.float32), torch.device("cuda:0"))
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        model(data)  # the weights are set with the first evaluation
        torch.cuda.synchronize()
    assert sum("tc_pack_kernel" in e.name for e in prof.events()) == packed


def test_linear_down_over_chunks_of_edges():
    """The largest elements of the messages are noted chunk by chunk; the linear then reads them for all atoms."""
    structs = synth.random_crystals(5, seed=32, nmin=20, nmax=40, zmax=20)
    model, _, _ = make_models(3, 128, MANY, 4.5, 20.0, torch.float32)
    data = to_device(oracle_batch(structs, MANY, 4.5, torch.float32), torch.device("cuda:0"))
    count = lambda names: sum("tc_gemm_fp16_kernel" in n for n in names)
    launches = count(_launched(model, data))
    whole = {k: v.clone() for k, v in model(data).items() if v is not None}
    assert data["edge_index"].shape[1] > 3 * 1024
    model.set_chunk_edges(1024)
    assert count(_launched(model, data)) == launches > 4
    out = model(data)
    for k, v in whole.items():
        assert (out[k] - v).abs().max().item() <= 2e-5 * max(1.0, v.abs().max().item()), k
    assert model.device_error() == 0


def test_linear_down_with_the_targets_in_two_parts():
    """With the exchange on its own stream the forward contraction runs over the targets without a ghost neighbour first and over the others
    afterwards, and both parts note their rows: the energy is that of the serial exchange, bit for bit."""
    s = synth.fcc_supercell(4, 3.61, 0.05, seed=21, species=tuple(MANY), fractions=(0.05,) * 20)
    model, oracle, _ = make_models(3, 128, MANY, 4.0, 20.0, torch.float32, targets=("energy", "forces"))
    ref = oracle(oracle_batch([s], MANY, 4.0, torch.float32))
    model, energy = model.to(torch.device("cuda:0")), []
    for overlap in (False, True):
        model.set_exchange_overlap(overlap)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            md = DomainMD(model, s["cell"], s["positions"], s["atomic_numbers"], masses=np.ones(len(s["positions"])), skin=0.4, device=torch.device("cuda:0"))
            energy.append(md.potential())
        assert md.domain.n_ghost > 0 and any("tc_gemm_fp16_kernel" in e.name for e in prof.events())
        assert abs(energy[-1] - float(ref["energy"][0])) / len(s["positions"]) < 1e-5
        assert (torch.as_tensor(md.gather()["forces"]) - ref["forces"].detach().double().cpu()).abs().max().item() < 1e-4
    assert energy[0] == energy[1] and model.device_error() == 0
