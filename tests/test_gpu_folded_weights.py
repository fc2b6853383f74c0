"""Weights that the library multiplies together when they are set (the product's final linear into the per-species coefficients, the first
linear_up into the species embedding): set in another order, and one at a time on a model that has been evaluated already, they give what a
model loaded with the same parameters gives, to the last bit; against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

from tace_b200 import lib as _lib
from tace_b200 import synth
from tace_b200.pack import RADIAL_TABLE_INTERVALS, pack_weights
from helpers import check_parity, make_models, oracle_batch, to_device

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _packed(model):
    rf = model.readout_fn
    spec = (model.get_cutoff(), int(rf.cfg["radial_basis"]["polynomial_cutoff"]), RADIAL_TABLE_INTERVALS) if model.uses_radial_table else None
    return pack_weights(rf.plan, rf.state_dict(), float(rf.cfg["avg_num_neighbors"]), radial_table_spec=spec)


def _set(model, packed, names, dtype):
    lib = _lib.load()
    for name in names:
        arr = np.ascontiguousarray(packed[name], dtype=np.float64 if dtype is torch.float64 else np.float32).reshape(-1)
        _lib.check(lib.tace_set_weight(model._handle, name.encode(), arr.ctypes.data_as(ctypes.c_void_p), arr.size), name)


def _names(model):
    lib, name, numel, out = _lib.load(), ctypes.c_char_p(), ctypes.c_int64(), []
    for i in range(lib.tace_weight_count(model._handle)):
        _lib.check(lib.tace_weight_info(model._handle, i, ctypes.byref(name), ctypes.byref(numel)), "tace_weight_info")
        out.append(name.value.decode())
    return out


@pytest.mark.parametrize("correlation,C,dtype,kind", [(1, 32, torch.float32, "aware"), (2, 64, torch.float32, "aware"), (3, 32, torch.float64, "agnostic"),
                                                      (2, 48, torch.float64, "identity"), (2, 128, torch.float32, "agnostic")])
def test_weights_set_again(correlation, C, dtype, kind):
    options = dict(correlation=correlation, resnet_linear_type=kind)
    structs = [synth.fcc_supercell(2, 3.65, 0.05, seed=3, species=(13, 29), fractions=(0.5, 0.5))]
    model, _, _ = make_models(2, C, [13, 29], 4.0, 12.0, dtype, seed=1, **options)
    other, oracle, _ = make_models(2, C, [13, 29], 4.0, 12.0, dtype, seed=5, **options)
    data = oracle_batch(structs, [13, 29], 4.0, dtype)
    gpu = to_device(data, DEV)
    before, want = model(gpu), other(gpu)
    before = {k: before[k].clone() for k in ("energy", "forces")}
    want = {k: want[k].clone() for k in ("energy", "forces")}
    check_parity(other(gpu), oracle(data), data["ptr"], dtype, f"correlation {correlation} {kind}")
    assert not torch.equal(before["energy"], want["energy"])

    names = _names(model)
    mine, theirs = _packed(model), _packed(other)
    for order in (names, names[::-1]):  # the derived forms before and after what they are derived from
        _set(model, theirs, order, dtype)
        out = model(gpu)
        assert torch.equal(out["energy"], want["energy"]) and torch.equal(out["forces"], want["forces"])
        _set(model, mine, order, dtype)
        out = model(gpu)
        assert torch.equal(out["energy"], before["energy"]) and torch.equal(out["forces"], before["forces"])

    # each factor by itself reaches the folded product, and back
    factors = ["emb", "t0.up.l0", "t0.up.b", "t0.lin.l0", "t0.lin.l2", "t0.lin.b", "t0.c.b", "t1.lin.l0", "t1.c.b", "t0.c0.l1", "t1.c0.l0"]
    factors += ["t1.res.b"] if kind != "identity" else []
    factors += [f"t0.c{j}.l2" for j in range(1, correlation)]
    for name in factors:
        _set(model, theirs, [name], dtype)
        assert not torch.equal(model(gpu)["energy"], before["energy"]), name
        _set(model, mine, [name], dtype)
        assert torch.equal(model(gpu)["energy"], before["energy"]), name


@pytest.mark.parametrize("dtype,tece", [(torch.float32, None), (torch.float64, None), (torch.float64, {"num_head": 4, "edge_ace_hidden": 8, "mmax": 2})])
def test_derived_coefficients_are_taken_from_what_they_derive_from(dtype, tece):
    """include/tace_b200.h: the content of the derived arrays is not read, of the right size they are accepted, of another refused; models
    with the edge block use them as they are set."""
    model, _, _ = make_models(2, 64, [13, 29], 4.0, 12.0, dtype, seed=1, tece=tece, radial={"apply_cutoff": False} if tece else None)
    gpu = to_device(oracle_batch([synth.fcc_supercell(2, 3.65, 0.05, seed=3, species=(13, 29), fractions=(0.5, 0.5))], [13, 29], 4.0, dtype), DEV)
    before = {k: v.clone() for k, v in model(gpu).items() if v is not None}
    derived = [n for n in _names(model) if n[3:4] == "c" and n[4:5] in "012" and (n[5] == "T" or n.endswith(("_hi", "_lo")))]
    assert len(derived) == 4 * 2 * (5 if dtype is torch.float32 else 1)  # two orders of three ranks and one of the scalar layer above
    packed = _packed(model)
    noise = {n: np.full(np.shape(packed[n]), 3.0) for n in derived}
    _set(model, noise, derived, dtype)
    out = model(gpu)
    for k, v in before.items():
        assert torch.equal(out[k], v) == (tece is None or k in ("energy", "node_energy")), k
    with pytest.raises(_lib.TaceError):
        _set(model, {derived[0]: np.zeros(7)}, derived[:1], dtype)
