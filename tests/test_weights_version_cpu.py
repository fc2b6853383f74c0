"""The weights reach the device when the model is first evaluated and again when they change: every way of changing them has to
change ``_weights_version``, and nothing else may."""
import copy
import pickle

import pytest
import torch

from helpers import make_models

PART = "representation.interactions.0.linear_up"


def _parent(model):
    return model.readout_fn.get_submodule(PART.rpartition(".")[0])


def _write_in_place(model):
    with torch.no_grad():
        model.readout_fn.get_submodule(PART).weight.mul_(2.0)


def _replace_submodule(model):  # every version counter as before
    _parent(model).linear_up = copy.deepcopy(_parent(model).linear_up)


def _replace_parameter(model):
    part = model.readout_fn.get_submodule(PART)
    part.weight = torch.nn.Parameter(part.weight.detach().clone())


def _replace_a_one_element_buffer(model):  # of the same value: the next in-place write goes to the new one
    rb = model.readout_fn.get_submodule("representation.radial_basis.radial_fn")
    rb.prefactor = rb.prefactor.clone()


def _first_buffer_of_a_module(model):
    _parent(model).register_buffer("extra", torch.zeros(2))


def _remove_a_buffer(model):
    del model.readout_fn.scale_shift.shift


CHANGES = [_write_in_place, _replace_submodule, _replace_parameter, _replace_a_one_element_buffer, _first_buffer_of_a_module, _remove_a_buffer]


@pytest.mark.parametrize("change", CHANGES)
def test_every_change_of_the_weights_is_seen(change):
    model, _, _ = make_models(1, 32, [13, 29], 3.0, 12.0, torch.float32)
    first = model._weights_version()
    assert model._weights_version() == first
    change(model)
    second = model._weights_version()
    assert second != first and model._weights_version() == second
    _write_in_place(model)  # and what the change brought in is watched too
    assert model._weights_version() not in (first, second)


def test_a_copy_or_a_pickled_model_watches_its_own_weights():
    model, _, _ = make_models(1, 32, [13, 29], 3.0, 12.0, torch.float32)
    model._weights_version()
    for other in (copy.deepcopy(model), pickle.loads(pickle.dumps(model))):
        before = other._weights_version()
        _write_in_place(model)
        assert other._weights_version() == before
        _write_in_place(other)
        assert other._weights_version() != before
