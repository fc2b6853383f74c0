"""Batch construction: structures -> the ``data`` dictionary ``TensorModel.forward`` consumes
(the role of ``from_atoms`` + PyG collation in the reference, ``tace/dataset/graph.py:36-161``,
``tace/interface/ase/calculator.py:132-152``), with the neighbour list built on the device."""

from __future__ import annotations

import functools
import math
from typing import Dict, Sequence

import numpy as np
import torch

from . import lib as _lib
from .neighbour_list import _list_at, complete_cell


@functools.lru_cache(maxsize=16)
def _element_table(model_numbers: tuple) -> np.ndarray:
    table = np.full(max(max(model_numbers), 118) + 1, -1, dtype=np.int64)
    for i, z in enumerate(sorted(model_numbers)):
        table[z] = i
    return table


def z_to_index(atomic_numbers: Sequence[int], model_numbers: Sequence[int]) -> np.ndarray:
    """tace/dataset/element.py:41-61 (TorchElement.z2idx): position of each Z in the sorted element list."""
    table = _element_table(tuple(map(int, model_numbers)))
    numbers = np.asarray(atomic_numbers, dtype=np.int64)
    if len(numbers) and numbers.max() < len(table):
        idx = table[numbers]
        if idx.min() >= 0:
            return idx
    elif len(numbers) == 0:
        return numbers
    raise ValueError("structure contains an element the model was not built for")


def _checked_species(species, n_atoms: int, n_elements: int) -> np.ndarray:
    """A caller's own element indices, one per atom and inside the model's list (on the device they index tables)."""
    species = np.asarray(species).reshape(-1)
    if len(species) != n_atoms:
        raise ValueError(f"species holds {len(species)} entries for {n_atoms} atoms")
    if n_atoms and not (0 <= species.min() and species.max() < n_elements):
        raise ValueError(f"species must hold indices in 0..{n_elements - 1} (the model's element list)")
    return species


def _structures_on_device(batch: Dict[str, np.ndarray], model_numbers: Sequence[int], cutoff: float, dtype: torch.dtype,
                          device: torch.device, returned):
    """Uploads the structures of ``batch`` and builds their neighbour list: the fields named in ``returned`` on the device, the
    addresses of all, edge list and shifts."""
    positions = np.asarray(batch["positions"])
    pbc_host = np.asarray(batch["pbc"], dtype=np.uint8)
    lattice_host = np.asarray(batch["lattice"], dtype=np.float64)
    ptr_host = np.asarray(batch["ptr"], dtype=np.int64)
    if pbc_host.all():
        cells = lattice_host  # fully periodic: the cell is used as given
    else:
        cells = np.stack([complete_cell(c, positions[a:b], p, cutoff)
                          for c, p, a, b in zip(lattice_host, pbc_host, ptr_host[:-1], ptr_host[1:])])
    n, b = len(positions), len(lattice_host)
    species_host = (_checked_species(batch["species"], n, len(model_numbers)) if "species" in batch
                    else z_to_index(np.asarray(batch["atomic_numbers"]), model_numbers))
    up, at = _upload(n, b, np.float64 if dtype == torch.float64 else np.float32,
                     (positions, cells, ptr_host, batch["batch"], positions, lattice_host, ptr_host, species_host, pbc_host), device, returned)
    return up, at, *_list_at(device, n, b, (at["pos64"], at["cells"], at["pbc"], at["ptr32"]), cutoff, -1, dtype)


def build_batch(batch: Dict[str, np.ndarray], model_numbers: Sequence[int], cutoff: float, dtype: torch.dtype,
                device: torch.device) -> Dict[str, torch.Tensor]:
    """``batch`` as returned by ``tace_b200.synth.collate``: host numpy arrays or (pinned) CPU
    tensors; an optional ``species`` entry (index into the model's element list) replaces the
    lookup from ``atomic_numbers``.  Uploads the structure, builds the neighbour list on ``device``
    and returns the model input dictionary."""
    up, at, edge_index, shifts = _structures_on_device(batch, model_numbers, cutoff, dtype, device, ("batch", "ptr", "positions", "lattice", "species"))
    n, n_el = len(up["positions"]), len(model_numbers)
    node_attrs = torch.empty(n, n_el, dtype=dtype, device=device)
    with _lib.on_device(device):
        _lib.check(_lib.load().tace_one_hot(at["species"], n, n_el, _lib.dtype_code(dtype), node_attrs.data_ptr(),
                                            _lib.stream_of(device)), "tace_one_hot")
    return {
        "positions": up["positions"],
        "lattice": up["lattice"],
        "node_attrs": node_attrs,
        "species": up["species"],
        "edge_index": edge_index,
        "edge_shifts": shifts,
        "batch": up["batch"],
        "ptr": up["ptr"],
    }


def model_inputs(batch: Dict[str, np.ndarray], model_numbers: Sequence[int], cutoff: float, dtype: torch.dtype,
                 device: torch.device) -> Dict[str, torch.Tensor]:
    """What ``TensorModel.forward`` reads of ``build_batch``'s dictionary, in the types that it uses, for callers who hand it to that
    function alone (``models.reads_inputs_only``) and keep nothing: no one-hot attributes beside the species, and structure offsets
    that need no conversion."""
    up, _, edge_index, shifts = _structures_on_device(batch, model_numbers, cutoff, dtype, device, ("ptr32", "positions", "lattice", "species"))
    return {"positions": up["positions"], "lattice": up["lattice"], "species": up["species"], "edge_index": edge_index, "edge_shifts": shifts,
            "ptr": up["ptr32"]}


_STAGED_BYTES = 1 << 20  # up to here the fields travel as one block; above, the copy into the block costs more than the transfers it saves


@functools.lru_cache(maxsize=64)
def _layout(n: int, b: int, real):
    """Places of the fields of ``n`` atoms in ``b`` structures in one block: (name, type, shape, offset) of each, and the size."""
    at, places = 0, []
    for name, kind, shape in (("pos64", np.float64, (n, 3)), ("cells", np.float64, (b, 3, 3)), ("ptr", np.int64, (b + 1,)),
                              ("batch", np.int64, (n,)), ("positions", real, (n, 3)), ("lattice", real, (b, 3, 3)),
                              ("ptr32", np.int32, (b + 1,)), ("species", np.int32, (n,)), ("pbc", np.uint8, (b, 3))):
        places.append((name, kind, shape, at))
        at += (math.prod(shape) * _BYTES[kind] + 15) & ~15
    return tuple(places), at


def _upload(n: int, b: int, real, values, device: torch.device, returned):
    """Host values (in the order of ``_layout``) on the device: tensors of the fields in ``returned`` and the addresses of all, by
    name.  A small batch is packed into one pinned block, every field at a multiple of 16 bytes and already in its final type: one
    transfer instead of one transfer and one conversion kernel per field.  The pinned block comes from torch's caching host
    allocator, which keeps it until the transfer has finished."""
    places, size = _layout(n, b, real)
    if size > _STAGED_BYTES:
        up = {name: torch.as_tensor(v).to(device, non_blocking=True).to(_TORCH[kind]).reshape(shape).contiguous()
              for (name, kind, shape, _), v in zip(places, values)}
        return up, {name: t.data_ptr() for name, t in up.items()}
    block = torch.empty(max(size, 16), dtype=torch.uint8, pin_memory=True)
    host = block.numpy()
    for (_, kind, shape, lo), v in zip(places, values):
        np.ndarray(shape, kind, host, lo)[...] = v
    dev = block.to(device, non_blocking=True)
    base, typed, up = dev.data_ptr(), {}, {}
    for name, kind, shape, lo in places:
        if name in returned:
            if kind not in typed:
                typed[kind] = dev.view(_TORCH[kind])
            up[name] = typed[kind].as_strided(shape, _STRIDES[len(shape)], lo // _BYTES[kind])
    return up, {name: base + lo for name, _, _, lo in places}


_TORCH = {np.float64: torch.float64, np.float32: torch.float32, np.int64: torch.int64, np.int32: torch.int32, np.uint8: torch.uint8}
_STRIDES = {1: (1,), 2: (3, 1), 3: (9, 3, 1)}  # [n], [n, 3] and [n, 3, 3] fields
_BYTES = {np.float64: 8, np.float32: 4, np.int64: 8, np.int32: 4, np.uint8: 1}
