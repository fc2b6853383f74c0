"""Batch construction: structures -> the ``data`` dictionary ``TensorModel.forward`` consumes
(the role of ``from_atoms`` + PyG collation in the reference, ``tace/dataset/graph.py:36-161``,
``tace/interface/ase/calculator.py:132-152``), with the neighbour list built on the device."""

from __future__ import annotations

import math
from typing import Dict, Sequence

import numpy as np
import torch

from . import lib as _lib
from .neighbour_list import _list_on_device, complete_cell


def z_to_index(atomic_numbers: Sequence[int], model_numbers: Sequence[int]) -> np.ndarray:
    """tace/dataset/element.py:41-61 (TorchElement.z2idx): position of each Z in the sorted element list."""
    table = np.full(max(max(model_numbers), int(np.max(atomic_numbers))) + 1, -1, dtype=np.int64)
    for i, z in enumerate(sorted(model_numbers)):
        table[z] = i
    idx = table[np.asarray(atomic_numbers, dtype=np.int64)]
    if (idx < 0).any():
        raise ValueError("structure contains an element the model was not built for")
    return idx


def build_batch(batch: Dict[str, np.ndarray], model_numbers: Sequence[int], cutoff: float, dtype: torch.dtype,
                device: torch.device) -> Dict[str, torch.Tensor]:
    """``batch`` as returned by ``tace_b200.synth.collate``: host numpy arrays or (pinned) CPU
    tensors; an optional ``species`` entry (index into the model's element list) replaces the
    lookup from ``atomic_numbers``.  Uploads the structure, builds the neighbour list on ``device``
    and returns the model input dictionary."""
    n_el = len(model_numbers)
    positions = np.asarray(batch["positions"])
    pbc_host = np.asarray(batch["pbc"], dtype=np.uint8)
    lattice_host = np.asarray(batch["lattice"], dtype=np.float64)
    ptr_host = np.asarray(batch["ptr"], dtype=np.int64)
    if pbc_host.all():
        cells = lattice_host  # fully periodic: the cell is used as given
    else:
        cells = np.stack([complete_cell(c, positions[a:b], p, cutoff)
                          for c, p, a, b in zip(lattice_host, pbc_host, ptr_host[:-1], ptr_host[1:])])
    species_host = np.asarray(batch["species"]) if "species" in batch else z_to_index(np.asarray(batch["atomic_numbers"]), model_numbers)
    real = np.float64 if dtype == torch.float64 else np.float32
    n, b = len(positions), len(lattice_host)
    fields = [("pos64", positions, np.float64, (n, 3)), ("cells", cells, np.float64, (b, 3, 3)),
              ("ptr", ptr_host, np.int64, (b + 1,)), ("batch", np.asarray(batch["batch"]), np.int64, (n,)),
              ("positions", positions, real, (n, 3)), ("lattice", lattice_host, real, (b, 3, 3)),
              ("ptr32", ptr_host, np.int32, (b + 1,)), ("species", species_host, np.int32, (n,)), ("pbc", pbc_host, np.uint8, (b, 3))]
    up = _upload(fields, device)
    pos64 = up["pos64"]
    edge_index, shifts = _list_on_device(pos64, up["cells"], up["pbc"], up["ptr32"], cutoff, -1, dtype)
    node_attrs = torch.empty(n, n_el, dtype=dtype, device=device)
    with _lib.on_device(device):
        _lib.check(_lib.load().tace_one_hot(up["species"].data_ptr(), n, n_el, _lib.dtype_code(dtype), node_attrs.data_ptr(),
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


_STAGED_BYTES = 1 << 20  # up to here the fields travel as one block; above, the copy into the block costs more than the transfers it saves


def _upload(fields, device: torch.device) -> Dict[str, torch.Tensor]:
    """Host fields (name, values, type, shape) on the device.  A small batch is packed into one pinned block, every field at a
    multiple of 16 bytes and already in its final type: one transfer instead of one transfer and one conversion kernel per
    field (nine fields of a 32-atom cell: 150 us of host work before, 35 us now).  The pinned block comes from torch's caching
    host allocator, which keeps it until the transfer has finished."""
    at, places = 0, []
    for _, _, kind, shape in fields:
        size = math.prod(shape)
        places.append((at, at + size * _BYTES[kind]))
        at += (size * _BYTES[kind] + 15) & ~15
    if at > _STAGED_BYTES:
        return {name: torch.as_tensor(values).to(device, non_blocking=True).to(_TORCH[kind]).reshape(shape).contiguous()
                for name, values, kind, shape in fields}
    block = torch.empty(max(at, 16), dtype=torch.uint8, pin_memory=True)
    host = block.numpy()
    for (_, values, kind, shape), (lo, hi) in zip(fields, places):
        host[lo:hi].view(kind).reshape(shape)[...] = values
    dev = block.to(device, non_blocking=True)
    typed = {kind: dev.view(_TORCH[kind]) for kind in {f[2] for f in fields}}
    return {name: typed[kind].as_strided(shape, _STRIDES[len(shape)], lo // _BYTES[kind])
            for (name, _, kind, shape), (lo, _) in zip(fields, places)}


_TORCH = {np.float64: torch.float64, np.float32: torch.float32, np.int64: torch.int64, np.int32: torch.int32, np.uint8: torch.uint8}
_STRIDES = {1: (1,), 2: (3, 1), 3: (9, 3, 1)}  # [n], [n, 3] and [n, 3, 3] fields
_BYTES = {np.float64: 8, np.float32: 4, np.int64: 8, np.int32: 4, np.uint8: 1}
