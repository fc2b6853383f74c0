"""What ``build_batch`` refuses on the host, before anything reaches the device."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from tace_b200.graph import build_batch

ELEMENTS = [13, 29, 47]


@pytest.mark.parametrize("species,match", [
    ([0, 1, 2, 3], "indices in 0..2"),       # one past the list
    ([0, -1, 2, 1], "indices in 0..2"),      # negative
    ([0, 1, 2, 2 ** 32], "indices in 0..2"),  # would wrap to 0 in 32 bits
    ([1], "1 entries for 4 atoms"),          # would be broadcast
])
def test_species_outside_the_element_list_are_refused(species, match):
    batch = dict(synth.collate([synth.fcc_supercell(1, 3.61, 0.05, seed=0)]), species=np.array(species, dtype=np.int64))
    with pytest.raises(ValueError, match=match):
        build_batch(batch, ELEMENTS, 4.0, torch.float32, torch.device("cpu"))
