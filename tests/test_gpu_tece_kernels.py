"""The edge-frame kernels of the TECE block at the shapes where their indexing can go wrong: every rank and order limit they are
instantiated for, one and several groups of 32 channels, heads that a warp can and cannot reduce, targets with fewer edges
than a block has warps, against the oracle in fp64 and fp32."""
import pytest
import torch

from tace_b200 import synth
from test_gpu_parity import run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,mmax,channels,heads", [
    (1, 0, 32, 4), (1, 1, 96, 3), (2, 0, 64, 1), (2, 1, 96, 4), (2, 2, 32, 16), (3, 0, 64, 2), (3, 1, 64, 1), (3, 2, 64, 8),
])
def test_edge_frame_kernels(L, mmax, channels, heads):
    structs = synth.random_crystals(2, seed=40 + L, nmin=2, nmax=9, zmax=3)
    for dtype in (torch.float64, torch.float32):
        run_case(structs, L, channels, [1, 2, 3], 4.0, dtype, radial={"apply_cutoff": False},
                 tece={"num_head": heads, "edge_ace_hidden": 8, "mmax": mmax})
