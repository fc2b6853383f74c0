"""The attention softmax of the edge block works on a warp per atom, its lanes dealt to groups of edges and heads: head counts that divide
a warp and ones that do not, atoms with one edge, less than a group of edges and many.  Against the oracle."""
import pytest
import torch

from test_gpu_parity import run_case
from test_gpu_tp_wide import _ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [1, 3, 8, 12])
def test_head_counts(heads):
    run_case([_ring(n) for n in (1, 2, 9, 33)], 2, 96, [13, 29], 4.0, torch.float64, radial={"apply_cutoff": False},
             tece={"num_head": heads, "edge_ace_hidden": 8, "mmax": 2})
