"""The linears at the sizes where their tiles end: the double-precision kernel (32 x 32 tiles, K steps of 16) with species that own
one atom, one tile less a row, exactly one tile and one row more; the tensor-core kernel where the products of several
correlation orders share one accumulator loop, mixed with widths it does not take.  Against the oracle."""
import numpy as np
import pytest
import torch

from tace_b200 import synth
from test_gpu_parity import run_case

pytestmark = pytest.mark.gpu


def _cluster(counts, elements):
    """Atoms on a jittered grid (about 2.4 A apart), counts[i] of elements[i]."""
    z = np.repeat(elements, counts)
    rng = np.random.default_rng(int(sum(counts)))
    n = int(np.ceil(len(z) ** (1.0 / 3.0)))
    grid = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)[: len(z)] * 2.4
    return synth.Structure(positions=grid + rng.normal(0.0, 0.05, grid.shape), atomic_numbers=rng.permutation(z), cell=np.eye(3) * (2.4 * n),
                           pbc=(True, True, True))


@pytest.mark.parametrize("L,channels", [(1, 32), (2, 96), (3, 32)])
def test_double_precision_tiles(L, channels):
    run_case([_cluster((1, 31, 32, 33), (1, 6, 7, 8))], L, channels, [1, 6, 7, 8], 3.0, torch.float64)


@pytest.mark.parametrize("correlation", [1, 2, 3])
@pytest.mark.parametrize("channels", [64, 96, 128])
def test_products_of_several_orders_in_one_loop(channels, correlation):
    run_case([_cluster((1, 17, 43, 3), (1, 6, 7, 8))], 2, channels, [1, 6, 7, 8], 3.0, torch.float32, correlation=correlation)
