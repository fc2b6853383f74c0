"""The tcgen05 GEMM on FP16 parts of scaled operands (through the C ABI) against products in double precision: both tile widths, K loops of one
step, an odd number of them and several drains, rows that fill tiles to 126 of 128, joined operands, added results, a matrix per group; and its
bounded waits.

Tolerance, relative and in the 2-norm: an operand in two FP16 parts is off by 2^-22 of itself at most (5e-7 for a product), and the tensor core
adds with truncation, 2.4e-8 for each of the up to 96 instructions between two drains: 1e-6 + 6e-6 * min(K, 512) / 512 is twice that
and more, while a product without one of the residuals is off by 1e-4."""
import pytest
import torch

from tace_b200 import lib as _lib
from tace_b200.pack import split_tf32

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def tolerance(K):
    return 1e-6 + 6e-6 * min(K, 512) / 512


def tops(A):
    """Bits of the largest |element| of every atom's rows; A [atoms][q][K]."""
    return A.abs().amax(dim=(1, 2)).view(torch.int32).contiguous()


class Call:
    """One launch: operands [(A [atoms][q][K], W [groups][N][K])], groups of atoms of the given sizes (None: one matrix for all)."""

    def __init__(self, operands, bias=None, sizes=None, C=None, top=tops):
        self.lib = _lib.load()
        atoms, self.q, _ = operands[0][0].shape
        self.N, self.keep, ops = operands[0][1].shape[1], [], []
        for A, W in operands:
            hi, lo = (torch.from_numpy(x) for x in split_tf32(W.numpy()))
            if sizes is not None:  # K-tile-major
                hi, lo = (x.reshape(len(sizes), self.N, -1, 32).permute(0, 2, 1, 3).contiguous() for x in (hi, lo))
            A = A.to(DEV)
            dev = [A, top(A), hi.to(DEV), lo.to(DEV), torch.empty(W.numel() + W.shape[0] * self.N, device=DEV)]
            self.keep += dev
            ops.append(_lib.TaceTcOperands(*(x.data_ptr() for x in dev), W.shape[2]))
        self.ops = (_lib.TaceTcOperands * len(ops))(*ops)
        self.atoms, self.bias, self.accumulate = atoms, None if bias is None else bias.to(DEV), int(C is not None)
        self.C = torch.full((atoms, self.q, self.N), float("nan"), device=DEV) if C is None else C.to(DEV)
        self.groups = self.tiles = None
        if sizes is not None:
            R = 128 // self.q
            count = lambda x: torch.tensor([0] + list(x), dtype=torch.int32).cumsum(0).to(torch.int32).to(DEV)
            self.groups, self.tiles = count(sizes), count((n + R - 1) // R for n in sizes)
        self.n_groups = 0 if sizes is None else len(sizes)
        self.err = torch.zeros(1, dtype=torch.int32, device=DEV)

    def __call__(self):
        ptr = lambda t: None if t is None else t.data_ptr()
        assert self.lib.tace_tc_gemm_fp16_f32(self.ops, len(self.ops), self.atoms, self.q, self.N, self.n_groups, ptr(self.groups), ptr(self.tiles),
                                              ptr(self.C), ptr(self.bias), self.accumulate, ptr(self.err), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return self.C.cpu()


def exact(operands, bias=None, sizes=None, C=None):
    atoms = operands[0][0].shape[0]
    group = torch.zeros(atoms, dtype=torch.long) if sizes is None else torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes))
    out = sum(torch.einsum("aqk,ank->aqn", A.double(), W.double()[group]) if sizes is not None else A.double() @ W[0].double().T for A, W in operands)
    if bias is not None:
        out = out + bias.double()[group][:, None, :]
    return out if C is None else out + C.double()


def error(got, want, dim=None):
    return ((got.double() - want).norm(dim=dim) / want.norm(dim=dim)).max().item()


def normal(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


@pytest.mark.parametrize("N", [64, 128, 192])
@pytest.mark.parametrize("atoms,q,K", [(1, 1, 32), (128, 1, 64), (129, 1, 96), (19, 7, 160), (40, 3, 544), (3000, 5, 512), (30, 1, 2944)])
def test_against_double_precision(N, atoms, q, K):
    operands = [(normal(atoms, q, K, seed=1), normal(1, N, K, seed=2))]
    bias = normal(1, N, seed=3)
    call = Call(operands, bias)
    got = call()
    assert int(call.err.item()) == 0
    assert error(got, exact(operands, bias)) < tolerance(K)


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("tiles,extra", [(1, -128), (1, 1), (2, 0), (5, 1), (6, 0), (6, 1), (7, 0), (13, 1)])
def test_tiles_of_a_block(N, tiles, extra):
    """Two warps describe every other tile of a block, six of them ahead: blocks with no tile, one to seven and thirteen, and blocks with one more
    than others."""
    sms = torch.cuda.get_device_properties(DEV).multi_processor_count
    rows = 128 * sms * tiles + extra
    A, W = normal(rows, 1, 32, seed=21), normal(1, N, 32, seed=22)
    call = Call([(A, W)])
    got = call()
    assert int(call.err.item()) == 0
    want = (A.to(DEV).double() @ W[0].to(DEV).double().T).cpu()
    for first in range(0, rows, 128 * sms):  # every row is looked at, and a wrong tile is not lost among the others
        part = slice(first, first + 128 * sms)
        assert error(got[part], want[part], dim=(1, 2)) < 2 * tolerance(32)


def test_the_kernel_is_the_one_on_fp16_parts():
    call = Call([(normal(300, 1, 128), normal(1, 128, 128, seed=1))])
    call()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
    assert sum("tc_gemm_fp16_kernel" in e.name for e in prof.events()) == 1


@pytest.mark.parametrize("N,q", [(128, 1), (64, 7)])
def test_joined_operands_added_to_the_result(N, q):
    """Weights of joined operands have scales of their own; segments of one, three and nine steps."""
    rows = normal(70, q, 32 * 13, seed=4)
    top = rows.abs().amax(dim=(1, 2)).view(torch.int32).to(DEV)
    operands = [(rows[..., :32].contiguous(), normal(1, N, 32, seed=5)), (rows[..., 32:128].contiguous(), 100 * normal(1, N, 96, seed=6)),
                (rows[..., 128:].contiguous(), .01 * normal(1, N, 288, seed=7))]
    before = normal(70, q, N, seed=8)
    call = Call(operands, C=before, top=lambda A: top)
    got = call()
    assert int(call.err.item()) == 0
    assert error(got, exact(operands, C=before)) < tolerance(416)


@pytest.mark.parametrize("N,q", [(128, 1), (64, 7), (128, 5)])
def test_a_matrix_per_group(N, q):
    """Groups without a row, with one, with exactly a tile and with several."""
    sizes = [0, 1, 128 // q, 3, 0, 2 * (128 // q) + 1, 5]
    operands = [(normal(sum(sizes), q, 96, seed=9), normal(len(sizes), N, 96, seed=10))]
    bias = normal(len(sizes), N, seed=11)
    call = Call(operands, bias, sizes)
    got = call()
    assert int(call.err.item()) == 0
    assert error(got, exact(operands, bias, sizes)) < tolerance(96)


def test_rows_of_every_magnitude():
    """Rows from 2^-60 to 2^60, and elements of a row over 2^-20 .. 1 of its largest: every row is as exact as the others."""
    A = normal(160, 1, 256, seed=12) * torch.exp2(torch.linspace(-60, 60, 160))[:, None, None] * torch.exp2(-20 * torch.rand(160, 1, 256, generator=torch.Generator().manual_seed(13)))
    operands = [(A, normal(1, 128, 256, seed=14))]
    call = Call(operands)
    got = call()
    assert int(call.err.item()) == 0
    assert error(got, exact(operands), dim=(1, 2)) < tolerance(256)


@pytest.mark.parametrize("N,K", [(128, 64), (128, 512), (64, 64), (64, 512)])
def test_every_instance_returns_from_an_expired_wait(N, K):
    """Load barriers that expect 16 bytes more than arrive: every role gives up after its shortened poll limit and the kernel returns; the
    same call without them is right afterwards.  More tiles than SMs, so every warp of every block has to leave as a whole."""
    operands = [(normal(128 * 400, 1, K, seed=15), normal(1, N, K, seed=16))]
    call = Call(operands)
    assert call.lib.tace_tc_gemm_set_test_mode(2048, 16) == 0
    try:
        call()
    finally:
        assert call.lib.tace_tc_gemm_set_test_mode(0, 0) == 0
    assert int(call.err.item()) in (1, 2, 3, 4, 5, 6)
    call.err.zero_()
    got = call()
    assert int(call.err.item()) == 0
    assert error(got[:512], exact([(operands[0][0][:512], operands[0][1])])) < tolerance(K)


@pytest.mark.parametrize("sizes", [None, [5, 200, 0, 140]])
def test_columns_of_every_magnitude(sizes):
    """Weights of results, and of groups, 2^-24 .. 1 apart: every column is as exact as the others."""
    n, K = 1 if sizes is None else len(sizes), 128
    W = normal(n, 128, K, seed=17) * torch.exp2(torch.linspace(-24, 0, n * 128).reshape(n, 128, 1))
    operands = [(normal(300 if sizes is None else sum(sizes), 1, K, seed=18), W)]
    call = Call(operands, sizes=sizes)
    got, want, first = call(), exact(operands, sizes=sizes), 0
    assert int(call.err.item()) == 0
    for size in sizes or [300]:
        if size:
            assert error(got[first:first + size], want[first:first + size], dim=(0, 1)) < tolerance(K)
        first += size


@pytest.mark.parametrize("N,q", [(128, 1), (64, 7)])
def test_joined_operands_of_every_magnitude(N, q):
    """Operands 2^-24 .. 2^24 apart whose weights bring their products to one magnitude."""
    operands = [(normal(70, q, K, seed=19) * 2. ** p, normal(1, N, K, seed=20) * 2. ** -p) for K, p in ((96, 24), (64, 0), (32, -24))]
    call = Call(operands)
    got = call()
    assert int(call.err.item()) == 0
    assert error(got, exact(operands)) < tolerance(192)
