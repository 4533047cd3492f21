"""Column sums of s8 weights (the zero-point term): exact, for whole and ragged column groups, few and many rows."""
import pytest
import torch

from gc_b200 import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("K,N", [(1, 16), (7, 1), (8, 130), (255, 128), (257, 144), (2056, 64), (4096, 1001), (300, 4112)])
@pytest.mark.parametrize("zp", [0, 3, 128])
def test_colsum_s8_exact(K, N, zp):
    g = torch.Generator().manual_seed(K * 7 + N)
    W = torch.randint(-128, 128, (K, N), generator=g, dtype=torch.int8)
    comp = lib.colsum_s8(W.to(DEV), zp)
    assert torch.equal(comp.cpu(), W.to(torch.int64).sum(0).mul(zp).to(torch.int32))


def test_colsum_s8_unaligned_base():
    W = torch.randint(-128, 128, (1 + 100 * 32,), dtype=torch.int8)
    Wd = W.to(DEV)[1:].view(100, 32)
    assert torch.equal(lib.colsum_s8(Wd, 5).cpu(), W[1:].view(100, 32).to(torch.int32).sum(0, dtype=torch.int32) * 5)
