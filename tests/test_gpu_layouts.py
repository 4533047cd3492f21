"""Operand and output layouts the copy engine cannot address (row pitch or base no whole number of 16 bytes), and the
exact-order f32 kernel, at the edges of their tiles."""
import numpy as np
import pytest
import torch

import oracle
from _util import assert_bf16_close, tbits
from gc_b200 import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rand(shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.rand(shape, generator=g) * 2 - 1


def _at(t, skip):
    """The same values on the device, `skip` elements behind an aligned address."""
    buf = torch.zeros(t.numel() + skip, dtype=t.dtype, device=DEV)
    buf[skip:] = t.reshape(-1).to(DEV)
    return buf[skip:].view(t.shape)


@pytest.mark.parametrize("M,N,K,ta,tb,bias,relu,skip", [
    (200, 131, 77, 0, 0, 1, 1, 0),      # every pitch odd
    (130, 1001, 264, 0, 0, 1, 0, 0),    # odd outputs only: K-major activations are used as they are
    (129, 257, 192, 0, 1, 0, 1, 0),     # only the result has odd rows: one column past a tile
    (67, 190, 65, 1, 1, 1, 0, 0),       # both operands transposed
    (256, 192, 128, 0, 0, 1, 1, 1),     # even pitches, bases two bytes off
    (33, 300, 2049, 0, 0, 1, 1, 0),     # few rows: weights on the MMA M side, K split
    (96, 333, 4099, 0, 0, 1, 1, 0),     # K split, f32 planes with odd rows
    (1, 3, 1, 0, 0, 1, 0, 0),           # smallest
])
def test_bf16_layouts_without_alignment(M, N, K, ta, tb, bias, relu, skip):
    A, B, b = (_rand(s, i).bfloat16() for i, s in enumerate([(M, K), (K, N), (N,)]))
    Y = lib.matmul_bf16(_at(A.t().contiguous() if ta else A, skip), _at(B.t().contiguous() if tb else B, skip),
                        _at(b, skip) if bias else None, bool(relu), bool(ta), bool(tb), out=_at(torch.zeros(M, N).bfloat16(), skip))
    torch.cuda.synchronize()
    assert lib.device_error() == 0
    want, acc = oracle.linear_bf16(tbits(A), tbits(B), tbits(b) if bias else None, relu=bool(relu), return_acc=True)
    assert_bf16_close(tbits(Y), want, K, what=f"{M}x{N}x{K}", pre=acc if bias else None)


@pytest.mark.parametrize("bn", [32, 96, 160])
@pytest.mark.parametrize("M,N,K,tb", [(130, 131, 200, 0), (300, 193, 129, 1), (129, 320, 64, 0)])
def test_recorded_tile_widths_of_no_whole_slab(M, N, K, tb, bn):
    """Tiles whose last 64-column slab reaches beyond the accumulator, with results the copy engine cannot store (N odd) and
    with results it can."""
    A, B, b = (_rand(s, i).bfloat16() for i, s in enumerate([(M, K), (K, N), (N,)]))
    lib.tune_cache_put(M, N, K, lib.MatmulConfig(0, bn, 1, 4, 8, 148, 0, 1))
    try:
        Y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        lib.matmul_bf16(A.to(DEV), (B.t().contiguous() if tb else B).to(DEV), b.to(DEV), True, False, bool(tb), out=Y)
        torch.cuda.synchronize()
    finally:
        lib.tune_cache_erase(M, N, K)
    assert lib.device_error() == 0
    want, acc = oracle.linear_bf16(tbits(A), tbits(B), tbits(b), relu=True, return_acc=True)
    assert_bf16_close(tbits(Y), want, K, what=f"{M}x{N}x{K} tile {bn}", pre=acc)


@pytest.mark.parametrize("M,N,K,ta,tb", [(700, 1300, 40, 0, 0), (65, 66, 17, 1, 0), (40, 130, 33, 0, 1), (5, 768, 100, 0, 0), (17, 31, 16, 1, 1),
                                         (640, 1024, 16, 1, 1), (1, 1, 1, 0, 0)])
def test_f32_bits(M, N, K, ta, tb):
    """64 x 64, 32 x 32 and 16 x 16 tiles, whole and ragged, K slabs whole and cut: the oracle's bits."""
    A, B, b = (_rand(s, i).float().numpy() for i, s in enumerate([(M, K), (K, N), (N,)]))
    dev = lambda x, t: torch.from_numpy(np.ascontiguousarray(x.T if t else x)).to(DEV)
    Y = lib.matmul_f32(dev(A, ta), dev(B, tb), dev(b, 0), True, bool(ta), bool(tb))
    assert np.array_equal(Y.cpu().numpy(), oracle.matmul_f32(A, B, b, relu=True))
