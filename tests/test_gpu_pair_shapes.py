"""Shapes that the selector gives to CTA pairs: ragged in rows, columns and K, every operand layout.  A pair adds the same
products in the same order as one CTA per tile, so the results are compared bit for bit."""
import pytest
import torch

from gc_b200 import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K,ta,tb", [
    (2048, 2048, 1024, 0, 0),     # whole tiles, the shortest K
    (1960, 1832, 1184, 0, 1),     # a ragged last tile each way
    (1504, 5056, 1248, 1, 0),     # the odd CTA of the last pair has no row, half a B tile no column
    (3000, 5000, 1024, 1, 1),
    (4096, 1001, 1100, 0, 0),     # rows of no whole 16 bytes: packed operands, results stored row by row
])
@pytest.mark.parametrize("bias", [False, True])
def test_pairs_equal_one_cta_per_tile(M, N, K, ta, tb, bias):
    cfg = lib.model_matmul_config(M, N, K)
    assert cfg.pair == 1
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    A, B = (torch.randn(s, generator=g, device=DEV).bfloat16() for s in ((K, M) if ta else (M, K), (N, K) if tb else (K, N)))
    b = torch.randn(N, generator=g, device=DEV).bfloat16() if bias else None
    Y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    lib.matmul_bf16(A, B, b, relu=bias, transpose_a=bool(ta), transpose_b=bool(tb), out=Y)
    # One CTA per tile in row blocks that the selector gives to it.  Forced configurations take aligned operands only, so
    # those that are not are padded with zeros to whole 16 bytes, as the packing pass pads them.
    pad_n, pad_k = -N % 8, -K % 8
    Bp = torch.nn.functional.pad(B, (0, pad_k, 0, pad_n) if tb else (0, pad_n, 0, pad_k))
    bp = torch.nn.functional.pad(b, (0, pad_n)) if bias else None
    want = torch.empty_like(Y)
    for r in range(0, M, 896):
        rows = min(896, M - r)
        a = (A[:, r:r + rows] if ta else A[r:r + rows]).contiguous()
        a = torch.nn.functional.pad(a, (0, 0, 0, pad_k) if ta else (0, pad_k))
        one = lib.model_matmul_config(rows, N, K)
        one.swapped, one.bn, one.splits, one.stages, one.pair, one.kpb = 0, 256, 1, 4, 0, 1
        y = lib.matmul_bf16(a, Bp, bp, relu=bias, transpose_a=bool(ta), transpose_b=bool(tb), cfg=one)
        want[r:r + rows] = y[:, :N]
    torch.cuda.synchronize()
    assert lib.device_error() == 0
    assert torch.equal(Y, want)
