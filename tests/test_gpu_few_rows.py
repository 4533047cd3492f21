"""The few-rows matmul (M <= 64): K ranges shared by clusters of CTAs, and fused elementwise runs."""
import numpy as np
import pytest
import torch

import oracle
from _util import assert_bf16_close, tbits
from gc_b200 import api, lib, partitions

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K,ta,tb", [
    (1, 128, 64, 0, 0),        # one tile, one K block
    (1, 129, 72, 0, 1),        # a second tile of one column
    (16, 4096, 4096, 0, 1),    # 32 tiles over all SMs: K shared by clusters
    (17, 1000, 8192, 0, 0),    # few tiles, long K, ragged columns
    (64, 38912, 512, 0, 0),    # 149 tiles: several rounds with a split
    (33, 2048, 4160, 1, 0),    # transposed activations (M padded to the 16-byte rule by the caller: 40)
    (63, 384, 16384, 0, 1),
])
def test_few_rows_match_the_oracle_every_time(M, N, K, ta, tb):
    if ta:
        M = (M + 7) // 8 * 8
    g = torch.Generator().manual_seed(M + N)
    A, B, b = ((torch.rand(s, generator=g) * 2 - 1).bfloat16() for s in ((M, K), (K, N), (N,)))
    Ad, Bd = (A.t().contiguous() if ta else A).to(DEV), (B.t().contiguous() if tb else B).to(DEV)
    want, acc = oracle.linear_bf16(tbits(A), tbits(B), tbits(b), relu=True, return_acc=True)
    first = None
    for _ in range(4):   # partial sums are added in one order whatever the timing
        Y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        lib.matmul_bf16(Ad, Bd, b.to(DEV), True, bool(ta), bool(tb), out=Y)
        torch.cuda.synchronize()
        assert lib.device_error() == 0
        first = Y if first is None else first
        assert torch.equal(Y, first)
    assert_bf16_close(tbits(first), want, K, what=f"{M}x{N}x{K}", pre=acc)


@pytest.mark.parametrize("M,N,K", [(1, 256, 128), (40, 1040, 2048), (64, 4096, 4096)])
def test_few_rows_u8s8_bit_exact(M, N, K):
    g = torch.Generator().manual_seed(K)
    A = torch.randint(0, 256, (M, K), generator=g, dtype=torch.uint8)
    W = torch.randint(-127, 128, (K, N), generator=g, dtype=torch.int8)
    scale, bias = torch.rand(N, generator=g) * 0.009 + 0.001, torch.rand(N, generator=g) * 2 - 1
    comp = lib.colsum_s8(W.to(DEV), 7)
    out, acc = lib.matmul_u8s8(A.to(DEV), W.to(DEV), scale.to(DEV), bias.to(DEV), comp, want_acc=True)
    wacc, wout = oracle.linear_u8s8(A.numpy(), W.numpy(), scale.numpy(), bias.numpy(), zp_a=7)
    assert np.array_equal(acc.cpu().numpy(), wacc) and np.array_equal(out.cpu().numpy(), wout)


@pytest.mark.parametrize("B,S,H,I", [(1, 3, 512, 1024), (2, 33, 1024, 520), (1, 80, 4096, 1288), (1, 5, 4608, 1024)])
def test_decoder_block_with_fused_runs_against_single_steps(B, S, H, I):
    """The decoder block with elementwise runs fused against the same steps one by one (GC_B200_FUSE=0 in a process of
    its own).  Reductions are not alike (another order of the sum), and a bf16 rounding that falls the other way goes
    through the matmuls behind it, so the two agree in most elements and elsewhere to roundings of the largest ones: three,
    2^-8 each.  Element by element, and bit by bit without a reduction, fused runs are tested with the partition runs."""
    import os
    import subprocess
    import sys

    code = f"""
import sys, torch
sys.path[:0] = [{os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'graph-compiler_b200')!r}]
from gc_b200 import api, partitions
B, S, H, I = {B}, {S}, {H}, {I}
js, ids, outs = partitions.llama2_mlp(B, S, H, I)
g = torch.Generator().manual_seed(3)
bf = lambda *s, k=1.0: (torch.randn(*s, generator=g) * k).bfloat16().cuda()
t = dict(x=bf(B, S, H), wo=bf(H, H, k=H ** -0.5), resid=bf(B, S, H), g1=bf(H), w_gate=bf(I, H, k=H ** -0.5), w_up=bf(I, H, k=H ** -0.5),
         w_down=bf(H, I, k=I ** -0.5), g2=bf(H), eps=torch.full((1,), 1e-5, device="cuda"))
o = [torch.empty(B, S, H, dtype=torch.bfloat16, device="cuda") for _ in outs]
exe = api.GraphCompiler().compile(js)
for _ in range(3):
    exe.execute({{ids[k]: v for k, v in t.items()}}, dict(zip(outs, o)))
torch.save([x.cpu() for x in o], sys.argv[1])
"""
    import tempfile

    got = []
    for fuse in ("1", "0"):
        with tempfile.NamedTemporaryFile() as f:
            r = subprocess.run([sys.executable, "-c", code, f.name], env=dict(os.environ, GC_B200_FUSE=fuse), capture_output=True, text=True, timeout=300)
            assert r.returncode == 0, r.stderr[-2000:]
            got.append(torch.load(f.name))
    for a, b in zip(*got):
        assert (a.float() - b.float()).abs().max() <= 3 * 2.0 ** -8 * b.float().abs().max()
        assert float((a == b).float().mean()) > 0.9


@pytest.mark.parametrize("M,N,K,tb", [
    (5, 640, 200, 1),       # rows that end inside a stage's second K block
    (16, 300, 1096, 0),     # an odd number of K blocks, ragged columns
    (64, 256, 4096, 0),     # two tiles: the widest cluster, eight rows for every CTA
    (47, 512, 4224, 1),     # K blocks that no split divides evenly, rows that no split divides evenly
    (3, 1024, 1984, 0),     # fewer rows than CTAs in the cluster
])
def test_few_rows_stages_of_two_k_blocks(M, N, K, tb):
    test_few_rows_match_the_oracle_every_time(M, N, K, 0, tb)


@pytest.mark.parametrize("M,N,K", [(16, 512, 8192), (33, 1040, 1096), (64, 4096, 520), (1, 130, 136)])
def test_few_rows_as_recorded(M, N, K):
    """Every share of K, one and two K blocks to a stage and short rings, set by a recorded configuration."""
    g = torch.Generator().manual_seed(M + K)
    A, B, b = ((torch.rand(s, generator=g) * 2 - 1).bfloat16() for s in ((M, K), (K, N), (N,)))
    Ad, Bd, bd = A.to(DEV), B.to(DEV), b.to(DEV)
    want, acc = oracle.linear_bf16(tbits(A), tbits(B), tbits(b), relu=True, return_acc=True)
    try:
        for splits, kpb, stages in [(1, 1, 2), (2, 2, 3), (3, 1, 8), (5, 2, 2), (7, 1, 5), (8, 2, 8), (64, 4, 8)]:
            lib.tune_cache_put(M, N, K, lib.MatmulConfig(1, 64, splits, stages, 8, 148, 0, kpb))
            Y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
            lib.matmul_bf16(Ad, Bd, bd, True, out=Y)
            torch.cuda.synchronize()
            assert lib.device_error() == 0
            assert_bf16_close(tbits(Y), want, K, what=f"{M}x{N}x{K} clusters of {splits}, {kpb} blocks, {stages} stages", pre=acc)
    finally:
        lib.tune_cache_erase(M, N, K)


def test_tuning_few_rows_records_only_what_beats_the_own_rule():
    from gc_b200 import tune

    M, N, K = 16, 1024, 8192
    best, us, results = tune.tune_matmul(M, N, K, iters=3)
    assert len(results) > 4 and all(t > 0 for _, t in results)
    recorded = lib.tune_cache_get(M, N, K)
    lib.tune_cache_erase(M, N, K)
    assert (recorded is None) == (repr(best) == results[0][0])
