"""Partitions whose steps hand buffers on to each other inside one call: packed weights, deferred partial sums."""
import pytest
import torch

from gc_b200 import api, lib, partitions

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bf(g, *shape, k=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * k).bfloat16()


@pytest.mark.parametrize("batch,hidden", [
    (16, (512, 1001, 999, 1003)),        # every weight matrix packed
    (1, (72, 131, 129, 130)),            # the smallest copies: one ring of the few-rows kernel holds them whole
    (64, (1024, 2051, 1024, 515)),       # packed, as it is, packed
])
def test_packed_weights_of_a_chain_of_few_rows(batch, hidden):
    """Layers whose weight rows are no whole number of 16 bytes share one block for the packed copies, so every layer finds
    the copy of another one there.  Two sets of weights in turn through one executable: the bits of single calls each time."""
    n = len(hidden) - 1
    js, ids, out_id = partitions.mlp(batch, hidden, "bf16", [True] * n, "relu")
    exe = api.GraphCompiler().compile(js)
    sets, want = [], []
    for seed in (1, 2):
        g = torch.Generator(device=DEV).manual_seed(seed)
        ts = [_bf(g, batch, hidden[0])] + [_bf(g, hidden[i], hidden[i + 1], k=(2.0 / hidden[i]) ** 0.5) for i in range(n)]
        ts += [_bf(g, hidden[i + 1], k=0.1) for i in range(n)]
        h = ts[0]
        for i in range(n):
            h = lib.matmul_bf16(h, ts[1 + i], ts[1 + n + i], relu=True)
        sets.append(ts)
        want.append(h)
    torch.cuda.synchronize()
    for turn in range(12):
        out = torch.full((batch, hidden[-1]), float("nan"), dtype=torch.bfloat16, device=DEV)
        exe.execute_on_stream(dict(zip(ids, sets[turn & 1])), {out_id: out})
        torch.cuda.synchronize()
        assert lib.device_error() == 0
        assert torch.equal(out, want[turn & 1]), f"turn {turn}"
