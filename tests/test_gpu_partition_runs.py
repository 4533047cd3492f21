"""Partitions whose steps hand buffers on to each other inside one call: packed weights, deferred partial sums."""
import json

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


def _tensor(tid, *shape):
    return {"id": tid, "dtype": "bf16", "shape": list(shape)}


def _partition(ops, inputs, outputs):
    graph = [{"kind": kind, "inputs": ins, "outputs": [out]} for kind, ins, out in ops]
    return json.dumps({"version": "3.5.0", "engine_kind": "cpu", "fpmath_mode": "any", "input_ports": inputs, "output_ports": outputs, "graph": graph})


M, N, K = 128, 1024, 4096   # few tiles and a long K: the selector splits K, so a run may add the partial sums itself


@pytest.mark.parametrize("reader", ["matmul", "earlier run"])
def test_a_split_result_with_a_second_reader_is_written(reader):
    """y = x w1 with its K split; a run of elementwise steps adds y to z, and z (or what z is made of) needs y as well."""
    assert lib.select_matmul_config(M, N, K).splits > 1
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w1, w2, s = _bf(g, M, K), _bf(g, K, N, k=K ** -0.5), _bf(g, N, N, k=N ** -0.5), _bf(g, N)
    t = {i: _tensor(i, M, N) for i in range(10, 16)}
    ops = [("MatMul", [_tensor(0, M, K), _tensor(1, K, N)], t[10])]
    z_in = 10
    if reader == "earlier run":
        ops += [("Multiply", [t[10], _tensor(3, N)], t[11]), ("ReLU", [t[11]], t[12])]
        z_in = 12
    ops += [("MatMul", [t[z_in], _tensor(2, N, N)], t[13]), ("Add", [t[10], t[13]], t[14]), ("Multiply", [t[14], _tensor(3, N)], t[15])]
    exe = api.GraphCompiler().compile(_partition(ops, [0, 1, 2, 3], [15]))
    y = lib.matmul_bf16(x, w1)
    z = lib.matmul_bf16(torch.relu(y * s) if reader == "earlier run" else y, w2)
    want = (y + z) * s
    for _ in range(3):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        exe.execute_on_stream({0: x, 1: w1, 2: w2, 3: s}, {15: out})
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert lib.device_error() == 0


def _floats(tid, *shape):
    return dict(_tensor(tid, *shape), dtype="f32")


R, C = 70, 1024


def test_a_result_over_an_operand_that_every_row_reads():
    """relu(x + v) stored over memory that holds v: one step after the other, v has been read by then."""
    ops = [("Add", [_tensor(0, R, C), _tensor(1, C)], _tensor(2, R, C)), ("ReLU", [_tensor(2, R, C)], _tensor(3, R, C))]
    exe = api.GraphCompiler().compile(_partition(ops, [0, 1], [3]))
    g = torch.Generator(device=DEV).manual_seed(1)
    for row in (0, R // 2, R - 1):
        x, out = _bf(g, R, C), _bf(g, R, C)
        v = out[row]
        want = torch.relu(x + v)
        exe.execute_on_stream({0: x, 1: v}, {3: out})
        torch.cuda.synchronize()
        assert torch.equal(out, want)


def test_a_row_result_in_place_of_a_row_operand():
    """s = row + one value, stored in place of row, and x * s: no part of a row may see the new value as the old one."""
    ops = [("Add", [_floats(0, R, 1), _floats(1, 1)], _floats(2, R, 1)), ("Multiply", [_floats(3, R, C), _floats(2, R, 1)], _floats(4, R, C))]
    exe = api.GraphCompiler().compile(_partition(ops, [0, 1, 3], [2, 4]))
    g = torch.Generator(device=DEV).manual_seed(2)
    row, one, x = (torch.randn(*s, generator=g, device=DEV) for s in ((R, 1), (1,), (R, C)))
    s, out = row + one, torch.empty_like(x)
    exe.execute_on_stream({0: row, 1: one, 3: x}, {2: row, 4: out})
    torch.cuda.synchronize()
    assert torch.equal(row, s) and torch.equal(out, x * s)


def test_a_result_in_the_place_of_an_operand_of_its_shape():
    """out = (x + y) * v over x: element by element, so the run stays one kernel."""
    ops = [("Add", [_tensor(0, R, C), _tensor(1, R, C)], _tensor(2, R, C)), ("Multiply", [_tensor(2, R, C), _tensor(3, C)], _tensor(4, R, C))]
    exe = api.GraphCompiler().compile(_partition(ops, [0, 1, 3], [4]))
    g = torch.Generator(device=DEV).manual_seed(3)
    x, y, v = _bf(g, R, C), _bf(g, R, C), _bf(g, C)
    want, n = (x + y) * v, lib.launch_count()
    exe.execute_on_stream({0: x, 1: y, 3: v}, {4: x})
    torch.cuda.synchronize()
    assert torch.equal(x, want) and lib.launch_count() - n == 1
