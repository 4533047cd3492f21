"""Partitions whose steps hand buffers on to each other inside one call: packed weights, deferred partial sums, runs of
elementwise steps as one kernel."""
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


TYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


def _skip(t, n):
    """The same values `n` elements behind an aligned address."""
    buf = torch.empty(t.numel() + n, dtype=t.dtype, device=DEV)
    buf[n:] = t.reshape(-1)
    return buf[n:].view(t.shape)


@pytest.mark.parametrize("skip", [0, 1])   # 1: no operand on 16 bytes, so every step by itself
@pytest.mark.parametrize("rows,cols", [(1, 8), (37, 24), (300, 1032), (2, 4104)])
@pytest.mark.parametrize("dtype", list(TYPES))
def test_a_run_without_reductions_has_the_bits_of_its_steps(dtype, rows, cols, skip):
    """Whole, vector, row and one-element operands on either side of every operation: each step rounds once to its type, which
    is what torch does."""
    f = lambda i, dt=dtype: dict(_tensor(i, rows, cols), dtype=dt)
    vec, row, one = dict(_tensor(1, cols), dtype=dtype), dict(_tensor(2, rows, 1), dtype=dtype), dict(_tensor(3, 1), dtype=dtype)
    ops = [("Subtract", [f(0), vec], f(10)), ("Divide", [f(10), row], f(11)), ("Multiply", [one, f(11)], f(12)), ("Negate", [f(12)], f(13)),
           ("Subtract", [row, f(13)], f(14)), ("Divide", [vec, f(14)], f(15)), ("Add", [f(15), f(0)], f(16)), ("ReLU", [f(16)], f(17)),
           ("Typecast", [f(17)], f(18, "f32")), ("Multiply", [f(18, "f32"), f(18, "f32")], f(19, "f32"))]
    exe = api.GraphCompiler().compile(_partition(ops, [0, 1, 2, 3], [14, 19]))
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    x, v, r, o = ((torch.rand(s, generator=g, device=DEV) + at).to(TYPES[dtype])   # x >= v and all positive: nothing divides by zero
                  for s, at in (((rows, cols), 1.5), ((cols,), 0.5), ((rows, 1), 0.5), ((1,), 0.5)))
    t14 = r - (-(o * ((x - v) / r)))
    t18 = torch.relu(v / t14 + x).float()
    out14, out19 = _skip(torch.full_like(x, float("nan")), skip), _skip(torch.full_like(t18, float("nan")), skip)
    n = lib.launch_count()
    exe.execute_on_stream({0: _skip(x, skip), 1: _skip(v, skip), 2: _skip(r, skip), 3: _skip(o, skip)}, {14: out14, 19: out19})
    torch.cuda.synchronize()
    assert lib.launch_count() - n == (len(ops) if skip else 1)
    assert torch.equal(out14, t14) and torch.equal(out19, t18 * t18)


@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("rows,cols", [(1, 512), (65, 1000), (3, 4096), (5, 4104)])   # 4104: more than a run reduces
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_a_run_with_a_row_mean(dtype, rows, cols, skip):
    """x / mean(x).  The mean of positive values: each of the cols - 1 additions rounds by at most 2^-24 of a partial sum, in any
    order, and so do the two divisions; a bf16 mean and a bf16 result round by half an ulp each on top, 2^-8 of the value at
    most (8 bits: an ulp is 2^-7 of the power of two below)."""
    f = lambda i: dict(_tensor(i, rows, cols), dtype=dtype)
    mean = dict(_tensor(9, rows, 1), dtype=dtype)
    attrs = {"axes": {"type": "s64[]", "value": [-1]}, "keep_dims": {"type": "bool", "value": 1}}
    graph = [{"kind": "ReduceMean", "inputs": [f(0)], "outputs": [mean], "attrs": attrs}, {"kind": "Divide", "inputs": [f(0), mean], "outputs": [f(10)]}]
    exe = api.GraphCompiler().compile(json.dumps({"version": "3.5.0", "engine_kind": "cpu", "fpmath_mode": "any", "input_ports": [0], "output_ports": [10], "graph": graph}))
    g = torch.Generator(device=DEV).manual_seed(cols)
    x = (torch.rand(rows, cols, generator=g, device=DEV) + 0.5).to(TYPES[dtype])
    out = _skip(torch.full_like(x, float("nan")), skip)
    exe.execute_on_stream({0: _skip(x, skip)}, {10: out})
    torch.cuda.synchronize()
    want = x.double() / x.double().mean(1, keepdim=True)
    bound = (cols + 2) * 2.0 ** -24 + (2 * 2.0 ** -8 if dtype == "bf16" else 0)
    assert ((out.double() - want).abs() <= bound * want * (1 + bound)).all()


@pytest.mark.parametrize("skip", [0, 1])
def test_deferred_sums_where_the_run_cannot_start(skip):
    """A result of no 16 bytes sends the run back to its steps: the partial sums it was to add are added first."""
    g = torch.Generator(device=DEV).manual_seed(6)
    x, w, r, s = _bf(g, M, K), _bf(g, K, N, k=K ** -0.5), _bf(g, M, N), _bf(g, N)
    t = {i: _tensor(i, M, N) for i in (2, 10, 11, 12)}
    ops = [("MatMul", [_tensor(0, M, K), _tensor(1, K, N)], t[10]), ("Add", [t[10], t[2]], t[11]), ("Multiply", [t[11], _tensor(3, N)], t[12])]
    exe = api.GraphCompiler().compile(_partition(ops, [0, 1, 2, 3], [12]))
    want = (lib.matmul_bf16(x, w) + r) * s
    for _ in range(3):
        out = _skip(torch.full_like(want, float("nan")), skip)
        exe.execute_on_stream({0: x, 1: w, 2: r, 3: s}, {12: out})
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert lib.device_error() == 0


def test_calls_that_are_refused():
    g = torch.Generator(device=DEV).manual_seed(7)
    a, b, out = _bf(g, 64, 128), _bf(g, 128, 256), torch.empty(64, 256, dtype=torch.bfloat16, device=DEV)
    for bad in ((a.cpu(), b), (a.float(), b), (a, b.t()), (a.t(), b), (a, _bf(g, 136, 256)), (a[None], b)):
        with pytest.raises(AssertionError):
            lib.matmul_bf16(*bad, out=out)
    q = _bf(g, 2, 64, 128)
    for bad in ((q.cpu(), q, q), (q.float(), q, q), (q, q.transpose(0, 1), q), (q, q, q.transpose(0, 1))):
        with pytest.raises(AssertionError):
            lib.attention_bf16(*bad, 0.1, out=torch.empty_like(q))
