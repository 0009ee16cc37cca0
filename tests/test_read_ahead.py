"""Kernels that may read an operand before their predecessor on the stream has ended read only what was complete before that
predecessor started: the order of the launches on the CPU, and on the GPU replayed programs whose weights and positions are
written by the launch before."""
import numpy as np
import pytest
import torch

from popxl_addons_b200 import xl
from popxl_addons_b200.xl import ops, read_ahead
from popxl_addons_b200.xl.opdef import OPS


def test_an_operand_is_complete_after_a_later_launch():
    order, w, x = read_ahead.LaunchOrder(), torch.zeros(4), torch.zeros(4)
    assert not order.complete(w)  # whatever was queued before may still write it
    order.launched(0)
    assert order.complete(w) and order.complete(w[2:])
    order.touch([w[:2]], None)  # a view's storage
    assert not order.complete(w) and not order.complete(w[2:]) and order.complete(x)
    order.launched(7)  # another stream's launch says nothing
    assert not order.complete(w)
    order.launched(0)
    assert order.complete(w)
    order.touch(w, [])
    for _ in range(200):  # many ops without a launch
        order.touch([torch.zeros(1)], [torch.zeros(2)])
    assert len(order._recent) < 70 and not order.complete(w) and order.complete(x)
    order.launched(0)
    assert order.complete(w)
    assert not read_ahead.allowed(w)  # nobody follows the order of this thread's launches
    with read_ahead.following(order):
        assert read_ahead.allowed(w, None, x)
        order.touch(x)
        assert not read_ahead.allowed(w, x)
        with read_ahead.following(None):
            assert not read_ahead.allowed(w)
        assert read_ahead.current() is order
    assert read_ahead.current() is None


@pytest.fixture
def asked(monkeypatch):
    """Stands in for the device kernels of two ops: counts their launches and records what `linear_rows` may read ahead."""
    answers = []

    def fake(name, weight_at=None):
        def run(*args, **kw):
            if weight_at is not None:
                answers.append(read_ahead.allowed(args[weight_at]))
            read_ahead.current().launched(0)
            return OPS[name].impl(*args, **kw)

        monkeypatch.setitem(OPS[name].native, "cpu", run)

    fake("gather")
    fake("linear_rows", 1)
    return answers


def _weights():
    w = xl.variable(np.eye(8, dtype=np.float32), xl.float32, "w")
    a = xl.variable(np.ones((3, 8), np.float32), xl.float32, "a")
    table = xl.variable(np.arange(80, dtype=np.float32).reshape(10, 8), xl.float32, "table")
    return w, a, table, xl.variable(np.array([1, 5, 7, 2, 0, 3, 9, 4], np.int32), xl.int32, "idx")


def test_which_weights_a_graph_lets_be_read_ahead(asked):
    ir = xl.Ir()
    with ir.main_graph:
        w, a, table, idx = _weights()
        g = ir.create_graph(lambda x, v: ops.linear_rows(x, v), a, w)
        ops.linear_rows(a, w)                                    # the first launch of a run
        ops.linear_rows(a, w)                                    # a weight that nobody writes
        ops.linear_rows(a, ops.gather(table, idx))               # written by the launch before
        late = ops.gather(table, idx)
        ops.linear_rows(a, w)
        ops.linear_rows(a, late)                                 # written two launches before
        ops.linear_rows(a, ops.linear_rows(w, w))                # the inner one, the outer one
        ops.add_(w, w)                                           # in place, by an op without a kernel of this library
        ops.linear_rows(a, w)
        ops.linear_rows(a, w)
        ops.call(g, a, ops.gather(table, idx))                   # as the input of a graph that is called
        ops.call(g, a, w)
        ops.linear_rows(w, ops.call(g, a, w)[0])                 # as its output
    session = xl.Session(ir, "cpu")
    session.use_native = True
    session.run()
    assert asked == [False, True, False, True, True, True, False, False, True, False, True, True, False]


def test_loops_and_programs(asked):
    ir = xl.Ir()
    with ir.main_graph:
        w, a, table, idx = _weights()

        def body(w_: xl.TensorByRef, a_: xl.Tensor):
            ops.linear_rows(a_, w_)
            ops.add_(w_, w_)  # the next iteration's weight

        graph = ir.create_graph(body, w, a)
        ops.gather(table, idx)
        ops.repeat(graph, 3, w, a)
    program, plain = xl.Program(ir, "p"), xl.Program(ir, "q")
    with program as p:
        ops.gather(p.use(table), p.use(idx))
        ops.linear_rows(p.use(a), p.use(w))
    with plain as q:
        ops.gather(q.use(table), q.use(idx))
    session = xl.Session(ir, "cpu")
    session.use_native = True
    session.run()
    assert asked == [True, False, False]
    session.run_program(program)
    assert asked[3:] == [True]
    assert session._launch_order(plain.graph) is None  # nothing in it asks


# ---- on the GPU ---------------------------------------------------------------------------------------------------------


def _replayed(build, variables, make_inputs, check, runs=150):
    """A captured program, replayed with new inputs each time; every result is compared. `build(use, streams)` records it."""
    ir = xl.Ir()
    with ir.main_graph:
        held = {name: xl.variable(*v, name) for name, v in variables.items()}
    program, streams = xl.Program(ir, "p"), {}
    with program as p:
        build(lambda name: p.use(held[name], by_ref=name in ("kc", "vc", "pos")), streams)
    session = xl.Session(ir, "cuda:0")
    g = torch.Generator().manual_seed(0)
    for _ in range(runs):
        inputs = make_inputs(g)
        out = session.run_program(program, {streams[k]: v for k, v in inputs.items()})
        check(inputs, torch.from_numpy(np.array(out[streams["y"]])), {k: session._vars[v][0] for k, v in held.items()})
    assert session._programs[program] is not None  # it was captured


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -14), (torch.float32, 2.0 ** -19)])
@pytest.mark.parametrize("rows", [1, 16, 40])
@pytest.mark.parametrize("inner", ["gather", "linear"])
def test_weights_written_by_the_launch_before(dtype, tol, rows, inner):
    """Scores against rows that a gather picked, and a product with the result of a product. The reference takes the weight as it
    was written (the inner product's rounding to bf16 included, which fp32 sums in another order flip for a few elements: one
    unit of 2^-8 of one of 512 terms), so results are fp32 sums of 512 terms."""
    dt, K, V, N = xl.float32 if dtype == torch.float32 else xl.bfloat16, 512, 4096, 1000
    n = N if inner == "gather" else 16 if rows <= 16 else 100
    gen = torch.Generator().manual_seed(rows)
    table = torch.randn(V, K, generator=gen).to(dtype)

    def build(use, streams):
        streams["a"] = xl.h2d_stream((rows, K), dt, "a")
        streams["y"] = xl.d2h_stream((rows, n), xl.float32, "y")
        a = ops.host_load(streams["a"])
        if inner == "gather":
            streams["by"] = xl.h2d_stream((n,), xl.int32, "by")
            w = ops.gather(use("table"), ops.host_load(streams["by"]))
        else:
            streams["by"] = xl.h2d_stream((n, K), dt, "by")
            w = ops.linear_rows(ops.host_load(streams["by"]), use("square"))
        ops.host_store(streams["y"], ops.linear_rows(a, w, xl.float32))

    def make(g):
        by = torch.randint(0, V, (n,), generator=g, dtype=torch.int32) if inner == "gather" else torch.randn(n, K, generator=g).to(dtype)
        return {"a": torch.randn(rows, K, generator=g).to(dtype), "by": by}

    def check(inputs, y, held):
        by = inputs["by"].cuda()
        w = held["table"][by.long()].double() if inner == "gather" else (by.double() @ held["square"].double().t()).to(dtype).double()
        want = (inputs["a"].cuda().double() @ w.t()).cpu()
        flips = 0 if inner == "gather" or dtype == torch.float32 else 2.0 ** -8
        assert float((y.double() - want).abs().max() / want.abs().max()) <= tol + flips

    square = (torch.randn(K, K, generator=gen) * K ** -0.5).to(dtype)
    _replayed(build, {"table": (table, dt), "square": (square, dt)}, make, check)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["diff", "window"])
def test_positions_written_by_the_launch_before(kind):
    """`advance_by_` directly before the attention of one token, which reads positions and the cache."""
    B, H, G, d, dv, S = 3, 8, 2, 64, 128, 1024
    gen = torch.Generator().manual_seed(1)
    maps = 2 if kind == "diff" else 1
    kc = torch.randn(B, G, *((2,) if kind == "diff" else ()), S, d, generator=gen).bfloat16()
    vc = torch.randn(B, G, S, dv, generator=gen).bfloat16()
    cols, ones, lam = (H + G) * maps * d + G * dv, torch.ones(d), torch.full((1,), 0.4)
    kw = dict(T=1, heads=H, scale=0.125)
    kw.update(dict(rotary_dim=0, out_scale=0.7) if kind == "diff" else dict(window=100, keep_first=4))

    def build(use, streams):
        for name in ("pos", "by"):
            streams[name] = xl.h2d_stream((B,), xl.int32, name)
        streams["qkv"] = xl.h2d_stream((B, cols), xl.bfloat16, "qkv")
        streams["y"] = xl.d2h_stream((B, H * dv), xl.float32, "y")
        qkv, by = ops.host_load(streams["qkv"]), ops.host_load(streams["by"])
        ops.var_updates.copy_var_update_(use("pos"), ops.host_load(streams["pos"]))
        ops.linear_rows(qkv, use("w"))  # any launch of this library, so that only `pos` is in doubt
        joint = () if kind == "diff" else (ops.cast(use("zeros"), xl.bfloat16),)
        ops.advance_by_(use("pos"), by)
        state = (use("kc"), use("vc"), use("pos"), use("count"))
        if kind == "diff":
            y = ops.diff_attention_(qkv, use("table"), use("table"), *state, use("lam"), **kw)
        else:
            y = ops.window_attention_(qkv, use("ones"), use("ones"), *state, *joint, **kw)
        ops.host_store(streams["y"], ops.cast(y, xl.float32))

    cache = [kc.clone(), vc.clone()]

    def make(g):
        half = lambda: torch.randint(0, S // 2, (B,), generator=g, dtype=torch.int32)
        return {"pos": half(), "by": half(), "qkv": torch.randn(B, cols, generator=g).bfloat16()}

    def check(inputs, y, held):
        pos, count = inputs["pos"] + inputs["by"], torch.ones(B, dtype=torch.int32)
        k, v = (c.float() for c in cache)
        q = inputs["qkv"].float()
        if kind == "diff":
            want = OPS["diff_attention_"].impl(q, ones[None], ones[None], k, v, pos, count, lam, chunk=0, eps=1e-6, **kw)
        else:
            want = OPS["window_attention_"].impl(q, ones, ones, k, v, pos, count, torch.zeros(B, H * dv), sink=None, eps=1e-6, **kw)
        cache[0], cache[1] = k.bfloat16(), v.bfloat16()
        assert torch.equal(held["pos"].cpu(), pos) and torch.equal(held["vc"].cpu(), cache[1])
        assert float((y - want).abs().max() / want.abs().max()) <= 1.2e-2  # 16-bit operands and probabilities

    variables = {"kc": (kc, xl.bfloat16), "vc": (vc, xl.bfloat16), "pos": (np.zeros(B, np.int32), xl.int32),
                 "count": (np.ones(B, np.int32), xl.int32), "lam": (lam, xl.float32), "ones": (ones, xl.float32),
                 "table": (torch.zeros(S, 1), xl.float32), "zeros": (torch.zeros(B, H * dv), xl.float32),
                 "w": (torch.randn(64, cols, generator=gen).bfloat16(), xl.bfloat16)}
    _replayed(build, variables, make, check)
