"""Scratch memory of the kernels: each stream's and each captured graph's own."""
import pytest
import torch

from popxl_addons_b200.ops import native as nat


@pytest.fixture
def on_cpu(monkeypatch):
    """The bookkeeping on the CPU backend, with a stream and a capture state that the test sets."""
    state = {"stream": 1, "capturing": False}
    monkeypatch.setattr(nat, "_stream", lambda: state["stream"])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    monkeypatch.setattr(nat, "_STREAM_SCRATCH", type(nat._STREAM_SCRATCH)())
    return state


def test_every_stream_has_its_own_and_the_number_is_bounded(on_cpu):
    dev = torch.device("cpu")
    a, w = nat.counters(10, dev, "counters x", 16), nat.workspace(4000, dev, "w")
    assert a.numel() == 16 and not a.any() and w.numel() >= 1000
    assert nat.counters(16, dev, "counters x", 16) is a and nat.workspace(8, dev, "w") is w
    on_cpu["stream"] = 2
    assert nat.counters(10, dev, "counters x", 16) is not a and nat.workspace(8, dev, "w") is not w
    for s in range(3, 100):
        on_cpu["stream"] = 1  # stays in use
        assert nat.counters(10, dev, "counters x", 16) is a
        on_cpu["stream"] = s
        nat.workspace(8, dev, "w")
    assert len(nat._STREAM_SCRATCH) == nat._MAX_STREAMS


def test_a_captured_graph_keeps_what_it_was_captured_with(on_cpu):
    dev = torch.device("cpu")
    a, w = nat.counters(10, dev, "counters x", 16), nat.workspace(8, dev, "w")
    with nat.capture_scratch(dev) as held:
        on_cpu["capturing"], on_cpu["stream"] = True, 9
        b = nat.counters(10, dev, "counters x", 16)
        assert b is not a and nat.counters(12, dev, "counters x", 16) is b and nat.workspace(8, dev, "w") is not w
        c = nat.counters(1000, dev, "counters x", 16)  # wider than before: what was captured so far keeps the old one
        assert c.numel() == 1000 and any(t is b for t in held.values()) and held["counters x"] is c
        with nat.capture_scratch(dev) as inner:
            assert nat.counters(10, dev, "counters x", 16) is not c and inner is not held
    d, e = nat.counters(10, dev, "counters x", 16), nat.counters(10, dev, "counters x", 16)
    assert d is not e  # a capture without a scope: none is kept
    on_cpu["capturing"], on_cpu["stream"] = False, 1
    assert nat.counters(10, dev, "counters x", 16) is a
    assert nat.counters(100, dev, "counters x", 16) is not a


# ---- on the GPU ---------------------------------------------------------------------------------------------------------


def _int4(N, K, M, seed, device="cuda"):
    g = torch.Generator(device=device).manual_seed(seed)
    packed = torch.randint(-32768, 32768, (N, K // 64, 16), generator=g, device=device, dtype=torch.int16).view(torch.uint16)
    scale, zero = (torch.rand(N, K // 64, 1, generator=g, device=device).half() for _ in range(2))
    return torch.randn(M, K, generator=g, device=device).bfloat16(), packed, scale, zero


@pytest.mark.gpu
def test_a_wider_weight_leaves_captured_products_alone():
    """A captured product whose tiles CTAs share, a product of more than 131072 channels that needs more counters, memory of the
    counters' size filled with other values, and the captured one again."""
    import numpy as np

    from popxl_addons_b200 import xl
    from popxl_addons_b200.xl import ops
    from popxl_addons_b200.xl.opdef import emit1
    import popxl_addons_b200.layers.linear_gq  # noqa: F401  (registers the op)

    x, packed, scale, zero = _int4(640, 4096, 3, 0)
    ir = xl.Ir()
    with ir.main_graph:
        held = [xl.variable(t.cpu().view(torch.uint8).numpy().view(np.uint16) if t.dtype == torch.uint16 else t.cpu(), dt, n)
                for t, dt, n in ((packed, xl.uint16, "packed"), (scale, xl.float16, "scale"), (zero, xl.float16, "zero"))]
    program = xl.Program(ir, "p")
    with program as p:
        src, dst = xl.h2d_stream((3, 4096), xl.bfloat16, "x"), xl.d2h_stream((3, 640), xl.float32, "y")
        y = emit1("linear_gq", [ops.host_load(src), *(p.use(v) for v in held)], {"dim": 0})
        ops.host_store(dst, ops.cast(y, xl.float32))
    session = xl.Session(ir, "cuda:0")
    first = [session.run_program(program, {src: x.cpu()})[dst] for _ in range(3)]
    wide = _int4(131072 + 640, 128, 2, 1)
    want = nat.gq_gemm_small_m(*wide, None)
    junk = [torch.full((n,), 3, dtype=torch.int32, device="cuda") for n in (2048, 4096, 8192) for _ in range(20)]
    for _ in range(3):
        assert np.array_equal(session.run_program(program, {src: x.cpu()})[dst], first[0])
    assert all(np.array_equal(f, first[0]) for f in first)
    assert torch.equal(nat.gq_gemm_small_m(*wide, None), want) and all((j == 3).all() for j in junk)


@pytest.mark.gpu
def test_products_and_attention_on_two_streams():
    """int4 products whose tiles CTAs share and decode attention split over the cache, interleaved on two streams."""
    ops_ = []
    for seed, (N, K) in enumerate(((640, 8192), (2048, 4096))):
        args = _int4(N, K, 2, seed)
        ops_.append(lambda args=args: nat.gq_gemm_small_m(*args, None))
    H, D, S = 4, 128, 2000
    for seed in range(2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
        qkv, kc, vc, pos = n(2, 3 * H * D), n(2, H, S, D), n(2, H, S, D), torch.full((1,), S - 1, dtype=torch.int32, device="cuda")
        ops_.append(lambda a=(qkv, kc, vc, pos): nat.attention_decode_packed_cuda(*a, H, D, D ** -0.5))
    want = [f() for f in ops_]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in range(2)], []
    for i in range(200):
        with torch.cuda.stream(streams[i % 2]):
            got.append([f() for f in (ops_ if i % 3 else ops_[::-1])][:: 1 if i % 3 else -1])
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for row in got for a, b in zip(row, want))
