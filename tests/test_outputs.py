"""Outputs of runs: C-contiguous whatever the layout of the tensor that was stored, and the caller's own however often the program runs
again; inputs reach the program that the caller passes, whether they are new, pinned or on the device."""
import numpy as np
import pytest
import torch

from popxl_addons_b200 import xl
from popxl_addons_b200.xl import ops

BACKENDS = ["cpu", pytest.param("cuda:0", marks=pytest.mark.gpu)]


def _program(dt=xl.float32):
    """y = 2 x and its transpose, z = x + a variable that counts the runs."""
    ir = xl.Ir()
    with ir.main_graph:
        count = xl.variable(np.zeros((), np.float32), xl.float32, "count")
    program = xl.Program(ir, "p")
    src, y, yt, z = xl.h2d_stream((3, 5), dt, "x"), *(xl.d2h_stream(s, d, n) for s, d, n in (((3, 5), dt, "y"), ((5, 3), dt, "yt"),
                                                                                       ((3, 5), xl.float32, "z")))
    with program as p:
        x, c = ops.host_load(src), p.use(count, by_ref=True)
        ops.add_(c, xl.constant(1.0, xl.float32))
        two = x + x
        ops.host_store(y, two)
        ops.host_store(yt, ops.transpose(two))
        ops.host_store(z, ops.cast(x, xl.float32) + c)
    return ir, program, src, (y, yt, z)


@pytest.mark.parametrize("device", BACKENDS)
@pytest.mark.parametrize("dt", [xl.float32, xl.float16])
def test_outputs_are_the_callers_own(device, dt):
    ir, program, src, streams = _program(dt)
    session = xl.Session(ir, device)
    g, kept = torch.Generator().manual_seed(0), []
    for k in range(9):  # the first run is eager, the second captured, then replays
        x = torch.randn(3, 5, generator=g).to(dt.as_torch())
        given = x
        if device != "cpu":
            given = (x, x.pin_memory(), x.cuda(), x.t().contiguous().pin_memory().t())[k % 4]
        fetch = k % 3 != 1
        out = session.run_program(program, {src: given}, fetch=fetch)
        kept.append((x, k + 1, fetch, [out[s] for s in streams]))
    if device != "cpu":
        assert session._programs[program] is not None
    for x, n, fetch, (y, yt, z) in kept:
        for got, want in ((y, x + x), (yt, (x + x).t()), (z, x.float() + n)):
            if fetch:
                assert got.flags.c_contiguous and got.shape == want.shape
                got = torch.from_numpy(np.array(got))
            else:
                assert got.is_contiguous()
                got = got.cpu().reshape(want.shape)
            assert torch.equal(got, want)


@pytest.mark.parametrize("device", BACKENDS)
def test_one_output_of_a_run_is_c_contiguous(device):
    ir = xl.Ir()
    with ir.main_graph:
        v = xl.variable(np.arange(12, dtype=np.float32).reshape(3, 4), xl.float32, "v")
        out = xl.d2h_stream((4, 3), xl.float32, "out")
        ops.host_store(out, ops.transpose(v))
    session = xl.Session(ir, device)
    got = session.run()[out]
    assert got.flags.c_contiguous and np.array_equal(got, np.arange(12, dtype=np.float32).reshape(3, 4).T)
    assert session.run(fetch=False)[out].is_contiguous()
