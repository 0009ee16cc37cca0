"""Launches that overlap: what a kernel has to hold before it lets its successor start."""
import glob
import os
import re

import pytest
import torch

import popxl_addons_b200
import popxl_addons_b200.xl.ops  # noqa: F401  (registers the ops)
from popxl_addons_b200.xl.opdef import OPS
from test_dunelix_ops import i32, rnd

CSRC = os.path.join(os.path.dirname(popxl_addons_b200.__file__), "csrc")


def kernels_with_tmem():
    """(file: kernel, body) of every kernel that allocates TMEM."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\b[^;{]*?(\w+)\(const __grid_constant__", text):
            at = end = text.index("{", m.end())
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            if re.search(r"\btmem_alloc\w*\(", text[at:end]):
                yield f"{os.path.basename(path)}: {m.group(1)}", text[at:end]


def test_a_kernel_holds_its_tmem_before_its_successor_starts():
    """A successor that allocates TMEM ahead of its own wait must not come first on an SM, so the launch of dependents stands behind the
    barrier that follows the allocation, in code that has passed this barrier."""
    found = dict(kernels_with_tmem())
    assert len(found) >= 7, sorted(found)
    for name, body in found.items():
        for m in re.finditer(r"xl_grid_launch_dependents\(\)", body):
            before = body[:m.start()]
            alloc = re.search(r"\btmem_alloc\w*\(", before)
            assert alloc, f"{name} starts its successor before it allocates TMEM"
            behind = before[alloc.end():]
            if "barrier.cluster.wait" in behind:  # the warps that pass the pair's second barrier at once: all but warp 0
                assert "else if (warp == 1)" in behind, f"{name}: warp 0 starts the successor ahead of the barrier"
            else:
                assert "__syncthreads()" in behind, f"{name} starts its successor while its allocation is under way"


def test_whole_warps_wait_together():
    """A bounded wait is a loop that lanes leave at different times, and warp-wide instructions follow it: a wait that is not a single
    thread's is one of `mbar_wait_warp` or stands in a vote. (Blocks are told by their indentation.)"""
    waits = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        lines = open(path).read().splitlines()
        for n, line in enumerate(lines):
            if not re.search(r"\bmbar_wait(_pair)?\(", line) or "__forceinline__" in line:
                continue
            waits += 1
            depth, around = len(line) - len(line.lstrip()), [line]
            for above in reversed(lines[:n]):
                indent = len(above) - len(above.lstrip())
                if above.strip() and indent < depth and not above.lstrip().startswith(("#", "//")):
                    depth = indent
                    around.append(above)
            single = any(re.search(r"elect_one\(\)|\blane (<|==)|threadIdx\.x ==", a) for a in around)
            assert single or any("__all_sync" in a for a in around[:2]), f"{os.path.basename(path)}:{n + 1}: {line.strip()}"
    assert waits > 20


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [2, 8])  # the few-rows products behind them allocate 32 columns on an SM with room for both
def test_portion_attention_ahead_of_few_rows_products(rows):
    """Heads of 48 and 64 features: both attentions, each followed by a product of few rows, replayed as a graph, give the bits of the same
    calls with the device idle in between."""
    from popxl_addons_b200.ops import native

    def op(name, *args, **kw):
        res = OPS[name].native["cuda"](*args, **kw)
        assert res is not NotImplemented
        return res

    gpu, B, H, G, dim, vdim, smax, N = ("cuda", torch.bfloat16), 1, 4, 2, 48, 64, 256, 256
    proj = rnd(gpu, B * rows, (H + G) * dim + G * vdim + H * vdim, seed=1)[0]
    qkv = rnd(gpu, B * rows, (H + G) * 2 * dim + G * vdim, seed=2)[0]
    w = rnd(gpu, N, H * vdim, std=0.1, seed=3)[0]
    one, none, lam = torch.ones(dim, device="cuda"), torch.zeros(1, device="cuda"), torch.tensor([0.8], device="cuda")
    pos, count = i32(gpu, 100), i32(gpu, rows)
    kc, vc = rnd(gpu, B, G, smax, dim, seed=4)[0], rnd(gpu, B, G, smax, vdim, seed=5)[0]
    kc2, vc2 = rnd(gpu, B, G, 2, smax, dim, seed=6)[0], rnd(gpu, B, G, smax, vdim, seed=7)[0]

    def chain(between):
        outs = []
        for _ in range(3):
            joint = torch.empty(B * rows, H * vdim, dtype=torch.bfloat16, device="cuda")
            op("window_attention_", proj, one, one, kc, vc, pos, count, joint, T=rows, heads=H, window=64, keep_first=1, scale=0.125,
               sink=-1.5, eps=1e-5)
            between()
            outs.append(op("linear_rows", joint, w, out_dtype=torch.float32))
            between()
            y = op("diff_attention_", qkv, none, none, kc2, vc2, pos, count, lam, T=rows, heads=H, rotary_dim=0, chunk=0, scale=0.125,
                   eps=1e-5, out_scale=0.4)
            between()
            outs.append(op("linear_rows", y, w, out_dtype=torch.float32))
            between()
        return outs

    want = chain(torch.cuda.synchronize)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(lambda: None)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    native.check_gemm_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,F", [(3, 41), (128, 256), (1000, 1024)])
def test_gated_units_wait_for_what_they_read(dtype, rows, F):
    """The gradient of a gated unit on what the launches before it wrote, and products of what it writes, as a graph: the bits of the same
    calls with the device idle in between."""
    from popxl_addons_b200.ops import native as nat

    gpu = ("cuda", dtype)
    gate, up, g = (rnd(gpu, rows, F, seed=s)[0] for s in (1, 2, 3))

    def chain(between):
        a, outs = gate, []
        for _ in range(4):
            y = nat.swish_cuda(a)
            between()
            da, du = nat.swiglu_grad_cuda(y, up, g)
            between()
            a = nat.gelu_cuda(da)
            between()
            outs += [da, du, a]
        return outs

    want = chain(torch.cuda.synchronize)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(lambda: None)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
