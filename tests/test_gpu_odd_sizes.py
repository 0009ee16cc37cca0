"""Products, cross-entropy, column sums and greedy choice at sizes whose rows do not start on 16-byte boundaries, against the
plain operations in 64 bits. Bounds: operands are 16-bit and exact in the reference, sums are fp32, so what differs is the
rounding of the result (half a unit of its last place, 2^-9 for bf16 and 2^-12 for fp16) and fp32 summation: the tensor cores cut
the running sum to 24 bits at least every eight terms, at most one unit of 2^-23 each time."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}


@pytest.fixture(scope="module")
def nat():
    from popxl_addons_b200.ops import native

    return native


def _near(got, want, dtype, scale=None, terms=0):
    scale = want.abs().max() if scale is None else scale
    assert float((got.double() - want).abs().max() / scale) <= ROUND[dtype] + terms / 8 * 2.0 ** -23


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N", [(1, 8, 1), (3, 9, 7), (129, 65, 255), (256, 64, 257), (300, 257, 1021), (64, 1021, 129),
                                   (513, 40, 33), (100, 33, 300)])
def test_products(nat, M, K, N, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)

    def n(*s):
        return torch.randn(*s, device="cuda", generator=g).to(dtype)

    a, b, bias = n(M, K), n(K, N), n(N)
    at, bt = n(K, M), n(N, K)
    for x, y in ((a, b), (at.t(), b), (a, bt.t()), (at.t(), bt.t())):
        want = x.double() @ y.double()
        y1 = nat.gemm(x, y)
        assert y1.is_contiguous()
        _near(y1, want, dtype)
        _near(nat.gemm(x, y, out_dtype=torch.float32), want, torch.float32, scale=want.abs().max() + 1, terms=K)
    want = torch.relu(a.double() @ b.double() + bias.double())
    _near(nat.gemm(a, b, bias=bias, act=3), want, dtype, scale=want.max() + 1)
    step = torch.tensor(3.0, device="cuda")
    acc = torch.randn(M, N, device="cuda", generator=g)
    want = acc.double() * 0.75 + (a.double() @ b.double()) * 0.25
    assert nat.gemm(a, b, out=acc, accumulate=2, step=step) is acc
    _near(acc, want, torch.float32, scale=want.abs().max() + 1, terms=K)
    # an operand that starts in the middle of an allocation
    x = n(M * K + 3)[3:].view(M, K)
    _near(nat.gemm(x, b), x.double() @ b.double(), dtype)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,N", [(1, 131), (31, 160), (33, 257), (128, 129), (140, 600), (300, 1031)])
@pytest.mark.parametrize("gap", [0, 1, 8])
def test_every_way_a_product_leaves_the_pair_kernel(nat, out_dtype, M, N, gap):
    """Overwritten, added to and as a running mean, with bias and activation or without, into rows of `gap` more columns than are written
    (aligned and not), down to a single row of a tile; the columns between the rows stay as they are."""
    g = torch.Generator(device="cuda").manual_seed(M + N + gap)
    K, step = 72, torch.tensor(3.0, device="cuda")
    a, b, bias = ((torch.randn(*s, device="cuda", generator=g) * 0.3).bfloat16() for s in ((M, K), (K, N), (N,)))
    buf = torch.randn(M, N + gap, device="cuda", generator=g).to(out_dtype)
    plain = a.double() @ b.double()
    before = nat.LAUNCHES["by_kernel"].get("gemm2cta_tcgen05", 0)
    for want, kw in ((plain, {}), (torch.nn.functional.gelu(plain + bias.double()), dict(bias=bias, act=1)), (plain + bias.double(), dict(bias=bias))):
        for acc in (0, 1, 2):
            held, full = buf.double()[:, :N], buf.clone()
            out = full[:, :N]
            assert nat.gemm(a, b, out=out, accumulate=acc, step=step if acc == 2 else None, **kw) is out
            sums = {0: want, 1: held + want, 2: held * 0.75 + want * 0.25}[acc]
            _near(out, sums, out_dtype, scale=sums.abs().max() + 1, terms=K)
            assert torch.equal(full[:, N:], buf[:, N:])
    assert nat.LAUNCHES["by_kernel"]["gemm2cta_tcgen05"] == before + 9


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,V", [(1, 5), (3, 7), (2, 8), (65, 4099), (66, 1001), (70, 8193), (4, 50257)])
def test_cross_entropy_and_its_column_sums(nat, rows, V, dtype):
    """Element by element and relative to the element, with labels and large logits in the first piece of 16 bytes and in the
    ragged last one, so that what a row's ends get wrong shows."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(rows, V, device="cuda", generator=g) * 3).to(dtype)
    x[:, 2: V // 2: 3] = float("-inf")  # masked classes
    lab = torch.randint(V // 2, V, (rows,), device="cuda", generator=g, dtype=torch.int32)
    lab[::3], lab[1::3] = 0, V - 1
    x[::2, V - 1 - V % 3], x[1::2, 1] = 8, 9
    one = torch.ones((), device="cuda")
    loss, d = nat.ce_with_grad_cuda(x, lab, one, None, "none")
    xd = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(xd, lab.long(), reduction="none")
    want.sum().backward()
    torch.testing.assert_close(loss.double(), want.detach(), rtol=2 * ROUND[dtype], atol=1e-6)
    # 16 bits: a rounding of the result, the fast exponential's relative 2^-22 per unit of its argument (up to 30) is far below it; fp16
    # has steps of 2^-24 near 0. fp32: two units of the exponential, the rounded argument (up to 30), V / 512 additions per thread
    # and the sums over threads and warps, a division. At the label the result is p - 1. (fp32 rows of whole 16-byte pieces and single
    # rows: the fast exponential, 2 + 1.2 per unit of its argument.)
    rel = ROUND[dtype] if dtype != torch.float32 else ((64 if rows > 1 and V % 4 else 128) + V / 512) * 2.0 ** -24
    near0 = {torch.float16: 2.0 ** -24, torch.bfloat16: 0.0, torch.float32: 0.0}[dtype]
    hit = torch.zeros_like(xd.grad).scatter_(1, lab.long()[:, None], 1.0)
    off = (d.double() - xd.grad).abs()
    assert (off <= rel * torch.maximum(xd.grad.abs(), hit) + near0).all()
    assert d.shape == x.shape
    ldd = d.stride(0) if rows > 1 else V
    assert (torch.as_strided(d, (rows, ldd), (ldd, 1))[:, V:] == 0).all()  # the padding behind every row
    s = nat.sum_cuda(d, (0,), False)
    if rows >= 64:
        assert s is not NotImplemented and s.shape == (V,)
        _near(s, d.double().sum(0), dtype, scale=d.double().abs().sum(0).max())
    b = torch.randn(V, 40, device="cuda", generator=g).to(dtype)
    if dtype != torch.float32:
        want = d.double() @ b.double()
        _near(nat.matmul_cuda(d, b), want, dtype, scale=want.abs().max() + 1, terms=V)


@pytest.mark.parametrize("V", [7, 1001, 50257])
@pytest.mark.parametrize("shift", [0.0, 40.0])
def test_cross_entropy_of_fp32_logits_is_as_exact_as_softmax(nat, V, shift):
    """Rows of an odd number of classes: loss and gradient against 64 bits, no further away than from fp32 softmax with exact
    exponentials, for logits of a trained model's spread around 0 and far from 0."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(64, V, device="cuda", generator=g) * 5 + shift
    lab = torch.where(torch.arange(64, device="cuda") % 2 == 0, x.argmax(1), torch.randint(0, V, (64,), device="cuda", generator=g)).int()
    x[::2] += 10 * torch.nn.functional.one_hot(lab[::2].long(), V)  # losses close to 0
    loss, d = nat.ce_with_grad_cuda(x, lab, torch.ones((), device="cuda"), None, "none")
    logp = torch.log_softmax(x.double(), 1)
    hit = torch.nn.functional.one_hot(lab.long(), V)
    want, want_loss = logp.exp() - hit, -logp.gather(1, lab.long()[:, None])[:, 0]
    p32 = torch.softmax(x, 1)
    loss32 = -torch.log(p32.gather(1, lab.long()[:, None])[:, 0])
    away = lambda got: float(((got.double() - want).abs() / torch.maximum(want.abs(), hit)).square().mean().sqrt())
    assert away(d) <= 1.25 * away(p32 - hit)
    away = lambda got: float((got.double() - want_loss).square().mean().sqrt())
    assert away(loss) <= 1.25 * away(loss32)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [7, 1001, 1000])
@pytest.mark.parametrize("reduction", ["none", "mean"])
def test_cross_entropy_of_labels_outside_the_classes(nat, V, dtype, reduction):
    """Rows of an odd number of classes: the nearest class, as in the op's reference. Rows of whole 16-byte pieces: masked, though
    they count in the mean. Against 64 bits, one rounding of the result."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(6, V, device="cuda", generator=g).to(dtype)
    lab = torch.tensor([-3, V, V + 400, 2, -100, V - 1], dtype=torch.int32, device="cuda")
    loss, d = nat.ce_with_grad_cuda(x, lab, torch.ones((), device="cuda"), None, reduction)
    given = lab.clamp(0, V - 1).long()
    counts = (lab != -100) if V % 8 else (lab >= 0) & (lab < V)
    xd = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(xd, given, reduction="none") * counts
    if reduction == "mean":
        want = want.sum() / 5
    want.sum().backward()
    torch.testing.assert_close(loss.double(), want.detach(), rtol=2 * ROUND[dtype], atol=2e-6)
    torch.testing.assert_close(d.double(), xd.grad, rtol=2 * ROUND[dtype], atol=1e-6)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,V,valid", [(1, 1, 1), (1, 3, 2), (5, 33, 33), (16, 50400, 50257), (40, 32001, 32001), (700, 8190, 8189),
                                          (2, 70001, 70001)])
def test_greedy_choice(nat, rows, V, valid, dtype):
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randint(-40, 40, (rows, V), device="cuda", generator=g).to(dtype)  # many equal maxima: the first one wins
    x[0, : valid // 2] = float("nan")
    x[-1] = float("-inf")
    m, i = nat.argmax_rows_cuda(x, valid, 7)
    seen = x[:, :valid].float().cpu()
    seen = torch.where(seen.isnan(), torch.full_like(seen, float("-inf")), seen)
    want = torch.stack([(row == row.max()).nonzero()[0, 0] for row in seen])
    want[-1] = 0
    torch.testing.assert_close(m.cpu(), seen.max(1).values)
    assert torch.equal(i.cpu().long() - 7, want)


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1024, 2049, 4 * 256 * 2 * 3 + 5])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("moment", [torch.float32, torch.bfloat16])
def test_adam_writes_the_master_and_the_16_bit_weight(nat, n, offset, moment):
    """Groups of four, the elements behind the last one and buffers that are not aligned; master, weight and step count from one launch, twice,
    with the ticket back at zero. Each step against the op's torch reference on the same values: a few fp32 roundings apart (1e-6), one
    bf16 step for the 16-bit outputs."""
    from popxl_addons_b200.xl.opdef import OPS

    g = torch.Generator().manual_seed(n + offset)
    master, grad, m, v = (torch.randn(n + offset, generator=g).cuda()[offset:] for _ in range(4))
    w, m, v = torch.cat([master[:offset], master]).bfloat16()[offset:], m.to(moment), v.abs_()
    step, ticket = torch.tensor(2.0, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = dict(has_step=True, has_master=True, bias_correction=True, _tensor_scalars=(), lr=1e-2, beta1=0.9, beta2=0.95,
              epsilon=1e-5, weight_decay=0.01, grad_scale=0.5)
    for count in (3, 4):
        want = [t.cpu() for t in (w, grad, m, v, step, master)]
        OPS["adam_fused_"].impl(*want, **kw)
        rc = nat._adam(w.data_ptr(), nat._CODE[w.dtype], grad.data_ptr(), nat._CODE[grad.dtype], m.data_ptr(), nat._CODE[m.dtype],
                       v.data_ptr(), master.data_ptr(), step.data_ptr(), ticket.data_ptr(), 1e-2, 0.9, 0.95, 1e-5, 0.01, 0.5, 1, n,
                       nat._stream())
        assert rc == 0 and int(ticket) == 0 and float(step) == float(want[4]) == count
        for a, b, tol in zip((w, m, v, master), (want[0], want[2], want[3], want[5]),
                             (2 ** -8, 1e-6 if moment == torch.float32 else 2 ** -8, 1e-6, 1e-6)):
            a, b = a.float().cpu(), b.float()
            assert torch.allclose(a, b, rtol=tol, atol=tol), (a - b).abs().max()


@pytest.mark.parametrize("n", [1, 3, 5, 1023, 4099])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("acc_dtype,dtype", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_running_mean_in_groups_and_the_elements_behind(nat, n, offset, acc_dtype, dtype):
    """One launch for all of it, aligned or not, against 64 bits: three fp32 roundings of the result, and that to the accumulator's type."""
    g = torch.Generator().manual_seed(n)
    acc, x = torch.randn(n + 1, generator=g).to(acc_dtype)[offset:n + offset], torch.randn(n + 1, generator=g).to(dtype)[offset:n + offset]
    bufs = [torch.empty(n + 1, dtype=t.dtype, device="cuda")[offset:n + offset].copy_(t) for t in (acc, x)]
    step = torch.tensor(3.0, device="cuda")
    rc = nat._acc_mean(bufs[0].data_ptr(), nat._CODE[acc_dtype], bufs[1].data_ptr(), nat._CODE[dtype], step.data_ptr(), n, nat._stream())
    assert rc == 0
    want = acc.double() * 0.75 + x.double() * 0.25
    tol = 2.0 ** -22 if acc_dtype == torch.float32 else 2.0 ** -8
    assert ((bufs[0].double().cpu() - want).abs() <= tol * (acc.double().abs() + x.double().abs())).all()


@pytest.mark.parametrize("rows,cols,n", [(1, 4, 1), (5, 3, 9), (33, 130, 64), (100, 768, 257), (7, 8, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("t", [0.0, 3.0])
def test_embedding_gradient_into_the_running_mean(nat, rows, cols, n, dtype, t):
    """Rows of a table gradient added straight into the running mean, against 64 bits: indices repeat and some are out of
    range. fp32 sums of up to n terms: 1e-6 * n relative to the largest."""
    g = torch.Generator().manual_seed(rows * cols + n)
    acc = torch.randn(rows, cols, generator=g)
    grad = torch.randn(n, cols, generator=g).to(dtype)
    idx = torch.randint(-1, rows + 1, (n,), generator=g, dtype=torch.int32)
    ok = (idx >= 0) & (idx < rows)
    dense = torch.zeros(rows, cols, dtype=torch.float64).index_add_(0, idx[ok].long(), grad[ok].double())
    want = acc.double() * (t / (t + 1)) + dense / (t + 1)
    dev = acc.cuda()
    out = nat.gather_grad_accumulate_mean_cuda(dev, grad.cuda(), idx.cuda(), torch.tensor(t, device="cuda"), 0, True)
    assert out is dev
    assert (dev.cpu().double() - want).abs().max() <= 1e-6 * max(1, n)


@pytest.mark.parametrize("rows,cols,n", [(40, 256, 5000), (3000, 768, 4097), (3, 8196, 2048), (2, 2001, 33), (600, 4, 9000), (9, 132, 70),
                                         (5, 12, 32768 + 300), (1, 64, 1024), (1000, 1, 300)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_gradient_repeats_itself(nat, rows, cols, n, dtype):
    """Tokens with the frequencies of a text's words, so that rows get up to all of them: runs that one warp takes and runs that a CTA
    shares, more tokens than a pair of launches sorts, ragged and single columns. The same inputs give the same bits. Each of m <=
    n additions rounds a partial sum of about 4 sqrt(m) at most, with random signs."""
    g = torch.Generator().manual_seed(rows * cols + n)
    idx = (rows ** torch.rand(n, generator=g, dtype=torch.float64) - 1).int().clamp(0, rows - 1)
    acc, grad, step = torch.randn(rows, cols, generator=g), torch.randn(n, cols, generator=g).to(dtype), torch.tensor(2.0, device="cuda")
    dense = torch.zeros(rows, cols, dtype=torch.float64).index_add_(0, idx.long(), grad.double())
    got = []
    for _ in range(8):
        dev = acc.cuda()
        assert nat.gather_grad_accumulate_mean_cuda(dev, grad.cuda(), idx.cuda(), step, 0, False) is dev
        got.append(dev.cpu())
    assert all(torch.equal(got[0], y) for y in got[1:])
    assert (got[0].double() - (acc.double() * (2 / 3) + dense / 3)).abs().max() <= 2.0 ** -24 * (4 * n + 16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("M,N,K,gs", [(1, 1, 128, 32), (8, 63, 256, 64), (9, 130, 384, 96), (16, 257, 1024, 128), (3, 640, 2048, 64),
                                      (16, 2052, 2304, 64), (1, 14336, 2048, 64)])
def test_int4_product_at_the_edges_of_its_tiles(nat, dtype, pairs, M, N, K, gs):
    """Ragged channels, each block size, both token tiles, both layouts of the scales, tiles that CTAs share, against 64 bits.
    Sums of x times (base + code) are at most (128 + 15) / 4.6 of the result's size each, cut to 24 bits every eight terms."""
    from popxl_addons_b200.layers.linear_gq import interleave_scale_zero

    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    codes = torch.randint(0, 16, (N, K // gs, gs // 4, 4), generator=g, device="cuda")
    word = (codes[..., 0] << 12) | (codes[..., 1] << 8) | (codes[..., 2] << 4) | codes[..., 3]
    packed = torch.where(word > 32767, word - 65536, word).to(torch.int16).view(torch.uint16)
    scale = (0.02 + 0.02 * torch.rand(N, K // gs, 1, generator=g, device="cuda")).half()
    zero = (-0.3 + 0.1 * torch.rand(N, K // gs, 1, generator=g, device="cuda")).half()
    w = codes.reshape(N, K // gs, gs).double() * scale.double() + zero.double()
    want = x.double() @ w.reshape(N, K).t()
    y = nat.gq_gemm_small_m(x, packed, *((interleave_scale_zero(scale, zero), None) if pairs else (scale, zero)), None)
    assert y is not NotImplemented
    _near(y, want, dtype, terms=31 * K)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,gs", [(5, 130, 256, 32), (16, 700, 4096, 64), (6, 64, 128, 64)])
def test_int4_product_with_activations_that_are_not_finite(nat, dtype, M, N, K, gs):
    """Infinite, missing and (bf16) nearly infinite activations give what they give as products with the weights: the sums of x times
    the base of the codes, which overflow, do not show. Other rows keep their bits. Tiles of one CTA and tiles that CTAs share."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    codes = torch.randint(0, 16, (N, K // gs, gs // 4, 4), generator=g, device="cuda")
    word = (codes[..., 0] << 12) | (codes[..., 1] << 8) | (codes[..., 2] << 4) | codes[..., 3]
    packed = torch.where(word > 32767, word - 65536, word).to(torch.int16).view(torch.uint16)
    scale, zero = (torch.full((N, K // gs, 1), v, device="cuda").half() for v in (0.02, -0.13))  # no weight is 0
    scale[7], zero[7] = 0, 0                                                                     # but in one channel all are
    bias = torch.randn(N, generator=g, device="cuda").to(dtype)
    plain = nat.gq_gemm_small_m(x, packed, scale, zero, bias)
    big = 2.0 ** 125 if dtype == torch.bfloat16 else 60000.0
    x[0, 3], x[1, K - 1], x[2, 5], x[3, 9] = float("inf"), float("-inf"), float("nan"), big
    y = nat.gq_gemm_small_m(x, packed, scale, zero, bias)
    w = (codes.reshape(N, K // gs, gs).float() * scale.float() + zero.float()).to(dtype).double().reshape(N, K)
    want = x.double() @ w.t() + bias.double()
    torch.testing.assert_close(y[:4].double(), want[:4], rtol=2 * ROUND[dtype], atol=0.05 + 2.0 ** -8 * K ** 0.5, equal_nan=True)
    assert y[0].isinf().sum() == N - 1 and y[3].isfinite().all()
    assert torch.equal(y[4:], plain[4:])


@pytest.mark.parametrize("M,K,N", [(128, 64, 256), (256, 256, 768), (128, 192, 64), (4096, 64, 5000)])
def test_products_wait_for_what_they_read(nat, M, K, N):
    """Products start while their predecessor runs: a chain in which each reads what the launch before wrote (an element-wise kernel, another
    product, a running mean), replayed as a graph, against the same calls with the device idle in between. The last shape has
    320 tiles, more than a wave, in a ragged last group of rows and columns."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w, back = ((torch.randn(*s, generator=g, device="cuda") * 0.1).bfloat16() for s in ((K, N), (N, K)))
    step = torch.ones((), device="cuda")

    def chain(x, between):
        mean, held = torch.zeros(K, N, device="cuda"), []
        for _ in range(6):
            h = nat.gelu_cuda(x)
            between()
            y = nat.gemm(h, w)
            between()
            x = nat.gemm(y, back)
            between()
            nat.gemm(h.t(), y, out=mean, accumulate=2, step=step)
            between()
            held += [y, x]
        return held + [mean]

    want = chain(x, torch.cuda.synchronize)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(x, lambda: None)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    h = nat.gelu_cuda(x)
    _near(want[0], h.double() @ w.double(), torch.bfloat16, terms=K)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,gs", [(1, 4, 128, 64), (8, 128, 256, 128), (9, 132, 384, 128), (16, 1000, 1152, 64), (16, 260, 2048, 256),
                                      (3, 124, 1024, 512), (16, 640, 6144, 1024), (2, 20004, 512, 64), (13, 2048, 10240, 64)])
def test_int4_product_through_the_ring(nat, dtype, M, N, K, gs):
    """Scales as pairs: every group size the ring takes, half a chunk at the end of K, ragged channels, tiles of one CTA and of many, more
    chunks than the ring holds; against 64 bits, against the kernel that takes the same weights with their scales apart, the same bits
    twice, and a row that is not finite. Sums of x times (base + code) as above."""
    from popxl_addons_b200.layers.linear_gq import interleave_scale_zero

    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    codes = torch.randint(0, 16, (N, K // gs, gs // 4, 4), generator=g, device="cuda")
    word = (codes[..., 0] << 12) | (codes[..., 1] << 8) | (codes[..., 2] << 4) | codes[..., 3]
    packed = torch.where(word > 32767, word - 65536, word).to(torch.int16).view(torch.uint16)
    scale = (0.02 + 0.02 * torch.rand(N, K // gs, 1, generator=g, device="cuda")).half()
    zero = (-0.3 + 0.1 * torch.rand(N, K // gs, 1, generator=g, device="cuda")).half()
    pairs, bias = interleave_scale_zero(scale, zero), torch.randn(N, generator=g, device="cuda").to(dtype)
    w = codes.reshape(N, K // gs, gs).double() * scale.double() + zero.double()
    want = x.double() @ w.reshape(N, K).t() + bias.double()
    first = nat.gq_gemm_small_m(x, packed, pairs, None, bias)
    for ctas in (None, 3, 1):
        y = nat.gq_gemm_small_m(x, packed, pairs, None, bias, ctas=ctas)
        _near(y, want, dtype, terms=31 * K)
        assert ctas or torch.equal(y, first)
    _near(nat.gq_gemm_small_m(x, packed, scale, zero, bias), want, dtype, terms=31 * K)
    x[M // 2, K - 1] = float("inf")
    y = nat.gq_gemm_small_m(x, packed, pairs, None, bias)
    assert y[M // 2].isinf().all() or (w.reshape(N, K)[:, K - 1] == 0).any()
    assert torch.equal(y[M // 2 + 1:], first[M // 2 + 1:]) and torch.equal(y[:M // 2], first[:M // 2])
    nat.check_gemm_errors()


@pytest.mark.parametrize("M,N,K,gs", [(16, 50400, 2048, 64), (16, 28672, 4096, 64), (9, 28672, 4096, 128), (8, 50400, 2048, 64), (1, 14336, 2048, 64)])
def test_int4_product_of_weights_from_memory(nat, M, N, K, gs):
    """Codes and the kernel's own instructions come from memory, the scales have just been written: the same bits as with all of it in L2. (A
    stage that was refilled while a warp still read it gave every second such launch of 16 tokens other results.)"""
    g = torch.Generator(device="cuda").manual_seed(N + M)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    packed = torch.randint(0, 32768, (N, K // gs, gs // 4), generator=g, device="cuda").to(torch.int16).view(torch.uint16)
    pairs = (torch.randn(K // gs, N, 2, generator=g, device="cuda") * 0.05).half()
    nat.gq_gemm_small_m(x, packed, pairs, None, None)
    want = nat.gq_gemm_small_m(x, packed, pairs, None, None)
    for _ in range(20):
        torch.randn(20_000_000, device="cuda").double()  # 240 MB: more than L2 holds
        written = pairs * 1
        assert torch.equal(nat.gq_gemm_small_m(x, packed, written, None, None), want)
    nat.check_gemm_errors()


@pytest.mark.parametrize("rows,N,K", [(1, 1, 4), (2, 7, 132), (3, 2367, 1028), (4, 32000, 1024), (5, 30, 2816), (8, 2369, 68), (11, 513, 2048),
                                      (16, 1024, 1020)])
def test_few_rows_product_in_32_bits(nat, rows, N, K):
    """Ragged weight rows and K, each number of rows a CTA takes, a slice of a wider matrix. fp32 sums of K terms whose sizes add
    up to about sqrt(K) times the result: a few units of 2^-24 * sqrt(K)."""
    from popxl_addons_b200.ops.native_sequence import product

    g = torch.Generator(device="cuda").manual_seed(rows * N + K)
    a = torch.randn(rows, K + 4, generator=g, device="cuda")[:, :K]
    w = torch.randn(N, K, generator=g, device="cuda")
    before = nat.LAUNCHES["by_kernel"].get("linear_f32", 0)
    y = product(a, w)
    assert nat.LAUNCHES["by_kernel"]["linear_f32"] == before + 1
    want = a.double() @ w.double().t()
    assert float((y.double() - want).abs().max() / want.abs().max()) <= 2.0 ** -22 * K ** 0.5


@pytest.mark.parametrize("T", [1, 2, 70])
@pytest.mark.parametrize("dim,vdim", [(64, 128), (20, 36), (6, 300)])
@pytest.mark.parametrize("kind", ["diff", "window"])
def test_general_attention_of_few_rows_equals_that_of_many(nat, kind, T, dim, vdim):
    """A row's keys split over the warps of a CTA (few rows) against one warp per row (the same rows among many sequences): fp32 sums
    in another order, 1e-5. 70 tokens at position 150 see blocks that some warps do not have."""
    from popxl_addons_b200.ops import native_sequence as ns

    H, G, S, B = 4, 2, 260, 80
    g = torch.Generator(device="cuda").manual_seed(dim + T)
    one = lambda *s: torch.randn(*s, generator=g, device="cuda")
    many = lambda t: t.expand(B, *t.shape[1:]).contiguous()
    pos, s = torch.full((B,), 150, dtype=torch.int32, device="cuda"), nat._stream()
    count = torch.full((B,), T, dtype=torch.int32, device="cuda")
    lam = torch.tensor(0.3, device="cuda")
    vc = one(1, G, S, vdim)
    q, kc = (one(1, T, H * 2 * dim), one(1, G, 2, S, dim)) if kind == "diff" else (one(1, G, T, H // G, dim), one(1, G, S, dim))
    out = []
    for n in (1, B):
        y = torch.zeros(n * T, H * vdim, device="cuda")
        qn, kn, vn = (t if n == 1 else many(t) for t in (q, kc, vc))
        if kind == "diff":
            rc = ns._diff_general(qn.data_ptr(), H * 2 * dim, kn.data_ptr(), vn.data_ptr(), y.data_ptr(), H * vdim, pos.data_ptr(),
                                  count.data_ptr(), lam.data_ptr(), n, T, H, G, dim, vdim, S, 128, 0.2, 1e-5, 0.7, 0, s)
        else:
            rc = ns._window_general(qn.data_ptr(), kn.data_ptr(), vn.data_ptr(), None, 0, y.data_ptr(), H * vdim, pos.data_ptr(),
                                    count.data_ptr(), n, T, H, G, dim, vdim, S, 90, 3, 0.2, 0.0, 0, s)
        assert rc == 0
        out.append(y.view(n, T, H * vdim))
    assert out[1].abs().max() > 0
    assert (out[0] - out[1]).abs().max() <= 1e-5 * out[1].abs().max()


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,N,K", [(17, 128, 64), (32, 129, 72), (33, 2048, 7680), (64, 300, 4096), (65, 8200, 8), (128, 1000, 520),
                                      (40, 32000, 2048)])
def test_few_rows_product_at_the_edges_of_its_tiles(nat, out, rows, N, K):
    """Each token tile, ragged weight rows and K, tiles that many CTAs share; twice, since the sums are added in a fixed order. The
    activations are a slice of a wider matrix."""
    from popxl_addons_b200.ops.native_sequence import product

    g = torch.Generator(device="cuda").manual_seed(rows * N + K)
    a = torch.randn(rows, K + 8, generator=g, device="cuda").bfloat16()[:, :K]
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    want = a.double() @ w.double().t()
    before = nat.LAUNCHES["by_kernel"].get("linear_small_m", 0)
    first = product(a, w, out)
    y = product(a, w, out)
    assert nat.LAUNCHES["by_kernel"]["linear_small_m"] == before + 2
    assert y.dtype == out and torch.equal(first, y)
    _near(y, want, out, terms=K)
    nat.check_gemm_errors()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,S,H,D,smax", [(1, 1, 1, 8, 1), (2, 5, 3, 16, 9), (3, 67, 4, 256, 70), (2, 3, 2, 12, 4)])
def test_prompt_into_the_caches(nat, dtype, B, S, H, D, smax):
    """Every element moved, none besides; 12 bf16 features are refused (the plain copies take them)."""
    from popxl_addons_b200.xl.opdef import OPS

    qkv = torch.randn(B * S, 3 * H * D, generator=torch.Generator().manual_seed(D)).to(dtype)
    got = [torch.full((B, H, smax, D), 7.0, dtype=dtype, device="cuda") for _ in range(2)]
    want = [g.cpu().clone() for g in got]
    res = nat.kv_cache_fill_cuda(qkv.cuda(), *got, seq_len=S, n_heads=H, head_dim=D)
    assert (res is NotImplemented) == (D * dtype.itemsize % 16 != 0)
    if res is not NotImplemented:
        OPS["kv_cache_fill_"].impl(qkv, *want, seq_len=S, n_heads=H, head_dim=D)
        assert all(torch.equal(g.cpu(), w) for g, w in zip(got, want))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,H,S,D,R,packed", [(2, 3, 5, 16, 8, True), (1, 2, 67, 128, 128, True), (2, 2, 9, 20, 12, True),
                                              (2, 3, 7, 24, 6, False), (1, 4, 33, 64, 16, False)])
@pytest.mark.parametrize("inplace", [False, True])
def test_rotary_in_pieces_and_in_pairs(nat, dtype, B, H, S, D, R, packed, inplace):
    """Vectors of pairs (sizes and strides that allow them) and single pairs, per-batch tables, both directions, against 64 bits: one
    rounding of the result."""
    g = torch.Generator().manual_seed(D + S)
    if packed:  # the query part of packed (tokens, 3 * H * D) rows
        x = torch.randn(B * S, 3 * H * D, generator=g).to(dtype).cuda()[:, :H * D].view(B, S, H, D).permute(0, 2, 1, 3)
    else:
        x = torch.randn(B, H, S, D, generator=g).to(dtype).cuda()
    angle = torch.rand(B, S, R // 2, generator=g) * 6
    sin, cos = angle.sin().to(dtype).cuda(), angle.cos().to(dtype).cuda()
    for inverse in (False, True):
        want = x.double().clone()
        sn, cs = sin.double()[:, None] * (-1 if inverse else 1), cos.double()[:, None]
        a, b = want[..., 0:R:2].clone(), want[..., 1:R:2].clone()
        want[..., 0:R:2], want[..., 1:R:2] = a * cs - b * sn, b * cs + a * sn
        y = x if inplace else torch.empty_like(x)
        nat.rotary_launch(x, sin, cos, y, R, inverse)
        _near(y, want, dtype)
