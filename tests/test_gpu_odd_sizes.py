"""Greedy choice at sizes whose rows do not start on 16-byte boundaries, with ties and without a finite maximum."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    from popxl_addons_b200.ops import native

    return native


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
