"""The ops of the decoding path on the host: what a launch works out before it starts, and their references."""
import torch

import popxl_addons_b200.xl.ops  # noqa: F401  (registers the ops)
from popxl_addons_b200.xl.opdef import OPS


def test_the_split_of_a_cache_is_worked_out_once_per_shape():
    """Up to 64 candidates in Python (57 to 120 us for caches of 2000 and more positions), for every layer and token of an eager step."""
    from popxl_addons_b200.ops import native

    first = native._attn_decode_plan(48, 20000, 128, 148)
    before = native._attn_decode_plan.cache_info().hits
    assert native._attn_decode_plan(48, 20000, 128, 148) == first
    assert native._attn_decode_plan.cache_info().hits == before + 1


def test_a_launch_is_booked_under_its_own_name():
    """A fused launch is one kernel: nothing is booked under the names of those whose work it does."""
    import os
    import re

    from popxl_addons_b200.ops import native

    before = {k: dict(v) if isinstance(v, dict) else v for k, v in native.LAUNCHES.items()}
    native.count_replay(["one+two"])
    grown = {k for k, v in native.LAUNCHES["by_kernel"].items() if v != before["by_kernel"].get(k, 0)}
    assert native.LAUNCHES["count"] == before["count"] + 1 and grown == {"one+two"}
    native.LAUNCHES["count"] -= 1
    del native.LAUNCHES["by_kernel"]["one+two"]
    for name in ("native.py", "native_sequence.py"):
        assert not re.search(r'_count\([^)\n]*"\w+\+\w', open(os.path.join(os.path.dirname(native.__file__), name)).read())


def test_rows_outside_the_table_are_zeros():
    """In the reference as in the kernel: the norm of such a row is the norm's bias."""
    table, w, b = torch.randn(7, 10), torch.randn(10), torch.randn(10)
    x, h = OPS["gather_layer_norm"].impl(table, torch.tensor([3, 7, 0, -1], dtype=torch.int32), w, b, 1e-5)
    assert torch.equal(x[[0, 2]], table[[3, 0]]) and not x[1].any() and not x[3].any()
    torch.testing.assert_close(h[[1, 3]], b.expand(2, 10))
