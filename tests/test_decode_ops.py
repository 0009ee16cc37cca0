"""The ops of the decoding path on the host: what a launch works out before it starts, and their references."""


def test_the_split_of_a_cache_is_worked_out_once_per_shape():
    """Up to 64 candidates in Python (57 to 120 us for caches of 2000 and more positions), for every layer and token of an eager step."""
    from popxl_addons_b200.ops import native

    first = native._attn_decode_plan(48, 20000, 128, 148)
    before = native._attn_decode_plan.cache_info().hits
    assert native._attn_decode_plan(48, 20000, 128, 148) == first
    assert native._attn_decode_plan.cache_info().hits == before + 1
