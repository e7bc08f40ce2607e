"""The launch rules that are functions of sizes only (no GPU needed: the kernel library's host
side answers them): how many K splits a product uses, and how many keys a decode-attention
segment holds. They decide reduction orders, so what they depend on is part of the contract."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    try:
        from vosti_b200 import ops
        library = ops.library()
    except Exception as error:                       # no nvcc on this machine
        pytest.skip(f"the kernel library cannot be built here: {error}")
    library.vosti_attention_decode_scratch.restype = ctypes.c_int64
    return library


def test_split_count_depends_on_the_weight_only_up_to_64_tokens(lib):
    for features, k in [(4096, 4096), (6144, 4096), (4096, 12288), (24576, 4096), (151936, 4096), (1000, 1000),
                        (5120, 17408)]:
        counts = {lib.vosti_gemm_tc_splits(t, features, k) for t in (1, 2, 7, 8, 31, 32, 33, 64)}
        assert len(counts) == 1, (features, k, counts)       # a decode batch's size does not change the sum order
        splits = counts.pop()
        tiles, k_blocks = -(-features // 128), -(-k // 64)
        assert 1 <= splits <= 16 and splits * tiles <= max(296, tiles)      # never a second round of CTAs
        assert splits == 1 or k_blocks // splits >= 4
        assert lib.vosti_gemm_tc_splits(129, features, k) == 1 and lib.vosti_gemm_tc_splits(4096, features, k) == 1


def test_decode_segment_length(lib):
    nq, nkv, d = 32, 8, 128
    for count in (1, 2, 8, 31, 64, 256, 1000):
        for longest in (1, 17, 128, 129, 2048, 2560, 4096, 4097, 20000, 131072):
            keys = lib.vosti_attention_decode_segment_keys(count, nq, nkv, d, longest)
            assert 128 <= keys <= 4096 and keys % 64 == 0
            segments = -(-longest // keys)
            assert lib.vosti_attention_decode_scratch(count, nq, nkv, d, longest) >= count * nq * segments * (d + 4)
    # many tokens: one segment per request as long as it fits; few tokens: cut finely
    assert lib.vosti_attention_decode_segment_keys(64, nq, nkv, d, 2560) == 2560
    # one CTA per (token, kv head, segment): the segment count that makes waves x (keys + 350) smallest.
    # While all CTAs fit the GPU at once (296 of them at these sizes) that is as many segments as fit,
    # at most 16 for up to 8 (token, kv head) pairs and 8 beyond, of equal length, a multiple of 64
    assert lib.vosti_attention_decode_segment_keys(1, nq, nkv, d, 2560) == 192        # 8 pairs x 14 segments
    assert lib.vosti_attention_decode_segment_keys(8, nq, nkv, d, 2560) == 640        # 64 pairs x 4
    assert lib.vosti_attention_decode_segment_keys(4, nq, nkv, d, 2560) == 320        # 32 pairs x 8
    assert lib.vosti_attention_decode_segment_keys(16, nq, nkv, d, 2560) == 1280      # 128 pairs x 2
    # in waves: 384 pairs are 2 waves of 2560 keys or 3 of 1280; 512 pairs are 2 waves of 2560 or 4 of 1280
    assert lib.vosti_attention_decode_segment_keys(48, nq, nkv, d, 2560) == 1280
    assert lib.vosti_attention_decode_segment_keys(64, nq, nkv, d, 2560) == 2560
    assert lib.vosti_attention_decode_segment_keys(256, nq, nkv, d, 2560) == 2560
    # too long for 8 segments of 4096 keys: the persistent kernel's cost model
    assert lib.vosti_attention_decode_segment_keys(8, nq, nkv, d, 40000) > 4096 // 2
    assert lib.vosti_set_decode_once(0) == 0
    try:
        # the persistent kernel's cost model alone
        assert lib.vosti_attention_decode_segment_keys(1, nq, nkv, d, 2560) == 128
        assert lib.vosti_attention_decode_segment_keys(64, nq, nkv, d, 2560) == 2560
        for count in (1, 8, 64):
            keys = lib.vosti_attention_decode_segment_keys(count, nq, nkv, d, 2560)
            assert lib.vosti_attention_decode_scratch(count, nq, nkv, d, 2560) == count * nq * -(-2560 // keys) * (d + 4)
    finally:
        assert lib.vosti_set_decode_once(1) == 0
    # a pinned length overrides the cost model for every shape of launch, and taking the pin
    # away gives the launches their own choice back
    shapes = [(c, n) for c in (1, 8, 64) for n in (600, 2560, 9000)]
    free = [lib.vosti_attention_decode_segment_keys(c, nq, nkv, d, n) for c, n in shapes]
    assert len(set(free)) > 1
    assert lib.vosti_set_decode_segment(576) == 0
    try:
        assert {lib.vosti_attention_decode_segment_keys(c, nq, nkv, d, n) for c, n in shapes} == {576}
        assert lib.vosti_set_decode_segment(100) != 0            # not a multiple of 64: refused, the pin stays
        assert lib.vosti_attention_decode_segment_keys(8, nq, nkv, d, 2560) == 576
    finally:
        assert lib.vosti_set_decode_segment(0) == 0
    assert [lib.vosti_attention_decode_segment_keys(c, nq, nkv, d, n) for c, n in shapes] == free


def test_no_product_is_split_when_one_order_of_arithmetic_is_asked_for(lib):
    assert lib.vosti_fixed_order() == 0
    lib.vosti_set_fixed_order(1)
    try:
        for features, k in [(4096, 4096), (4096, 12288), (151936, 4096), (1000, 1000)]:
            assert {lib.vosti_gemm_tc_splits(t, features, k) for t in (1, 8, 64, 65, 128, 129, 4096)} == {1}
    finally:
        lib.vosti_set_fixed_order(0)
    assert lib.vosti_gemm_tc_splits(8, 4096, 12288) > 1


def test_narrow_products_over_many_tokens_split_where_that_is_faster(lib):
    """The sizes on both sides of the line at which splitting was measured faster and slower than one pass."""
    for tokens, features, k in [(129, 8, 1024), (2400, 128, 1024), (3200, 64, 1280), (3840, 128, 1536), (5000, 64, 2048),
                                (6300, 128, 2560), (9400, 128, 4096), (9400, 8, 12288)]:
        assert lib.vosti_gemm_tc_splits(tokens, features, k) > 1, (tokens, features, k)
    for tokens, features, k in [(4800, 8, 1024), (4096, 64, 1024), (4800, 32, 1280), (6300, 32, 1536), (8192, 128, 2048),
                                (9400, 128, 2560), (9473, 8, 12288), (2048, 129, 4096), (2048, 128, 960)]:
        assert lib.vosti_gemm_tc_splits(tokens, features, k) == 1, (tokens, features, k)


def test_latent_portions_take_the_kernel_that_was_measured_faster():
    """Steps (heads, tokens and keys of the requests) on both sides of the line between tiles of 32 and of 128 rows."""
    from vosti_b200 import ops

    def takes(heads, q, past, window=0):
        kv = [a + b for a, b in zip(q, past)]
        tiles = -(-max(q) * heads // 32) * len(q)
        return ops.latent_takes_tiles(q, kv, heads, window, tiles < ops.LATENT_MMA_SPLIT_BELOW)

    singles = lambda n, count, keys: ([n] + [1] * count, [0] + [keys] * count)
    for heads, (q, past) in [(16, ([1024], [0])), (16, ([600, 600], [0, 100])), (8, ([2048], [0])), (16, singles(300, 20, 2000)),
                             (16, singles(640, 60, 500)), (64, ([8] * 16, [100] * 16)), (64, ([128], [0])), (64, singles(8, 300, 1000)),
                             (64, singles(16, 150, 600)), (128, ([64], [0])), (128, singles(8, 300, 100))]:
        assert takes(heads, q, past), (heads, q, past)
    for heads, (q, past) in [(16, ([8], [0])), (16, ([64], [0])), (8, ([64], [0])), (64, ([64], [0])), (128, ([8], [0])),
                             (16, singles(8, 300, 100)), (16, singles(8, 300, 1000)), (16, singles(16, 150, 600)),
                             (8, singles(16, 150, 600)), (64, singles(8, 300, 100)), (16, ([9] * 40, [100] * 40))]:
        assert not takes(heads, q, past), (heads, q, past)
    assert takes(16, [700], [0], window=128) and not takes(16, *singles(8, 300, 5000), window=100)


def test_cuda_core_attention_takes_the_way_that_was_measured_faster():
    """Steps (query and kv heads, tokens and keys of the requests) where warps (0), blocks of rows (1) and both (2) were."""
    from vosti_b200.ops import simt_way
    some = ([64, 1, 5, 1, 40, 1, 2, 1], [500, 2000, 1500, 900, 40, 2500, 1200, 700])
    beside = lambda n, kv, count, keys: ([n] + [1] * count, [kv] + [keys] * count)
    for way, nq, nkv, (q, kv) in [
            (1, 32, 8, ([384], [384])), (1, 32, 8, ([4], [3000])), (1, 16, 16, ([16], [16])), (1, 32, 8, ([8] * 4, [2000] * 4)),
            (1, 16, 16, ([8] * 64, [1000] * 64)), (1, 32, 8, ([4] * 64, [1000] * 64)), (1, 16, 16, some), (1, 64, 2, beside(128, 128, 32, 3000)),
            (2, 16, 16, beside(300, 900, 60, 1500)), (2, 32, 8, beside(300, 900, 60, 1500)),
            (0, 16, 16, beside(128, 128, 32, 3000)), (0, 32, 8, beside(64, 64, 12, 2000)), (0, 16, 16, ([5] * 8, [3000] * 8)),
            (0, 16, 16, ([4] * 16, [1000] * 16)), (0, 16, 16, ([4] * 64, [1000] * 64)), (0, 16, 16, ([8] * 4, [2000] * 4)),
            (0, 16, 16, ([32] + [3] * 9, [400] + [2000] * 9)), (0, 32, 8, ([32] + [3] * 9, [400] + [2000] * 9)),
            (0, 32, 8, ([5] * 8, [3000] * 8)), (0, 32, 8, ([1] * 12, [2000] * 12)), (0, 32, 1, ([4], [4])), (0, 16, 16, ([8], [8])),
            (0, 66, 2, ([384], [384]))]:
        assert simt_way(q, kv, nq, nkv) == way, (nq, nkv, q, kv, simt_way(q, kv, nq, nkv))
    assert simt_way([128] + [0] + [9], [128, 50, 9], 32, 8, window=40) == 1


def test_delta_rules_take_the_form_that_was_measured_faster(lib):
    """Steps (heads, values a head, tokens of the requests) on both sides of the line between chunks and token by token, for
    both rules. Of 3,279 measured steps the rule takes chunks in 20 where they were more than 3 % slower, none of them here."""
    from vosti_b200.ops import delta_step_layout, delta_takes_chunks
    takes = lambda pair, heads, dv, q: delta_takes_chunks(delta_step_layout(q)[1], heads, dv, pair)
    gated = {True: [(16, 128, [96]), (16, 128, [256]), (16, 128, [2048]), (16, 128, [128] * 2), (16, 128, [256] * 4), (16, 128, [1031, 700, 317]),
                    (16, 128, [300] + [1] * 30), (16, 128, [80]), (16, 128, [64] + [1] * 30), (16, 128, [256] * 8), (16, 128, [256] * 16),
                    (4, 128, [64]), (4, 128, [96]), (4, 128, [128]), (4, 128, [256] * 8), (2, 128, [128] * 2), (8, 128, [128] * 4),
                    (32, 128, [256]), (32, 128, [700]), (32, 128, [96] * 4), (16, 64, [128] * 2), (8, 256, [96]), (8, 256, [96] * 4),
                    (8, 256, [128]), (64, 128, [256]), (64, 128, [64] + [1] * 30)],
             False: [(16, 128, [49]), (16, 128, [64] * 4), (16, 128, [64] * 16), (64, 128, [64]), (64, 128, [80]), (4, 128, [49])]}
    general = {True: [(16, 128, [128]), (16, 128, [256]), (16, 128, [2048]), (16, 128, [128] * 2), (16, 128, [64] * 4), (16, 128, [96] * 4),
                      (16, 128, [128] * 4), (16, 128, [64] * 16), (16, 128, [256] * 16), (16, 128, [1031, 700, 317]), (16, 128, [96] + [1] * 30),
                      (4, 128, [96]), (4, 128, [128]), (4, 128, [256]), (8, 128, [128] * 4), (32, 128, [128]), (32, 128, [128] * 16),
                      (32, 128, [256] * 8), (4, 128, [300] + [1] * 30), (64, 128, [128]), (64, 128, [64] * 4), (64, 128, [96] * 8)],
               False: [(16, 128, [49]), (16, 128, [80]), (16, 128, [96]), (16, 128, [112]), (16, 128, [49] * 16), (2, 128, [64]), (4, 128, [64]),
                       (4, 128, [96] * 4), (64, 128, [49] * 4)]}
    for pair, table in ((False, gated), (True, general)):
        for want, steps in table.items():
            for step in steps:
                assert takes(pair, *step) == want, (pair, step)
    arrays, values = delta_step_layout([20, 70, 100, 1])
    assert values == {"chunks": 7, "longs": 2, "shorts": 2, "longest": 100, "tokens": 170, "short_longest": 20, "short_tokens": 21}
    assert arrays["plan"] == [2] * 4 + [1] * 3 + [0, 32, 64, 96, 0, 32, 64] + [2, 1] + [0, 4]
    assert delta_step_layout([1, 48, 3]) == ({}, {"chunks": 0, "longs": 0, "shorts": 3})


def test_products_of_few_tiles_split_where_that_is_faster(lib):
    """The number of cuts at sizes on both sides of the line at which cutting K was measured faster and slower than one pass."""
    for tokens, features, k, cuts in [(200, 4096, 12288, 4), (300, 4096, 12288, 2), (512, 4096, 12288, 2), (256, 6144, 4096, 3), (130, 4096, 4096, 4),
                                      (300, 4096, 4096, 2), (653, 2048, 4096, 3), (512, 1024, 8192, 6), (1000, 1024, 8192, 4)]:
        assert lib.vosti_gemm_tc_pair_splits(tokens, features, k) == cuts, (tokens, features, k)
    for tokens, features, k in [(128, 4096, 12288), (653, 4096, 12288), (300, 6144, 4096), (256, 3664, 2048), (512, 2048, 2048), (130, 8192, 2048),
                                (200, 24576, 4096), (256, 5120, 1536), (700, 1024, 512), (2048, 128, 4096)]:
        assert lib.vosti_gemm_tc_pair_splits(tokens, features, k) == 1, (tokens, features, k)


def test_delta_preparation_takes_the_tokens_a_warp_that_were_measured_faster(lib):
    """(tokens, heads of q, k and v) on both sides of the line between one and four tokens a warp; the times are beside the rule."""
    for tokens, units in [(1, 24), (395, 24), (600, 24), (1200, 24), (1500, 24), (200, 48), (350, 48), (700, 48), (1200, 8), (3000, 8)]:
        assert lib.vosti_delta_prep_tokens(tokens, units) == 1, (tokens, units)
    for tokens, units in [(2048, 24), (3000, 24), (1000, 48), (1500, 48), (2048, 48), (1 << 20, 8192)]:
        assert lib.vosti_delta_prep_tokens(tokens, units) == 4, (tokens, units)


def test_float32_weights_go_to_the_product_whose_single_row_was_faster(lib):
    """Weights on both sides of the line between the tensor cores and the chain of multiply-adds; rows that do not start on whole words stay."""
    for n, k in [(16, 2048), (2048, 2048), (2048, 2304), (160, 4096), (4096, 1024), (4096, 1536), (8192, 1024), (4096, 4096), (24576, 4096), (4096, 12288)]:
        assert lib.vosti_gemm_f32_supported(n, k), (n, k)
    for n, k in [(512, 1024), (1024, 1024), (3072, 1024), (1024, 1536), (2048, 1920), (3072, 1920), (4096, 512), (8, 4096), (4096, 4098), (2048, 2049),
                 (512, 1026)]:
        assert not lib.vosti_gemm_f32_supported(n, k), (n, k)


def test_a_product_that_is_cut_needs_its_workspace(lib):
    """One that is missing or too small is refused before anything else happens, in the narrow and in the paired product alike."""
    def call(tokens, features, k, elems):
        code = lib.vosti_gemm_tc(None, None, None, tokens, features, k, 0, ctypes.c_void_p(16 if elems else 0), ctypes.c_int64(elems), 0, 0, 0,
                                 None, None)
        return code, lib.vosti_last_error().decode()

    lib.vosti_last_error.restype = ctypes.c_char_p
    for tokens, features, k, parts in [(8, 4096, 4096, lib.vosti_gemm_tc_splits(8, 4096, 4096)), (200, 4096, 12288, 4)]:
        for elems in (0, parts * tokens * features - 1):
            code, message = call(tokens, features, k, elems)
            assert code != 0 and f"workspace too small for {parts} splits" in message, (tokens, elems, message)


def test_float32_tiles_never_ask_for_more_tensor_memory_than_an_sm_has(lib):
    """CTAs of a cluster wait for their tensor memory without a limit: shared memory keeps as many of them on an SM as it has columns for."""
    columns = [lib.vosti_gemm_f32_columns_an_sm(tile) for tile in range(6)]
    assert all(0 < c <= 512 for c in columns) and lib.vosti_gemm_f32_columns_an_sm(6) == -1, columns


def test_weight_bytes_of_a_decode_step_in_closed_form():
    """What bench.py counts as the weights a decode step must read: every tensor the model
    expects except the embedding table (read by rows), two bytes each. For the 8B sizes that is
    13.892 GB of layers + the final norm + 1.245 GB of output head."""
    import importlib.util
    import math
    import os
    from vosti_b200.config import model_spec_from_config
    from vosti_b200.models import expected_weights
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bench.py")
    spec = importlib.util.spec_from_file_location("bench_for_test", path)
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    for size, (_, config) in bench.SIZES.items():
        names = expected_weights(model_spec_from_config(config))
        total = sum(2 * math.prod(w.shape) for name, w in names.items() if name != "model.embed_tokens.weight")
        assert bench.closed_form_weight_bytes(config) == total, size
    layers = bench.closed_form_weight_bytes(bench.SIZES["8b"][1]) - 2 * 151936 * 4096
    assert abs(layers - 13.892e9) < 2e6 and 2 * 151936 * 4096 == 1_244_659_712


def test_latent_attention_forms_keys_and_values_where_that_was_faster():
    """Whole mixers of 16 heads and rank 512, then of others: (tokens, keys before them, whether formed heads were measured faster)."""
    from vosti_b200 import ops
    for new, past, formed in [([33], [0], True), ([128], [0], True), ([700], [0], True), ([2048], [0], True), ([131], [700], True),
                              ([500] * 3, [0, 64, 0], True), ([1024] + [1] * 8, [0] + [1000] * 8, True), ([5, 17, 200], [0, 30, 1400], True),
                              ([64, 64], [0, 0], True), ([20], [1500], False), ([8], [64], False), ([16] * 20, [100] * 20, False),
                              ([100] + [1] * 12, [0] + [1500] * 12, False), ([1] * 16, [700] * 16, False)]:
        assert ops.latent_forms_heads(new, [a + b for a, b in zip(new, past)], 16, 512) is formed, (new, past)
    for heads, rank, new, past, formed in [
            (8, 512, [33], [0], True), (8, 512, [300], [1500], True), (8, 512, [64], [1000], False), (8, 512, [300] + [1] * 30, [0] + [500] * 30, False),
            (32, 512, [64], [1000], True), (32, 512, [1024] + [1] * 8, [0] + [1000] * 8, True), (32, 512, [30], [1000], False),
            (64, 512, [64], [0], True), (64, 512, [131], [700], True), (128, 512, [64], [0], True), (128, 512, [40] * 8, [0] * 8, True),
            (16, 256, [64], [0], True), (16, 256, [131], [700], True), (16, 256, [64], [1000], False), (16, 256, [100] + [1] * 12, [0] + [1500] * 12, False),
            (64, 256, [64], [1000], True), (64, 256, [24], [200], False), (64, 256, [30], [1000], False)]:
        assert ops.latent_forms_heads(new, [a + b for a, b in zip(new, past)], heads, rank) is formed, (heads, rank, new, past)


def test_latent_attention_forms_no_heads_where_a_batch_must_not_change_a_prompt(lib, monkeypatch):
    from types import SimpleNamespace
    from vosti_b200 import ops

    def forms(q, kv):
        ctx = SimpleNamespace(num_requests=len(q), host_q_lens=q, host_kv_lens=kv, layout={})
        return ops._latent_forms_heads(ctx, heads=16, dim=128, rot=64, dv=128, rank=512, window=0, scale=0.07, page_size=16, q_width=3664)

    alone, beside = ([100], [100]), ([100] + [1] * 12, [100] + [1500] * 12)
    assert forms(*alone) and not forms(*beside)              # the same prompt in two forms
    for name, value in (("INVARIANCE", "decode"), ("FIXED_ORDER", True)):
        with monkeypatch.context() as m:
            m.setattr(ops, name, value)
            assert not forms(*alone) and not forms(*beside)
