"""The host-side rules that pick a kernel's shape (no GPU needed): slices of the decode attention, key parts of
the prefill attention, tile and K slices of the streaming matrix product, and which product a projection runs."""
import numpy as np
import pytest

from slipstream_b200.ops import functions as F

SMS = 148  # the rules take the device's number of multiprocessors; here a B200's, without a device


def test_decode_slices_fill_one_wave_and_go_wide_only_for_few_long_requests():
    for n_requests in (1, 2, 3, 8, 24, 64, 300):
        for ctx in (1, 64, 1000, 8192, 32768):
            s = F.decode_slices(n_requests, 4, 7, ctx, sms=SMS)
            assert s in (1, 2, 4, 8) and s <= max(1, (ctx + 63) // 64)
            assert s == 1 or n_requests * 4 * s <= 2 * SMS
            w = F.decode_slices(n_requests, 4, 7, ctx, wide=True, sms=SMS)
            assert w == s or (w % 8 == 0 and w > 8 and n_requests * 4 * w <= 2 * SMS and ctx >= 64 * 8 * w)
    assert F.decode_slices(1, 4, 7, 32768, wide=True, sms=SMS) == 64 and F.decode_slices(8, 4, 7, 32768, wide=True, sms=SMS) == 8
    assert F.is_long_context(8192) and not F.is_long_context(8191)


def test_prefill_key_parts_only_while_all_blocks_run_at_once():
    assert F.prefill_key_parts([2048], [2048], 18, 4, sms=SMS) == 1          # 456 blocks
    assert F.prefill_key_parts([64], [4096], 18, 4, sms=SMS) == 8            # 16 blocks of 64 key tiles
    assert F.prefill_key_parts([512], [4096], 18, 4, sms=SMS) == 2           # 116 blocks
    assert F.prefill_key_parts([64], [600], 18, 4, sms=SMS) == 1             # too few key tiles to share
    assert F.prefill_key_parts([1] * 8 + [256], [4096] * 9, 18, 4, sms=SMS) == 2
    assert F.prefill_key_parts([], [], 18, 4, sms=SMS) == 1
    rng = np.random.default_rng(0)
    for _ in range(200):
        n = int(rng.integers(1, 6))
        seq = rng.integers(1, 20000, n)
        q = np.minimum(seq, rng.integers(1, 3000, n))
        parts = F.prefill_key_parts(q, seq, 18, 4, sms=SMS)
        blocks = int(((q + 17) // 18).sum()) * 4
        assert parts in (1, 2, 4, 8)
        assert parts == 1 or (blocks * parts <= 2 * SMS and (int(seq.max()) - 1) // 64 + 1 >= 8 * parts)


def test_streaming_product_plan_and_routing():
    for tokens in (1, 8, 16, 17, 33, 64):
        for features, k in ((4608, 3584), (3584, 3584), (37888, 3584), (3584, 18944), (152064, 3584), (96, 64)):
            swapped, bn, slices = F.gemm_plan(tokens, features, k, SMS)
            assert swapped and bn >= tokens and bn in (16, 32, 64) and 1 <= slices <= 8
            assert slices <= (k + 63) // 64
    # few tokens: every projection streams its weights through our kernel; 17 to 64: the large ones
    assert all(F.streams_weights(8, f, k, SMS) for f, k in ((4608, 3584), (3584, 3584), (37888, 3584), (3584, 18944)))
    assert F.streams_weights(64, 37888, 3584, SMS) and F.streams_weights(64, 3584, 18944, SMS) and not F.streams_weights(64, 3584, 3584, SMS)
    assert not F.streams_weights(65, 37888, 3584, SMS) and not F.streams_weights(8, 3584, 3580, SMS)
    assert F.many_tokens_swiglu_fits(2048, 37888, SMS) and not F.many_tokens_swiglu_fits(512, 37888, SMS)
    # prompt portions: the two-SM kernel from 2,048 tokens at the 7B and 14B layer sizes, the library elsewhere
    for features, k in ((4608, 3584), (3584, 3584), (3584, 18944), (7168, 5120), (5120, 13824)):
        assert F.many_tokens_fits(2048, features, k, SMS) and not F.many_tokens_fits(2047, features, k, SMS)
    for features, k in ((1152, 896), (896, 4864), (2048, 1536), (3584, 3580)):
        assert not F.many_tokens_fits(4096, features, k, SMS)


def test_gated_products_of_about_one_tile_a_multiprocessor_keep_their_sums_in_one_block():
    for tokens in (1, 16, 24, 64):
        assert all(F.gemm_plan(tokens, f, k, SMS, True)[2] == 1 for f, k in ((9728, 896), (17920, 1536), (13440, 20000), (18944, 8192)))
        assert F.gemm_plan(tokens, 9728, 1536, SMS, True) == F.gemm_plan(tokens, 9728, 1536, SMS)
        assert F.gemm_plan(tokens, 37888, 3584, SMS, True) == F.gemm_plan(tokens, 37888, 3584, SMS)
        for f, k in ((7680, 896), (9728, 8192), (17920, 896)):  # more than 16 columns: within one wave of two blocks an SM
            _, bn, slices = F.gemm_plan(tokens, f, k, SMS)
            assert bn == 16 or slices * (f // 128) <= SMS + 3 * SMS // 4


def test_float32_outputs_keep_their_slices():
    assert F.gemm_plan(24, 5120, 5120, SMS)[2] == 6 and F.gemm_plan(24, 5120, 5120, SMS, out_f32=True)[2] == 8
    assert F.gemm_plan(48, 5120, 5120, SMS)[2] == F.gemm_plan(48, 5120, 5120, SMS, out_f32=True)[2]


def test_gated_products_in_one_block_keep_the_sums_of_their_slices():
    for tokens in (1, 16, 24, 64):
        for features in range(128, 20000, 128):
            for k in (64, 200, 256, 320, 896, 4096, 8192):
                sums, slices = F.gated_sums(tokens, features, k, SMS), F.gemm_plan(tokens, features, k, SMS, out_f32=True)[2]
                _, bn, gated = F.gemm_plan(tokens, features, k, SMS, True)
                tiles = features // 128
                # the sums of the slices, in as many columns of tensor memory as a block alone on its SM may take
                assert sums == 1 or gated == 1 and sums == slices and sums <= 8 and sums * bn <= 256
                assert gated == 1 or sums == 1
                assert sums == 1 or tiles <= SMS and ((k + 63) // 64 > 4 or tiles <= SMS // 2)


def test_where_a_projection_adds_itself_to_the_stream():
    """The last projection of a branch takes over the add and prepares the norm behind it in decode steps of up to
    16 tokens, where its K slices are a cluster and the width is a multiple of 128; for long prompt portions only
    when asked for."""
    for features, k in ((3584, 3584), (3584, 18944), (896, 4864), (5120, 13824), (128, 256)):
        for tokens in (1, 8, 16):
            assert F.adds_to_stream(tokens, features, k, SMS), (tokens, features, k)
        assert not F.adds_to_stream(17, features, k, SMS) and not F.adds_to_stream(64, features, k, SMS)
    assert not F.adds_to_stream(8, 3600, 3584, SMS)       # a width that is no multiple of 128
    assert not F.adds_to_stream(8, 3584, 3580, SMS)       # K that the tensor-core product does not take
    assert not F.adds_to_stream(8, 128, 64, SMS)          # one K step: nothing to cut into slices
    assert not F.adds_to_stream(2048, 3584, 3584, SMS)    # the two-SM kernel could; it did not pay
    try:
        F.set_norm_fusion(True, long_portions=True)
        assert F.adds_to_stream(2048, 3584, 3584, SMS) and not F.adds_to_stream(2047, 3584, 3584, SMS)
        F.set_norm_fusion(False)
        assert not F.adds_to_stream(8, 3584, 3584, SMS) and not F.adds_to_stream(2048, 3584, 3584, SMS)
    finally:
        F.set_norm_fusion(True)
    assert F.adds_to_stream(8, 3584, 3584, SMS)


def test_head_sizes_between_the_boxes_leave_the_mma_sync_kernel_only_for_enough_keys():
    from types import SimpleNamespace
    import torch

    out = torch.empty(4, 64, dtype=torch.bfloat16)
    runs = lambda longest, d, out=out, gate=None, **told: F._prefill_on_tcgen05(
        SimpleNamespace(max_seq_len=longest, extras={("few_keys", k): v for k, v in ((d, told.get("few")),) if v is not None}), d, 8, 2, 16, out, gate)
    for d, few in ((32, 128), (48, 128), (80, 64), (96, 64), (112, 64)):
        assert F.tcgen05_prefill_fits(d, 8, 2, 16) and not F.tcgen05_attention_fits(d, 8, 2, 16, 0)
        assert not runs(few, d) and runs(few + 1, d)
        assert runs(0, d, few=False) and not runs(5000, d, few=True)                     # a captured step is told
        assert not runs(5000, d, gate=out)                                               # gated before rounding there
        assert not runs(5000, d, out=out.view(-1)[1:65].view(1, 64))                     # 16-byte stores
    assert runs(1, 64, gate=out) and runs(1, 128)
    for d, n_q, n_kv, page in ((16, 8, 2, 16), (160, 8, 2, 16), (40, 8, 2, 16), (96, 8, 2, 12), (96, 8, 2, 128), (96, 129, 1, 16)):
        assert not F.tcgen05_prefill_fits(d, n_q, n_kv, page)


def test_expert_tiles_and_float32_key_parts():
    for experts in (1, 8, 100):
        widths = [F.expert_tile(p, experts, True, False, True) for p in range(1, 40 * experts)]
        assert widths == sorted(widths) and set(widths) == {16, 32, 64, 128}
    assert F.expert_tile(5000, 8, True, True, False) == 256 and F.expert_tile(8, 8, False, False, False) == F.MOE_TILE
    assert F.float32_key_parts(8, 20, 4, 12, 128, sms=SMS) == 20 and F.float32_key_parts(100, 20, 4, 12, 128, sms=SMS) == 2
    assert F.float32_key_parts(400, 20, 4, 12, 128, sms=SMS) == 1
    assert F.float32_key_parts(8, 20, 5000, 28, 128, sms=SMS) == 1  # the slices' scratch would pass its bound


def test_float32_decode_deals_out_slices_within_the_scratch_memory():
    for blocks in (1, 8, 100, 5000):
        for slices in (2, 16, 250):
            parts = F.float32_decode_parts(blocks, slices, 4, 12, 128, sms=SMS)
            assert 2 <= parts <= slices and (parts == 2 or blocks * parts <= 8 * SMS)  # (2: the slices meet in scratch memory)
    assert F.float32_decode_parts(8, 1, 4, 12, 128, sms=SMS) == 1
    bound = F.FLOAT32_SCRATCH // (12 * 16 * (128 + 2) * 4)  # rows whose slices just fit
    assert F.float32_decode_parts(8, 16, bound, 12, 128, sms=SMS) > 1 == F.float32_decode_parts(8, 16, bound + 1, 12, 128, sms=SMS)



def paged_layer(dim, page_size=16, **kind):
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts import PagedAttention, RotaryEncoding

    layer = PagedAttention("attn", 64, 4, 2, dim, RotaryEncoding(dim, 1e4), page_size=page_size, **kind)
    layer.runtime = SimpleNamespace(dtype=torch.bfloat16, device=0)
    return layer


def test_a_layer_off_the_tcgen05_kernel_does_not_answer_for_another_of_its_head_size(monkeypatch):
    from types import SimpleNamespace

    monkeypatch.setattr(F, "_device_sm_count", lambda index: SMS)
    taken, other = paged_layer(96), paged_layer(96, page_size=12)
    for length, wanted in ((30, 0), (9000, 8)):
        plan = SimpleNamespace(is_decode_only=False, q_lens=np.array([30]), seq_lens=np.array([length]))
        assert taken.capture_variant(length, plan) == wanted and other.capture_variant(length, plan) is None
        ctx = SimpleNamespace(is_decode_only=False, extras={})
        for layer in (taken, other):
            layer.prepare_capture(ctx, layer.capture_variant(length, plan), 16384)
        # as in the step that is not captured
        assert ctx.extras == {("few_keys", 96): wanted == 0, ("prefill_key_parts", 64, 2, 0): max(wanted, 1)}


def test_gated_layers_of_the_mma_sync_kernel_are_captured_in_one_form(monkeypatch):
    from types import SimpleNamespace

    monkeypatch.setattr(F, "_device_sm_count", lambda index: SMS)
    gated, plain = paged_layer(96, gate=True), paged_layer(96)
    assert gated.capture_group() != plain.capture_group()
    answers = [[layer.capture_variant(n, SimpleNamespace(is_decode_only=False, q_lens=np.array([30]), seq_lens=np.array([n])))
                for n in (30, 300, 9000)] for layer in (gated, plain, paged_layer(64, gate=True))]
    assert answers[0] == [None] * 3 and answers[1][0] == 0 and len(set(answers[1])) == 3 and len(set(answers[2])) == 2


def test_steps_of_short_portions_run_the_recurrences_token_by_token_captured_or_not():
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts.recurrent import MatrixMemoryMixer
    from slipstream_b200.parts.state_space import StateSpaceMixer

    parts = [StateSpaceMixer("s", 64, 4, 16, 16), MatrixMemoryMixer("m", 64, 2, 16, 16, 15.0)]
    for part in parts:
        part.runtime = SimpleNamespace(dtype=torch.bfloat16)
    assert parts[0].capture_group() == parts[1].capture_group()
    for longest, short in ((2, True), (F.SCAN_FEW, True), (F.SCAN_FEW + 1, False), (700, False)):
        plan = SimpleNamespace(is_decode_only=False, q_lens=np.array([1, longest]))
        assert F.only_short_portions(SimpleNamespace(extras={}, max_q_len=longest)) == short
        for part in parts:
            # the static context of a captured step says 2 for every length
            captured = SimpleNamespace(is_decode_only=False, extras={}, max_q_len=2, static_tiles=len)
            assert not F.only_short_portions(captured)
            part.prepare_capture(captured, part.capture_variant(longest, plan), 4096)
            assert F.only_short_portions(captured) == short
    assert parts[0].capture_variant(5) is None and parts[0].capture_variant(5, SimpleNamespace(is_decode_only=True)) is None


def test_recurrences_without_a_kernel_for_chunks_are_captured_in_one_form():
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts.recurrent import MatrixMemoryMixer
    from slipstream_b200.parts.state_space import StateSpaceMixer

    chunked = StateSpaceMixer("s", 64, 4, 16, 16)
    chunked.runtime = SimpleNamespace(dtype=torch.bfloat16)
    for part, dtype in ((StateSpaceMixer("s", 64, 4, 16, 16), torch.float32), (StateSpaceMixer("s", 64, 4, 12, 16), torch.bfloat16),
                        (MatrixMemoryMixer("m", 64, 2, 16, 20, 15.0), torch.bfloat16)):
        part.runtime = SimpleNamespace(dtype=dtype)
        assert part.capture_group() != chunked.capture_group()
        captured = SimpleNamespace(is_decode_only=False, extras={"short_portions": True})
        for longest in (3, 300):
            variant = part.capture_variant(longest, SimpleNamespace(is_decode_only=False, q_lens=np.array([longest])))
            assert variant is None
            part.prepare_capture(captured, variant, 4096)
        assert captured.extras == {"short_portions": True}


def test_latent_layers_off_the_tcgen05_kernel_are_captured_in_one_form():
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts import RotaryEncoding
    from slipstream_b200.parts.latent_attention import LatentAttention

    def layer(dtype, **kind):
        part = LatentAttention("l", 64, 4, 32, 16, 32, 48, 80, 0.2, RotaryEncoding(16, 1e4), **kind)
        part.runtime = SimpleNamespace(dtype=dtype)
        return part

    taken, off = layer(torch.bfloat16), [layer(torch.float32), layer(torch.bfloat16, page_size=12)]
    plan = lambda: SimpleNamespace(is_decode_only=False)  # noqa: E731
    assert [taken.capture_variant(n, plan()) for n in (30, 300)] == [True, False]
    for part in off:
        assert part.capture_group() != taken.capture_group() and part.capture_variant(30, plan()) is None
        ctx = SimpleNamespace(is_decode_only=False, extras={})
        taken.prepare_capture(ctx, True, 4096)
        part.prepare_capture(ctx, None, 4096)
        assert ctx.extras == {("few_keys", 96): True}


def test_attention_layers_share_an_answer_only_where_it_would_be_the_same(monkeypatch):
    """The runner asks one layer of a group: layers of other heads, pages or head counts are asked themselves."""
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts import PagedAttention, RotaryEncoding

    monkeypatch.setattr(F, "_device_sm_count", lambda index: SMS)
    layers = []
    for heads, kv_heads, page in ((4, 2, 16), (4, 2, 12), (28, 4, 16), (32, 32, 16), (4, 2, 32)):
        layers.append(PagedAttention("attn", 64, heads, kv_heads, 96, RotaryEncoding(96, 1e4), page_size=page))
        layers[-1].runtime = SimpleNamespace(dtype=torch.bfloat16, device=0)
    assert layers[0].capture_group() == layers[4].capture_group()
    for tokens, length in ((30, 30), (30, 9000), (500, 9000), (2000, 2000)):
        plan = SimpleNamespace(is_decode_only=False, q_lens=np.array([tokens]), seq_lens=np.array([length]))
        answers = {}
        for layer in layers:
            assert answers.setdefault(layer.capture_group(), layer.capture_variant(length, plan)) == layer.capture_variant(length, plan)


def test_decode_tiles_are_dealt_out_where_that_was_measured_to_pay_captured_or_not(monkeypatch):
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts import PagedAttention, RotaryEncoding

    def uneven(n, mean):
        weights = np.array([2 + i % 5 for i in range(n)])
        return (weights * n * mean / weights.sum()).astype(np.int32)

    spreads = lambda lens, n_kv=4, group=7, d=128, reach=0: F.spreads_decode(np.asarray(lens, dtype=np.int32), n_kv, group, d, reach, SMS)  # noqa: E731
    assert spreads(uneven(48, 1800)) and spreads(uneven(40, 1200)) and spreads(uneven(24, 1800), 8, 4) and spreads(uneven(40, 1200), 4, 8, 64)
    assert not spreads(uneven(48, 300)) and not spreads([1200] * 64) and not spreads([1200] * 48, 4, 8, 64) and not spreads([1])
    assert not spreads(uneven(48, 1800), reach=512)           # a window leaves little to deal out
    assert not spreads(uneven(48, 1800), 4, 9)                # more heads than lie beside the merge
    assert not spreads(uneven(200, 1800), 1) and not spreads(uneven(8, 1800)) and not spreads(uneven(600, 1800))
    # a captured step is told what a step run kernel by kernel finds out from its lengths
    monkeypatch.setattr(F, "_device_sm_count", lambda index: SMS)
    layer = PagedAttention("attn", 64, 28, 4, 128, RotaryEncoding(128, 1e4), page_size=16)
    layer.runtime = SimpleNamespace(dtype=torch.bfloat16, device=0)
    for lens in (uneven(48, 1800), uneven(48, 300), uneven(48, 9000), np.array([9000])):
        plan = SimpleNamespace(is_decode_only=True, q_lens=np.ones(lens.size, dtype=np.int32), seq_lens=lens)
        ctx = SimpleNamespace(is_decode_only=True, num_requests=lens.size, device=None, extras={}, set_query_tiles=lambda *a: None)
        layer.prepare_capture(ctx, layer.capture_variant(int(lens.max()), plan), 16384)
        assert ctx.extras["decode_wide"] == F.is_long_context(int(lens.max()))
        assert ctx.extras[("decode_spread", 4, 7, 128, layer.sees)] == spreads(lens)
    assert layer.capture_variant(5000) == 0  # (no lengths yet: the form for any)


def test_layers_off_the_spread_decode_kernel_are_captured_in_one_form(monkeypatch):
    """Head sizes and pages that the kernel does not take, the engine's own page size among them: the rule is not asked, and
    such a layer does not change what one of the same heads and reach was told."""
    from types import SimpleNamespace
    import torch
    from slipstream_b200.parts import PagedAttention, RotaryEncoding
    from slipstream_b200.parts.base import Runtime

    monkeypatch.setattr(F, "_device_sm_count", lambda index: SMS)
    lens = (np.array([2 + i % 5 for i in range(48)]) * 450).astype(np.int32)
    plan = SimpleNamespace(is_decode_only=True, q_lens=np.ones(48, dtype=np.int32), seq_lens=lens)

    def layer(dim=128, page=None, pages=16, dtype=torch.bfloat16):
        made = PagedAttention("attn", 64, 28, 4, dim, RotaryEncoding(dim, 1e4), page_size=page)
        made.runtime = Runtime(torch.device("cuda:0"), dtype, pages)
        return made

    taken = [layer(), layer(64), layer(page=32, pages=128), layer(pages=8)]
    others = [layer(d) for d in (32, 80, 96, 192, 256)] + [layer(page=48), layer(pages=128), layer(dtype=torch.float32)]
    assert F.spreads_decode(lens, 4, 7, 96, 0, SMS)  # (the rule alone would say yes)
    assert [x.capture_variant(int(lens.max()), plan) for x in taken] == [2] * 4
    assert [x.capture_variant(int(lens.max()), plan) for x in others] == [0] * 8
    assert len({layer().capture_group(), layer(pages=128).capture_group(), layer(page=48).capture_group()}) == 2
    ctx = SimpleNamespace(is_decode_only=True, num_requests=48, device=None, extras={}, set_query_tiles=lambda *a: None)
    for x in (layer(), layer(pages=128)):
        x.prepare_capture(ctx, x.capture_variant(int(lens.max()), plan), 16384)
    assert ctx.extras[("decode_spread", 4, 7, 128, 0)] is True


def bare_runner(monkeypatch, layer, max_num_seqs, max_model_len=4096):
    """A model runner of one layer that records the graphs it captures instead of capturing them."""
    from types import SimpleNamespace
    from slipstream_b200.engine import runner as module
    monkeypatch.setattr(F, "_device_sm_count", lambda index: SMS)
    monkeypatch.setattr(module, "DecodeGraph", lambda runner, bucket, variants: SimpleNamespace(bucket=bucket, variants=variants))
    made = module.ModelRunner.__new__(module.ModelRunner)
    made.use_cuda_graphs, made.max_num_seqs, made.max_model_len, made.variant_parts, made._graphs = True, max_num_seqs, max_model_len, [layer], {}
    return made


def decode_plan(lens):
    from types import SimpleNamespace
    lens = np.asarray(lens, dtype=np.int32)
    return SimpleNamespace(is_decode_only=True, q_lens=np.ones(lens.size, dtype=np.int32), seq_lens=lens, rows=0)


def spread_layer(heads=28, kv_heads=4, **kind):
    import torch
    from slipstream_b200.parts import PagedAttention, RotaryEncoding
    from slipstream_b200.parts.base import Runtime
    layer = PagedAttention("attn", 64, heads, kv_heads, 128, RotaryEncoding(128, 1e4), **kind)
    layer.runtime = Runtime(torch.device("cuda:0"), torch.bfloat16)
    return layer


def test_the_rule_for_dealing_tiles_out_asks_for_the_requests_of_the_captured_step(monkeypatch):
    """36 requests run in the graph for 48, whose blocks are too many to cut a request's keys: they ask as those would.  In a graph of
    as many blocks as multiprocessors, where keys are cut, none does; nor behind 512 requests."""
    runner = bare_runner(monkeypatch, spread_layer(), 600)
    lens = [(2 + i % 5) * 450 for i in range(48)]
    for live, bucket, form in ((33, 48, 2), (36, 48, 2), (37, 48, 2), (48, 48, 2), (30, 32, 0), (24, 24, 0)):
        graph = runner._decode_graph(bucket, decode_plan(lens[:live]))
        assert (graph.bucket, graph.variants) == (bucket, (form,)), live
    one_long = np.array([20000] + [100] * 400, dtype=np.int32)
    assert [F.spreads_decode(one_long, 4, 7, 128, 0, SMS, rows=n) for n in (0, 512, 600)] == [True, True, False]


@pytest.mark.parametrize("kind, most, graphs", [(dict(), 64, 11), (dict(kv_heads=28), 64, 15), (dict(heads=4, kv_heads=1), 64, 9), (dict(page_size=48), 64, 9),
                                                (dict(window=128), 64, 9)])
def test_a_prepared_runner_captures_nothing_when_requests_become_uneven(monkeypatch, kind, most, graphs):
    runner = bare_runner(monkeypatch, spread_layer(**kind), most)
    assert runner.capture_decode_graphs() == graphs == len(runner._graphs)
    rng = np.random.default_rng(0)
    for live in (1, 5, 20, 24, 33, 40, 48, 50, 64):
        for mean in (1, 100, 700, 1500, 2300):
            for lens in ([mean] * live, rng.uniform(0.3, 1.7, live) * mean + 1, [4000] + [mean] * (live - 1)):
                runner._decode_graph(runner._graph_bucket(live), decode_plan(lens))
    assert len(runner._graphs) == graphs and runner.capture_decode_graphs() == 0
