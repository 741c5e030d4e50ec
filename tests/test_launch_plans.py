"""Host-side launch decisions that need no GPU: how the decode attention cuts a context into
splits, and which prefill attention kernel takes which head layout."""
import itertools
from types import SimpleNamespace

import pytest

from nanoinfer_b200.kernels import ops


@pytest.mark.parametrize("head_dim", [64, 128])
def test_decode_splits_are_bounded_and_leave_no_empty_split(head_dim):
    for n_items, n_kv, ctx in itertools.product([1, 2, 3, 8, 16, 19, 24, 32, 37, 40, 56, 64, 96, 128, 300],
                                                [1, 2, 8], [1, 63, 64, 65, 500, 2112, 3072, 4096, 16384, 131072]):
        s = ops.decode_splits(n_items, n_kv, head_dim, ctx, n_sms=148)
        assert 1 <= s <= 64
        chunks = -(-ctx // 64)
        assert s <= chunks                                  # a split holds at least one 64-key chunk
        per_split = -(-chunks // s)                          # the kernel's own cut of the longest context
        assert -(-chunks // per_split) == s                  # ... leaves no split of it empty
        if s > 1:
            assert per_split * 64 >= 256 or s == chunks      # no splits of a handful of keys


def test_decode_splits_follow_the_resident_blocks():
    # few pairs: as many fat blocks as fit at three per SM, of at least 256 / 384 keys
    assert ops.decode_splits(1, 8, 64, 3072, n_sms=148) == 12
    assert ops.decode_splits(8, 8, 64, 3072, n_sms=148) == 6
    assert 8 * 8 * ops.decode_splits(8, 8, 64, 131072, n_sms=148) <= 3 * 148
    # middle batches of 64-wide heads: lean blocks, four per SM
    assert ops.decode_splits(32, 8, 64, 3072, n_sms=148) == 2 and 32 * 8 * 2 <= 4 * 148
    assert ops.decode_splits(24, 8, 64, 3072, n_sms=148) == 3
    # large batches: one block per pair with heads of 64; with heads of 128 the last wave is filled
    assert ops.decode_splits(64, 8, 64, 3072, n_sms=148) == 1
    assert ops.decode_splits(64, 8, 128, 7168, n_sms=148) == 4
    assert ops.decode_splits(64, 8, 128, 300, n_sms=148) == 1           # too short to split
    assert ops.decode_splits(32, 8, 128, 3072, n_sms=148) == 1          # three per SM: 256 blocks are one wave


def test_tensor_core_prefill_attention_cases():
    assert ops.attention_prefill_tc_supports(32, 8, 64, 16)
    assert ops.attention_prefill_tc_supports(24, 8, 128, 16)        # odd group of three
    assert ops.attention_prefill_tc_supports(5, 1, 64, 128)
    assert not ops.attention_prefill_tc_supports(8, 8, 64, 16)      # one query head per kv head
    assert not ops.attention_prefill_tc_supports(8, 3, 64, 16)      # heads do not divide
    assert not ops.attention_prefill_tc_supports(8, 2, 96, 16)      # head size
    assert not ops.attention_prefill_tc_supports(8, 2, 64, 4)       # page size
    assert not ops.attention_prefill_tc_supports(8, 2, 64, 48)


def test_stream_objects_belong_to_their_device(monkeypatch):
    """The default stream has the raw handle 0 on every device: an event must be recorded on the current device's stream."""
    import torch
    place = {"device": 0, "raw": 0}
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: place["device"], raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: place["raw"], raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: (place["device"], place["raw"]))
    monkeypatch.setattr(ops, "_stream_objects", {})
    for device, raw in [(0, 0), (1, 0), (1, 77), (0, 77), (0, 0), (1, 0)]:
        place.update(device=device, raw=raw)
        assert ops.current_stream_object() == (device, raw)


@pytest.mark.parametrize("heads, kv_heads", [(3, 3), (1, 1), (4, 2), (6, 3)])
def test_the_delta_rules_projection_has_whole_groups_of_16_bytes(heads, kv_heads):
    """An odd number of heads leaves the logits of beta and decay off a multiple of four columns: zero rows make up for it,
    so that the FP32 projection of a layer by itself can take the blocks of four tokens."""
    import torch
    from nanoinfer_b200.config import MixerSpec
    from nanoinfer_b200.parts.recurrent import GatedDeltaRule
    runtime = lambda dtype: SimpleNamespace(dtype=dtype, weight=lambda t: t.to(dtype).contiguous(), gain=lambda t: t.float().contiguous())
    width, d, v = 8, 64, 4
    spec = MixerSpec(kind="gated_delta", num_heads=heads, num_kv_heads=kv_heads, head_dim=d, extra=(("value_dim", v), ("conv_taps", 4)))
    weights = {s: torch.randn(*w.shape) for s, w in GatedDeltaRule.weight_slots(spec, width).items()}
    part = GatedDeltaRule(spec, width, weights, runtime(torch.bfloat16))
    cols = part.b_col + 2 * heads
    assert part.in_blocks and part.w_in.shape[0] == cols + -cols % 4
    assert torch.equal(part.w_in[cols - heads:cols], weights["a"].to(torch.bfloat16)) and not bool(part.w_in[cols:].any())
    state = torch.zeros(1, part.cache_need().shape[0])
    assert ops.delta_block_takes(torch.zeros(2, part.w_in.shape[0]), 0, state)
    plain = GatedDeltaRule(spec, width, weights, runtime(torch.float32))
    assert not plain.in_blocks and plain.w_in.shape[0] == cols


@pytest.mark.parametrize("heads, dim, lens, blocks", [
    (16, 128, [8], False), (16, 128, [24], False), (16, 128, [64], True), (16, 128, [8] + [1] * 8, False), (16, 128, [32] + [1] * 32, False),
    (16, 128, [64] + [1] * 64, False), (16, 128, [256] + [1] * 64, True), (16, 128, [256] + [1] * 200, False), (16, 128, [1024] + [1] * 200, True),
    (16, 128, [8] * 8, False), (16, 128, [16] * 32, True), (8, 64, [8] + [1] * 200, False), (8, 64, [256] + [1] * 200, True),
    (8, 64, [16] * 16, False), (8, 256, [16], False), (8, 256, [16] * 8, True), (8, 256, [128] + [1] * 64, True), (8, 256, [64] + [1] * 200, False),
    (16, 128, [1201, 847], True), (16, 128, [2048], True)])
def test_the_delta_rule_goes_by_blocks_where_they_are_done_first(heads, dim, lens, blocks):
    """Points of the measured table on both sides of the line: short portions and steps of mostly single tokens token by token."""
    assert ops.delta_block_pays(sum(lens), len(lens), max(lens), heads, dim, dim) == blocks


def test_each_path_loads_the_libraries_that_it_launches():
    """The FP32 attention kernels belong to float32 models: a bfloat16 one neither builds nor loads them, and the other way round."""
    from nanoinfer_b200.engine.step import kernel_libraries
    from nanoinfer_b200.parts.mixer import PagedAttention
    part = object.__new__(PagedAttention)
    part.kernel_modules = ("pointwise",)
    f32, bf16 = kernel_libraries([part, None], False), kernel_libraries([part, None], True)
    assert {"attention_generic", "rope_kv", "pointwise"} <= f32 & bf16
    assert "attention_f32" in f32 and "attention_f32" not in bf16
    assert "attention_decode" in bf16 and "attention_decode" not in f32


@pytest.mark.parametrize("cluster", [False, True])
def test_blocks_that_only_ask_for_weights_hold_nobody_up(cluster):
    """The decode attention's blocks go out item first, then kv head, then split.  Beside several splits, whose merge may leave
    an SM room for one block, those without a token are further splits: all of them come behind all that have one, in whole
    clusters.  Beside one split they are further items, and three blocks per SM hold all there are."""
    extra = ops.load("attention_decode").ni_attention_decode_extra
    sms, some = 148, 0
    for items, n_kv, splits in itertools.product([1, 2, 3, 8, 19], [1, 2, 8], range(1, 17)):
        if cluster and splits < 2:
            continue
        more = extra(items, n_kv, splits, cluster, 1 << 20, sms)
        assert extra(items, n_kv, splits, cluster, 0, sms) == 0
        own = items * n_kv * splits
        if 2 * own > sms:
            assert more == 0
            continue
        assert more > 0
        some += 1
        if splits == 1:
            assert (items + more) * n_kv <= 3 * sms < (items + more + 1) * n_kv
            continue
        number = lambda x, y, z: (z * n_kv + y) * items + x
        assert more % (splits if cluster else 1) == 0
        assert number(items - 1, n_kv - 1, splits - 1) == own - 1 and number(0, 0, splits) == own
        assert items * n_kv * (splits + more) <= 3 * sms < items * n_kv * (splits + more + (splits if cluster else 1))
    assert some > 20


@pytest.mark.parametrize("dim, vdim, lens, tiles", [
    (128, 128, [64], False), (128, 128, [32] * 4, False), (128, 128, [100] * 3, True), (128, 128, [16] * 32, True), (128, 128, [8] * 16, False),
    (128, 128, [256] + [1] * 64, False), (128, 128, [512] + [1] * 200, False), (128, 128, [1201, 847], True), (128, 48, [300], True),
    (128, 20, [300], False), (64, 128, [300], False), (256, 128, [300], False)])
def test_the_delta_rule_goes_by_tiles_where_they_are_done_first(dim, vdim, lens, tiles):
    assert ops.delta_tile_pays(sum(lens), len(lens), dim, vdim) == tiles
    assert ops.delta_tile_pays(sum(lens), len(lens), dim, vdim, 16, max(lens)) == tiles


@pytest.mark.parametrize("heads, lens, tiles", [
    (4, [32] * 8, False), (4, [16] * 32, False), (4, [100] * 3, True), (4, [256] + [1] * 15, True), (4, [128] * 8, True), (8, [16] * 16, False), (8, [16] * 32, True),
    (16, [32] * 8, True), (32, [256] + [1] * 15, True), (32, [1024] + [1] * 63, True), (64, [256] + [1] * 15, False), (64, [512] + [1] * 31, False),
    (64, [1024] + [1] * 63, False), (64, [16] * 16, True), (64, [512] * 8, True), (64, [2048], True)])
def test_tiles_are_weighed_with_the_heads_and_the_longest_portion(heads, lens, tiles):
    assert ops.delta_tile_pays(sum(lens), len(lens), 128, 128, heads, max(lens)) == tiles


def test_only_constant_weights_are_read_ahead_of_the_kernel_in_front(monkeypatch):
    """A product by itself takes any w, the work of the kernel in front included; the runtime's weights are constant."""
    import torch

    from nanoinfer_b200.engine.runtime import Runtime
    asked = []
    monkeypatch.setattr(ops, "load", lambda module: SimpleNamespace(ni_gemm_f32_tc=lambda *a: asked.append(a[10]) or 0))
    monkeypatch.setattr(ops, "_dev", lambda t, name, dtype=None: t.data_ptr())
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "_error_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ops, "_heads_of", lambda x, w, out, what: (x.data_ptr(), x.stride(0), w.data_ptr(), out.data_ptr(), 3, 8, 1024, 2))
    x, w, out = torch.zeros(3, 1024), torch.zeros(8, 1024), torch.zeros(3, 8)
    ops.linear_f32(x, w, out)
    ops.linear_f32(torch.zeros(3, 2048), torch.zeros(2, 8, 1024), torch.zeros(3, 16))
    ops.gemm_f32_tc(x, w, out)
    assert asked == [0, 0, 0]
    rt = object.__new__(Runtime)
    rt.dtype, rt.device = torch.float32, torch.device("cpu")
    rt.linear(x, w)
    rt.heads_linear(torch.zeros(3, 2048), torch.zeros(2, 8, 1024))
    assert asked[3:] == [1, 1]
