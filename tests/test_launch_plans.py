"""The choices made on the host before a launch (splits of decode attention, splits and occupancy of
the tcgen05 product) as pure functions: bounds that the kernels rely on, for any sizes."""

import random

from acorninfer_b200.kernels.attention import decode_splits
from acorninfer_b200.kernels.ops import gemm_tc_plan, gemm_tc_splits


def test_decode_splits_stay_within_what_the_kernels_take():
    rng = random.Random(0)
    for _ in range(2000):
        rows, nkv = rng.randint(1, 4096), rng.choice([1, 2, 3, 4, 5, 8, 16, 32])
        bound = rng.choice([1, 16, 63, 64, 65, 1000, 4096, 40000, 1 << 20])
        s = decode_splits(rows, nkv, bound, rng.choice([16, 64, 128, 256]))
        assert 1 <= s <= 32
        assert s <= max(1, -(-bound // 64))          # never more splits than chunks of 64 keys


def test_decode_splits_follow_the_measured_cases():
    # few pairs: many CTAs in flight; a count just above a multiple of 296: shorter CTAs; a well
    # filled last wave: no split
    assert decode_splits(1, 8, 4096, 128) >= 16
    assert decode_splits(8, 8, 4096, 128) == 4
    assert decode_splits(32, 8, 4096, 128) == 1 and decode_splits(64, 8, 4096, 128) == 1 and decode_splits(96, 8, 4096, 128) == 1
    assert decode_splits(40, 8, 4096, 128) > 1 and decode_splits(20, 8, 4096, 128) > 1 and decode_splits(80, 8, 4096, 128) > 1
    assert decode_splits(8, 8, 48, 128) == 1              # a single chunk cannot be split
    # the estimate is in bytes: a smaller head size makes a pair's keys cheaper, which never asks for more splits
    assert decode_splits(8, 8, 4096, 32) <= decode_splits(8, 8, 4096, 128)


def test_decode_plans_of_the_tma_kernel():
    """One wave of clusters or none up to 2,048 keys, several waves of longer rows; the measured cases; what the kernels take."""
    from acorninfer_b200.kernels.attention import decode_plan
    want = {1: 16, 2: 8, 3: 8, 5: 6, 6: 5, 7: 4, 8: 4, 9: 3, 10: 3, 11: 2, 12: 2, 16: 2, 19: 1, 32: 1, 37: 1, 41: 1, 64: 1}
    assert {r: decode_plan(r, 8, 2048) for r in want} == want
    assert decode_plan(1, 8, 48) == 1 and decode_plan(1, 1, 1 << 20) == 32
    rng = random.Random(2)
    for _ in range(2000):
        rows, nkv, bound = rng.randint(1, 4096), rng.choice([1, 2, 3, 5, 8, 16, 32]), rng.choice([1, 63, 64, 65, 1000, 4096, 40000, 1 << 20])
        limit = rng.choice([2, 8, 16])
        s = decode_plan(rows, nkv, bound, 148, limit)
        assert 1 <= s <= 32 and s <= max(1, -(-bound // 64))
        assert s == 1 or rows * nkv * s <= 296 or (bound > 2048 and rows * nkv > 148 and s <= min(limit, 8))
    # rows beyond a wave, and rows whose second split does not fit one, at long contexts: the last wave of whole rows takes longer
    assert decode_plan(64, 8, 4096) == 1 and decode_plan(37, 8, 16384) == 1 and decode_plan(40, 8, 2048) == 1
    for rows in (38, 40, 44, 48, 76, 80):
        assert all(decode_plan(rows, 8, bound) > 1 for bound in (4096, 8192, 16384)), rows
    assert decode_plan(20, 8, 4096) == 3 and decode_plan(40, 8, 16384, merge_limit=2) == 2


def test_gemm_plans_are_valid_for_any_shape():
    rng = random.Random(1)
    for _ in range(3000):
        M, N, K = rng.randint(1, 300), rng.randint(1, 200000), 8 * rng.randint(1, 4096)
        splits, per_sm = gemm_tc_plan(M, N, K)
        assert splits in (1, 2, 4, 8) and per_sm in (2, 3)
        assert gemm_tc_splits(M, N, K) == splits
        if splits > 1:
            assert -(-K // 64) // splits >= 4        # every split keeps at least four steps of K
        if per_sm == 3:
            assert M <= 64 and splits == 2       # three short rings to an SM: tiles of up to 64 tokens
        if M > 64:
            assert per_sm == 2


def test_gemm_plans_of_the_decode_shapes():
    # Qwen3-8B layer sizes at 8 rows: qkv, o, gate_up, down, output matrix
    assert gemm_tc_plan(8, 6144, 4096) == (4, 2)
    assert gemm_tc_plan(8, 4096, 4096) == (8, 2)
    assert gemm_tc_plan(8, 24576, 4096) == (2, 3)    # 192 tiles on 148 SMs: half tiles, three CTAs to an SM
    assert gemm_tc_plan(8, 4096, 12288) == (8, 2)
    assert gemm_tc_plan(8, 151936, 4096) == (1, 2)


def test_paired_kernel_is_asked_for_where_its_tiles_fill_the_device():
    """256 x 256 tiles in rounds of one tile to a pair of SMs: 74 pairs on 148 SMs."""
    from acorninfer_b200.kernels.ops import fused_rows_ok, pair_rows_ok
    import torch
    assert pair_rows_ok(2048, 4096)            # 128 tiles: two rounds, 0.86 full
    assert not pair_rows_ok(1536, 4096)        # 96 tiles: two rounds, 0.65 full
    assert not pair_rows_ok(200, 4096)         # below one tile of rows
    assert not pair_rows_ok(2048, 1024, max_rows=8192) and pair_rows_ok(4608, 1024, max_rows=8192)    # a narrow model needs more rows: 32 tiles, 72 tiles on 74 pairs
    assert not pair_rows_ok(1800, 4096)        # eight token tiles, the last one a fifth full: 0.76
    # the widest product taken alone needs less: gate/up of 24,576 columns from about 360 rows on
    assert pair_rows_ok(384, 24576, min_fill=0.6) and not pair_rows_ok(300, 24576, min_fill=0.6)
    assert not pair_rows_ok(257, 24576, min_fill=0.6)     # the second token tile holds one row
    assert pair_rows_ok(3072, 4096) and not pair_rows_ok(4096, 4096)       # the longest steps: not every product (the power cap)
    assert pair_rows_ok(4096, 24576, min_fill=0.6, max_rows=8192) and not pair_rows_ok(12288, 24576, min_fill=0.6, max_rows=8192)
    assert not pair_rows_ok(2048, 1024)        # 32 tiles on 74 pairs
    assert pair_rows_ok(2048, 4096, num_sms=64) == (128 / (4 * 32) >= 0.8)
    # the one-CTA kernel's range is independent of the width; between the two ranges nothing is fused
    assert fused_rows_ok(8, torch.bfloat16) and fused_rows_ok(32, torch.bfloat16, 4096)
    assert not fused_rows_ok(33, torch.bfloat16, 4096) and not fused_rows_ok(1536, torch.bfloat16, 4096)
    assert fused_rows_ok(2048, torch.bfloat16, 4096) and not fused_rows_ok(2048, torch.bfloat16)
    # every product of the part has to fill the device: at 1,024 rows the q/k/v product of 6,144 columns does not
    assert fused_rows_ok(1024, torch.bfloat16, 4096) and not fused_rows_ok(1024, torch.bfloat16, (6144, 4096))
    assert fused_rows_ok(2048, torch.bfloat16, (6144, 4096)) and fused_rows_ok(2048, torch.bfloat16, (24576, 4096))
    assert not fused_rows_ok(2048, torch.float32, 4096)


def test_tile_of_48_rows_is_for_layers_that_fuse_throughout(monkeypatch):
    """33 to 48 rows: gate/up products take the one-CTA kernel's tile between fused neighbours only, layers whose rotation is not in
    the epilogue of their q/k/v product do not ask for it."""
    import torch
    from acorninfer_b200.kernels import ops
    from acorninfer_b200.parts.attention import Attention
    from acorninfer_b200.parts.base import POSITION_ENCODINGS, BuildContext, PartSpec, build_part
    from acorninfer_b200.parts.feed_forward import SwiGLU
    monkeypatch.setattr(ops, "device_sms", lambda device: 148)
    taken = []
    monkeypatch.setattr(ops, "linear", lambda x, w, **kw: taken.append(kw.get("swiglu", False)) or torch.zeros(1, w.shape[0]))
    monkeypatch.setattr(ops, "swiglu", lambda gu, **kw: gu)
    ctx = BuildContext(dtype=torch.bfloat16, device=torch.device("cpu"), page_size=16)
    ff = SwiGLU(ctx, 1024, 64)
    ff.bind({n: torch.zeros(s.shape, dtype=torch.bfloat16) for n, s in ff.tensor_specs().items()})
    x = torch.zeros(40, 1024, dtype=torch.bfloat16)
    for rows, between in ((x, object()), (ops.NormedRows(x, None, 1e-6, 1024), None), (x, None), (x[:32], None)):
        ff.forward(rows, None, epilogue=between)
    assert taken == [True, False, True, False, False, False, True, False]       # of the gate/up and the down product in turn
    for rotary in (128, 64):
        ctx.positions["rope"] = build_part(POSITION_ENCODINGS, PartSpec("rope", {"head_dim": 128, "theta": 1e6, "rotary_dim": rotary}, ""), ctx)
        att = Attention(ctx, hidden_size=1024, num_heads=8, num_kv_heads=2, head_dim=128, position="rope", scale=128 ** -0.5)
        att.bind({n: torch.zeros(s.shape, dtype=torch.bfloat16) for n, s in att.tensor_specs().items()})
        assert att.fusable(40) == (rotary == 128) and att.fusable(32) and not att.fusable(49)
