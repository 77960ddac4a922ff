"""Host-side choices of how a product is cut into blocks (no GPU needed)."""

import os
import re

import pytest
import torch

from enginekernel_b200.ops import build, kernels
from enginekernel_b200.parts.base import Workspace


@pytest.mark.parametrize("n_out,k,epi", [
    (6144, 2560, kernels.EPI_BF16), (2560, 4096, kernels.EPI_BF16), (9728, 2560, kernels.EPI_SWIGLU),
    (2560, 9728, kernels.EPI_BF16), (151936, 2560, kernels.EPI_F32), (1024, 1024, kernels.EPI_BF16),
    (4096, 12288, kernels.EPI_BF16), (128, 64, kernels.EPI_BF16), (20011, 2560, kernels.EPI_F32),
])
def test_k_split_of_the_swapped_form(n_out, k, epi):
    split = kernels.swap_k_split(n_out, k, epi)
    tiles = -(-n_out // (64 if epi == kernels.EPI_SWIGLU else 128))
    k_blocks = -(-k // 64)
    assert 1 <= split <= kernels.TC_MAX_CLUSTER
    assert split & (split - 1) == 0                        # clusters of 3, 5, 6, 7 blocks run slowly
    assert split == 1 or tiles * split <= 2 * kernels.sm_count()      # one filling of the machine
    assert split == 1 or k_blocks // split >= 8            # a block keeps a ring's worth of K


@pytest.mark.parametrize("n_out,k,split", [(4096, 1024, 4), (1024, 2048, 8), (2560, 4096, 8), (6144, 2560, 4), (4160, 2048, 4),
                                           (3072, 768, 2), (128, 64, 1), (151936, 2560, 1)])
def test_k_split_of_narrow_products(n_out, k, split):
    assert kernels.narrow_k_split(n_out, k, kernels.EPI_BF16) == split
    tiles, most = -(-n_out // 128), kernels.swap_k_split(n_out, k, kernels.EPI_BF16)
    assert split == most or (tiles * split <= 1.1 * kernels.sm_count() and -(-k // 64) // split >= 4)


def test_the_benchmark_shape_gets_the_splits_the_profiles_name():
    assert kernels.swap_k_split(6144, 2560, kernels.EPI_BF16) == 4      # q/k/v
    assert kernels.swap_k_split(2560, 4096, kernels.EPI_BF16) == 8      # attention output
    assert kernels.swap_k_split(9728, 2560, kernels.EPI_SWIGLU) == 1    # gate/up
    assert kernels.swap_k_split(2560, 9728, kernels.EPI_BF16) == 8      # down


def test_short_prompts_of_general_layers_make_no_table_of_tiles():
    """The rule at its line: several sequences, and more than two and a half fillings of the machine with two blocks an SM."""
    sms = kernels.sm_count()
    pays = lambda tokens, seqs: kernels.attention_prefill_tiles_pay(tokens, seqs, 16, 8)      # 64 tokens a tile, 8 key heads
    line = 5 * sms // 8 + 1                                 # tiles (of 8 blocks each) from which it pays
    assert not pays(9, 1) and not pays(36, 8) and not pays(512, 3) and not pays(64 * (line - 3), 2)
    assert pays(64 * (line - 2), 2) and pays(64 * line, 8) and not pays(1 << 20, 1)


@pytest.mark.parametrize("dim,lane_columns", [(20, 2), (32, 2), (33, 4), (128, 4)])
def test_segments_are_planned_with_the_columns_that_the_scan_takes(dim, lane_columns, monkeypatch):
    """64 columns: keys of up to 32 values are walked two columns a lane, wider ones four; the scan is cut for the blocks
    that it launches, and its launch gets the same number."""
    assert kernels.decay_scan_lane_columns(64, 2048, dim) == lane_columns
    blocks = 64 * 64 // (kernels.SCAN_COLUMNS * lane_columns)
    want = min(kernels.SCAN_BLOCKS_PER_SM * kernels.sm_count() // blocks, 2048 // kernels.SCAN_MIN_SEGMENT)
    length = -(-(-(-2048 // want)) // 64) * 64
    plan = (-(-2048 // length), length)
    assert kernels.decay_scan_segments(1, 64, 64, 2048, lane_columns=lane_columns) == plan
    launched = []
    monkeypatch.setattr(kernels, "_need_cuda", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_decay_scan", lambda *args: launched.append(args))
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    rows = kernels.decay_scan_rows(dim)
    f32, i32 = (lambda *s: torch.zeros(*s)), (lambda n: torch.zeros(n, dtype=torch.int32))
    kernels.decay_scan(f32(2048, 64 * 64), f32(2048, dim), f32(2048, dim), f32(2048, 64 * 64), f32(2048, 64),
                       f32(2048, 64), f32(1, 64 * 64 * rows), i32(2), i32(2048), i32(2048), 1, 64, 1, dim, 64, n_tokens=2048,
                       max_new=2048, workspace=Workspace(torch.device("cpu")))
    assert launched[0][-4:-1] == (*plan, lane_columns)


@pytest.mark.parametrize("name,source,constant", [
    ("DELTA_CHUNK", "delta_chunk.cu", "kChunk"), ("MOE_TILE_ROWS", "moe.cu", "kTileRows"),
    ("MOE_PAIR_TILE_ROWS", "moe_pair.cu", "kMoeTile"), ("MOE_PAIR_EVEN", "moe_pair.cu", "kMoeEven"),
    ("PREFILL_F32_ROWS", "attention_prefill_f32.cu", "kF32Rows"), ("PREFILL_TC_ROWS", "attention_prefill_tc.cu", "kFaRows"),
    ("SCAN_COLUMNS", "recurrent.cu", "kScanCols")])
def test_sizes_that_host_and_kernels_share(name, source, constant):
    """What the host sizes grids and scratch by is what the kernels are built with."""
    with open(os.path.join(build.CSRC, source)) as f:
        (value,) = re.findall(rf"constexpr int {constant} = (\d+)", f.read())
    assert getattr(kernels, name) == int(value)


@pytest.mark.parametrize("inter,gated", [(20, True), (20, False), (9, True), (24, True)])
def test_experts_of_any_size_run_on_pairs_of_sms(inter, gated):
    """bfloat16 experts whose size is no whole number of 16-byte pieces: laid out so that both products take the form on
    pairs of SMs, with zeros behind the last value; in 32-bit as they are."""
    from enginekernel_b200.parts.spec import PartSpec
    from enginekernel_b200.registry import lookup_part
    h, n = 32, 3
    g = torch.Generator().manual_seed(1)
    w = {"router": torch.randn(n, h, generator=g)}
    for e in range(n):
        w.update({f"gate_{e}": torch.randn(inter, h, generator=g), f"up_{e}": torch.randn(inter, h, generator=g),
                  f"down_{e}": torch.randn(h, inter, generator=g)})
    params = dict(hidden_size=h, intermediate_size=inter, experts=n, top=2, activation="silu", gated=gated)
    for dtype in (torch.bfloat16, torch.float32):
        part = lookup_part("feed_forward", "routed_experts")(PartSpec("routed_experts", params, {k: k for k in w}), dtype, "cpu")
        part.load(w)
        if dtype == torch.bfloat16:
            assert kernels.moe_on_pairs(torch.zeros(5, h, dtype=dtype), part.w_up, part.w_down)
        for e in range(n):
            rows = part.w_up[e, :2 * inter].view(inter, 2, h) if gated else part.w_up[e, :inter].view(inter, 1, h)
            assert torch.equal(rows[:, -1], w[f"up_{e}"].to(dtype)) and torch.equal(rows[:, 0], w[f"gate_{e}" if gated else f"up_{e}"].to(dtype))
            assert torch.equal(part.w_down[e, :, :inter], w[f"down_{e}"].to(dtype))
        assert not part.w_up[:, (2 if gated else 1) * inter:].any() and not part.w_down[:, :, inter:].any()


def test_the_delta_rule_goes_by_chunks_from_96_tokens_a_sequence():
    by = kernels.delta_by_chunks
    assert by(96, 1, 128, 128) and not by(95, 1, 128, 128) and by(4 * 96, 4, 64, 4) and not by(4 * 96 - 1, 4, 64, 4)
    assert by(500, 1, 64, 128) and not by(500, 1, 64, 132) and not by(500, 1, 128, 130)      # values up to twice the keys, whole fours
    assert not by(500, 1, 32, 32) and not by(500, 1, 256, 128) and not by(1, 1, 128, 128)    # keys of 64 and 128


def test_where_32_bit_prompt_attention_takes_blocks_of_64_tokens():
    """From two pages of keys and 1,024 (token, head) rows a round of blocks, two an SM, on; never beyond what its grid holds."""
    sms = kernels.sm_count()
    wins = lambda tokens, seqs, heads, visible: kernels.attention_prefill_f32_wins(tokens, seqs, heads, visible, None)
    assert wins(64, 1, 16, 128) and not wins(64, 1, 16, 127) and not wins(63, 1, 16, 128)
    heads = 2 * sms // 2                                       # two blocks a head (64 tokens, one sequence): one round
    assert wins(64, 1, heads, 128)
    assert (64 * (heads + 1) >= 2 * kernels.PREFILL_F32_ROUND) == wins(64, 1, heads + 1, 128)     # a second round for one head
    assert wins(64 * 65534, 1, 16, 10**6) and not wins(64 * 65535, 1, 16, 10**6)


def test_launch_record_groups_costs_and_issues_again():
    """The record behind the per-kernel tables, without a GPU: entries keep their order, are named
    with their label, sum their costs by name, and are issued again by name."""
    from enginekernel_b200.ops import lib
    issued = []
    with lib.LaunchRecord() as rec:
        assert lib.recording()
        lib.record_library_call("library_matmul[8x4]", lambda: issued.append("a"), bytes=100, flops=64)
        lib.record_library_call("library_matmul[2x4]", lambda: issued.append("b"), bytes=10, flops=16)
        lib.record_library_call("library_matmul[8x4]", lambda: issued.append("c"), bytes=100, flops=64)
        with pytest.raises(RuntimeError):
            lib.LaunchRecord().__enter__()                 # one record at a time
    assert not lib.recording()
    lib.record_library_call("late", lambda: issued.append("x"))        # nothing is active: not kept
    assert rec.names() == ["library_matmul[8x4]", "library_matmul[2x4]"]
    assert rec.cost("library_matmul[8x4]") == {"bytes": 200, "flops": 128, "launches": 2}
    assert rec.cost() == {"bytes": 210, "flops": 144, "launches": 3}
    assert rec.issue(0, "library_matmul[8x4]") == 2 and issued == ["a", "c"]
    assert rec.issue(0) == 3 and issued == ["a", "c", "a", "b", "c"]
