"""The host core without a device: every kernel launcher it names exists in the
kernel library it names, and its C interface answers for configuration, plans
and registries (no GPU)."""
import ctypes
import json
import os
import re

import pytest

from kipp_b200 import native as N
from kipp_b200.csrc import build
from tiny import TINY_A, TINY_B

HOST = os.path.join(os.path.dirname(os.path.abspath(build.__file__)), "host")


def test_every_launcher_the_host_core_names_exists():
    src = open(os.path.join(HOST, "kernels.hpp")).read()
    named = re.findall(r'kernel_symbol<\w+>\("(\w+)", "(\w+)"\)', src)
    assert len(named) >= 15
    for library, symbol in named:
        lib = ctypes.CDLL(build.compile_library(library, verbose=False))
        assert hasattr(lib, symbol), f"lib{library}.so lacks {symbol}"


def test_registries_and_plans():
    lib = N.lib()
    reg = json.loads(lib.kipp_registered().decode())
    assert "Qwen3ForCausalLM" in reg["architectures"]
    assert {"attention", "swiglu", "rmsnorm", "rotary", "token_embedding", "output_head", "pre_norm_block",
            "external", "frequency_table", "no_position"} <= set(reg["part_kinds"])
    plan = json.loads(N.text_result(lib.kipp_plan_from_config, json.dumps(TINY_B).encode()))
    assert len(plan["layers"]) == 3 and plan["head"]["part"]["tied_to"] is None
    mixer = plan["layers"][1]["part"]["mixer"]
    assert (mixer["num_heads"], mixer["num_kv_heads"], mixer["head_dim"]) == (8, 1, 32)
    assert mixer["position"] == {"kind": "rotary", "head_dim": 32, "theta": 1000000.0}
    tied = json.loads(N.text_result(lib.kipp_plan_from_config, json.dumps(TINY_A).encode()))
    assert tied["head"]["part"]["tied_to"] == "model.embed_tokens.weight"
    # a plan with a part kind nobody registered is refused by name
    plan["layers"][0]["part"]["ffn"]["kind"] = "gelu_mlp"
    with pytest.raises(ValueError, match="unknown part kind 'gelu_mlp'"):
        N.text_result(lib.kipp_plan_tensor_specs, json.dumps(plan).encode())


def test_split_rule_of_the_decode_attention():
    lib = N.lib()
    # few (token, kv head) pairs: many short splits; many pairs: few long ones
    few, many = lib.kipp_attention_split_length(1, 2048, 8, 148, 0), lib.kipp_attention_split_length(64, 2048, 8, 148, 0)
    assert few == 64 and many >= 512 and many % 64 == 0        # one token: one tile per split (latency)
    assert lib.kipp_attention_split_length(1, 100, 8, 148, 0) == 64
    assert lib.kipp_attention_split_length(8, 2048, 8, 148, 0) == 384      # 6 splits: 384 CTAs, one wave
    # from the token's own context: an eighth of it, in whole 64-key tiles, at least one tile
    assert lib.kipp_attention_split_length(1, 8192, 8, 148, 1) == 1024
    assert lib.kipp_attention_split_length(1, 700, 8, 148, 1) == 128
    assert lib.kipp_attention_split_length(1, 300, 8, 148, 1) == 64
    assert lib.kipp_attention_split_length(1, 2049, 8, 148, 1) == 320
    # dealt out as a stream where splits of one length would need several waves or leave one half empty
    def stream(n, keys):
        arr = (ctypes.c_int * n)(*([keys] * n))
        return lib.kipp_attention_stream_pays(n, arr, 8, 148)
    assert [stream(n, 2049) for n in (1, 8, 16, 64)] == [0, 0, 0, 1]      # 512 pairs on 444 places: four waves of splits
    assert stream(8, 8031) == 0 and stream(64, 4097) == 1


def test_a_cluster_has_a_place_for_every_split():
    """Where a token's splits are a cluster, no length that the block tables have room for is planned as more splits than it has
    CTAs: a captured step, whose tables are rounded up, then cuts its tokens as a plain launch does."""
    lib = N.lib()
    taken = 0
    for kv_heads in (1, 2, 4, 5, 8, 16):
        for n in (*range(1, 70), 100, 128):
            most = {}
            for room in (64, 112, 320, 640, 960, 1008, 1024, 2048, 3072, 4096):
                ctas = lib.kipp_attention_cluster_splits(n, (ctypes.c_int * n)(*[1] * n), kv_heads, 148, room)
                assert 0 <= ctas <= 4
                if ctas == 0:
                    continue
                taken += 1
                for tiles in range(1, -(-room // 64) + 1):
                    if tiles not in most:
                        keys = lib.kipp_attention_split_length(n, 64 * tiles, kv_heads, 148, 0)
                        most[tiles] = -(-64 * tiles // keys)
                    assert most[tiles] <= ctas, (kv_heads, n, room, tiles)
    assert taken > 500
    tokens = lambda n, keys: (n, (ctypes.c_int * n)(*[keys] * n))                    # noqa: E731
    assert lib.kipp_attention_cluster_splits(*tokens(16, 1000), 8, 148, 1024) == 3
    assert lib.kipp_attention_cluster_splits(*tokens(11, 1000), 8, 148, 1024) == 0   # 900 keys are planned as five splits


def test_a_clusters_ctas_fit_an_sm_as_they_are_counted():
    """The planner's waves hold three CTAs an SM; a kernel whose shared memory leaves room for two is not taken."""
    fits = build.load_library("attention_mma").kipp_attn_decode_cluster_fits
    assert all(fits(64, group, 1, ctas) for group in (1, 4, 16) for ctas in (1, 2, 3, 4, 8))
    assert all(fits(128, 8 * group, 8, ctas) for group in (1, 4, 8, 12) for ctas in (1, 2, 3, 4))
    assert not any(fits(128, group, 1, ctas) for group in (14, 16) for ctas in (1, 2, 3, 4))
    assert not fits(128, 17, 1, 4) and not fits(96, 4, 1, 4) and not fits(128, 8, 1, 9) and not fits(128, 8, 1, 0)


def test_state_space_scans_count_the_work_that_lasts():
    """The scan's form follows the blocks that last as long as the longest entry: one long prompt beside many single
    tokens is scanned as the prompt alone, entries alike as all of them."""
    leaves = build.load_library("recurrent").kipp_ssd_scan_leaves
    for dim, heads in ((128, 64), (128, 80), (64, 32), (256, 24), (32, 100)):
        alone = leaves(dim, 64, heads, 1, 2000, 2000)
        assert alone == 1
        for others in (1, 7, 31, 200):
            assert leaves(dim, 64, heads, 1 + others, 2000 + others, 2000) == alone
        assert leaves(dim, 64, heads, 64, 64 * 100, 100) == leaves(dim, 64, heads, 64, 64 * 100, 0) == 2


def test_rows_with_a_top_k_are_sampled_without_histograms_by_lane():
    """Only rows that may weigh a long part need them: not where every row's top-k fits the list."""
    by_lane = build.load_library("sampling").kipp_sample_rows_by_lane
    for rows, n in ((1, 151936), (64, 151936), (148, 151936), (128, 32000), (8, 10000)):
        assert by_lane(rows, n, 0) == by_lane(rows, n, 4097) == 1
        assert by_lane(rows, n, 1) == by_lane(rows, n, 50) == by_lane(rows, n, 4096) == 0
    assert by_lane(4, 8000, 0) == 0
