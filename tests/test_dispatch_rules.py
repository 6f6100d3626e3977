"""Rules that choose between kernels, on the CPU: they need only sizes."""
import random
from types import SimpleNamespace

import pytest
import torch

from oxidize_b200.ops import attn_plan
from oxidize_b200.ops import cuda as C
from oxidize_b200.ops import cuda_quant


@pytest.mark.parametrize("qtype,n,k,tokens,once", [
    # either side of the line, as measured: fused / decoded once, us
    ("Q6_K", 28672, 4096, 1025, False),  # 330 / 341
    ("Q6_K", 28672, 4096, 1500, True),  # 408 / 404
    ("Q6_K", 8192, 8192, 1025, True),  # 217 / 212
    ("Q6_K", 4096, 14336, 1025, False),  # 186 / 222
    ("Q6_K", 4096, 4096, 2048, True),  # 90 / 81
    ("Q6_K", 1024, 4096, 1500, False),  # 39 / 54
    ("Q8_0", 28672, 4096, 2048, False),  # 461 / 497
    ("Q8_0", 4096, 4096, 2048, False),  # 80 / 81
    ("Q8_0", 4096, 4096, 3000, True),  # 117 / 110
    ("Q8_0", 6144, 4096, 3000, True),  # 153 / 148
    ("Q8_0", 512, 512, 4096, False),  # 16 / 21
    ("Q4_K", 4096, 4096, 4096, False), ("NVFP4", 28672, 4096, 4096, False),
    ("Q4_0", 4096, 4096, 1025, True), ("Q4_0", 4096, 4096, 1024, False)])
def test_packed_matrices_are_decoded_once_where_that_is_faster(qtype, n, k, tokens, once):
    assert cuda_quant.decode_once(qtype, True, tokens, n, k, 148) == once


@pytest.mark.parametrize("qtype", ["Q4_K", "Q6_K", "Q8_0", "NVFP4", "Q4_0"])
def test_rows_that_are_not_staged_are_decoded_once(qtype):
    """Q6_K rows of 1536 values (1260 bytes) at 1025 tokens: 102 us fused, 30 decoded once."""
    assert cuda_quant.decode_once(qtype, False, 1025, 2048, 1536, 148)
    assert not cuda_quant.decode_once(qtype, False, 1024, 2048, 1536, 148)


def test_a_limit_that_was_set_is_kept(monkeypatch):
    monkeypatch.setattr(C, "mmq_max_tokens", 8)
    assert cuda_quant.decode_once("Q4_K", True, 9, 512, 512, 148) and not cuda_quant.decode_once("Q6_K", False, 8, 512, 512, 148)
    monkeypatch.setattr(C, "mmq_max_tokens", 0)
    assert not cuda_quant.decode_once("Q6_K", False, 4096, 512, 512, 148)


# ------------------------------------------------------------------------------------- attention of long portions
def _choose(lens, heads, pages="bf16", window=0, **more):
    return attn_plan.choose(lens, *heads, pages, window, 148, **more)


FEW, SMALL, MANY = (8, 1, 128), (8, 2, 64), (32, 8, 128)


@pytest.mark.parametrize("lens,heads,pages,window,take", [
    # measured, us: the tcgen05 kernel / the mma.sync one
    ([(256, 8000)], FEW, "bf16", 0, []),  # 168 / 86: eight CTAs, as 64 rows of 32 heads are
    ([(256, 32000)], FEW, "bf16", 0, []),  # 635 / 279
    ([(1024, 8000)], FEW, "bf16", 0, [0]),  # 172 / 279
    ([(512, 8000)], SMALL, "bf16", 0, []),  # 168 / 119
    ([(2048, 8000)], SMALL, "bf16", 0, [0]),  # 174 / 266
    ([(64, 8000)], MANY, "bf16", 0, []),  # 168 / 86
    ([(64, 8000)] * 4, MANY, "bf16", 0, [0, 1, 2, 3]),  # 172 / 276
    ([(256, 8000)], MANY, "bf16", 0, [0]),  # 174 / 272
    ([(33, 33)] * 32, MANY, "bf16", 0, []), ([(140, 140), (83, 83)], MANY, "q4", 0, []),  # short ones, over no long context
    ([(161, 161), (146, 146), (122, 122)], (64, 8, 128), "q4", 0, [0, 1, 2]),
    ([(256, 8000)], FEW, "bf16", 1024, []),  # 33 / 27
    ([(256, 8000)], MANY, "bf16", 1024, [0]),  # 35 / 57
    ([(256, 8000)], FEW, "q8", 0, []),  # 169 / 119, conversion of the pages included
    ([(256, 8000)], FEW, "f16", 0, []),  # 171 / 154
    ([(512, 8000)], FEW, "f16", 0, [0]),  # 171 / 285
    # the tail of a long prompt next to a whole one, and among decoding sequences
    ([(500, 500), (40, 12000)], MANY, "bf16", 0, [0]),
    ([(40, 12000), (500, 500)], MANY, "q4", 0, [1]),
    ([(512, 4096)] + [(1, 1000)] * 63, MANY, "q8", 0, [0]),
    ([(1, 500)] * 8, MANY, "bf16", 0, []), ([(31, 500)], MANY, "bf16", 0, []), ([(300, 200)], MANY, "bf16", 0, []),
    ([(0, 40), (512, 512), (0, 0)], MANY, "bf16", 0, [1])])
def test_sequences_for_the_tcgen05_attention(lens, heads, pages, window, take):
    assert _choose(lens, heads, pages, window) == take


def test_a_step_chooses_by_sequence_not_by_order():
    gen = random.Random(3)
    lens = [(500, 500), (40, 12000), (300, 900), (64, 64), (1, 3000), (700, 900)]
    want = {lens[i] for i in _choose(lens, MANY, "q8")}
    assert (700, 900) in want and (40, 12000) not in want
    for _ in range(5):
        gen.shuffle(lens)
        assert {lens[i] for i in _choose(lens, MANY, "q8")} == want


def test_converted_pages_stay_within_their_bytes():
    lens, heads = [(512, 32000), (512, 30000), (600, 1000)], (32, 32, 128)
    page = 32 * 64 * 128
    need = lambda take: sum(attn_plan.pages_seen(*lens[i], 0) for i in take) * page  # noqa: E731
    assert _choose(lens, heads, "q8", most_bytes=1 << 40) == [0, 1, 2]
    few = _choose(lens, heads, "q8")
    assert need([0, 1, 2]) > attn_plan.MAX_PAGES_BYTES >= need(few) and 2 in few and len(few) == 2
    assert _choose(lens, heads, "q8", most_bytes=0) == [] and _choose(lens, heads, "bf16", most_bytes=0) == [0, 1, 2]
    # a window's pages count, not the context's
    assert _choose([(512, 128000)], heads, "q8", 4096) == [0] and attn_plan.pages_seen(512, 128000, 4096) == 288


def test_more_sequences_than_the_mask_has_bits():
    assert _choose([(512, 512)] * (attn_plan.MAX_SEQS + 1), MANY) == []


def test_a_server_leaves_room_for_converted_pages(monkeypatch):
    from oxidize_b200.engine.kv_pool import KVCacheSpec
    from oxidize_b200.engine.llm import LLM, EngineConfig

    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *_: (100 << 30, 180 << 30))
    blocks = {}
    for pages in ("bf16", "q8"):
        spec = KVCacheSpec(80, 8, 128, 16, pages)
        config = EngineConfig(max_model_len=131072, max_num_seqs=256, gpu_memory_utilization=0.99)
        one = SimpleNamespace(config=config, device=torch.device("cuda"), cfg=SimpleNamespace(state_shapes=[], state_windows=[]))
        blocks[pages] = LLM._auto_blocks(one, spec), spec.bytes_per_block()
    free = int((100 - 0.01 * 180) * (1 << 30))
    assert abs(blocks["bf16"][0] * blocks["bf16"][1] - free) < blocks["bf16"][1]
    left = free - blocks["q8"][0] * blocks["q8"][1]
    assert 0 <= left - attn_plan.MAX_PAGES_BYTES < blocks["q8"][1]
    # no more than the longest sequences could take, and nothing for pages that are read as they are
    assert attn_plan.reserve_bytes(KVCacheSpec(2, 2, 64, 16, "q4"), 100, 3) == 2 * 64 * 64 * 7 * 3
    assert attn_plan.reserve_bytes(KVCacheSpec(2, 2, 64, 16, "bf16"), 100, 3) == attn_plan.reserve_bytes(KVCacheSpec(2, 2, 96, 16, "q4"), 100, 3) == 0
