"""Rules that choose between kernels, on the CPU: they need only sizes."""
import pytest

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
