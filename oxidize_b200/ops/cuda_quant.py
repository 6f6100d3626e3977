"""Linear layers over packed weights (Q4_K / Q6_K / Q8_0 / Q4_0 / NVFP4 GGUF blocks and
block-scaled fp8) on the GPU.

Everything goes through ``oxb_gemm_quant``.  Calls with one or two tokens take the dp4a GEMV
(``csrc/gemv_quant.cuh``: int8 activations, the packed bytes go straight into the arithmetic); larger
batches the tcgen05 GEMM whose producer warps decode the blocks into tensor memory.  Either way the weights are read from HBM once, in their packed form.  Formats without a
fused decoder (Q5_K, Q4_1 …), or a K that is not a multiple of 64, are decoded to a bf16 staging
buffer first.
"""
from __future__ import annotations

import torch

from . import cuda as C

FUSED_TYPES = {"Q4_K": 5, "Q6_K": 7, "Q8_0": 3, "Q4_0": 4, "NVFP4": 8}
QT_FP8B = 9
# Past this many tokens a matrix may be decoded to bf16 once, ahead of a bf16 GEMM, instead of by every token tile.
DECODE_ONCE_ABOVE = 1024
# The fused kernel then loses a few us per wave of tiles of 256 tokens (a tile of 128 takes 0.6 of one), and decoding once costs time per
# weight tile: fused while its waves, times SMs, are at most this many per weight tile.  us fused / decoded once: Q6_K 28672 x 4096
# at 1025 tokens (5.3) 330 / 341, at 1500 (6.6) 408 / 404; 8192 x 8192 at 1025 (6.9) 217 / 212; 4096 x 4096 at 2048 (9.3) 90 / 81.  Q8_0
# 28672 x 4096 at 2048 (8.6) 461 / 497; 4096 x 4096 at 2048 (9.3) 80 / 81, at 3000 (13.9) 117 / 110; 6144 x 4096 at 3000 (12.3) 153 / 148.
# Q4_K and NVFP4 are ahead at every size up to 4096 tokens (28672 x 4096 at 4096: 791 / 853, 842 / 1050).
FUSED_WAVES = {"Q4_K": float("inf"), "NVFP4": float("inf"), "Q8_0": 10.0, "Q6_K": 6.0}


def decode_once(qtype: str, whole: bool, tokens: int, n: int, k: int, sms: int) -> bool:
    """Whether a product of ``tokens`` rows decodes its [n, k] matrix once.  ``whole``: its rows are whole super-blocks of 256 values on
    16-byte boundaries, which the fused kernel stages by TMA; others are read value by value, by every tile (Q6_K 2048 x 1536
    at 1025 tokens: 102 us fused, 30 decoded once)."""
    if C.mmq_max_tokens >= 0:
        return 0 < C.mmq_max_tokens < tokens
    if tokens <= DECODE_ONCE_ABOVE:
        return False
    if not whole:
        return True
    if qtype not in FUSED_WAVES:
        return True
    tiles = -(-n // 128)
    w256, w128 = (-(-tiles * -(-tokens // t) // sms) for t in (256, 128))
    waves = w256 if w256 < w128 else 0.6 * w128  # (as the plan of the fused kernel chooses)
    # (one wave of small tiles: the other form's two launches alone take longer; Q6_K 1024 x 4096 at 2048 tokens 39 / 42)
    return waves >= 1 and waves * sms > FUSED_WAVES[qtype] * tiles


def _launch(x, data_ptr, qt, row_bytes, scales_ptr, scale_ld, out_view, bias, ld_out, N, K):
    s = C.scratch(x.device)
    C._check(C.lib().oxb_gemm_quant(x.data_ptr(), data_ptr, qt, row_bytes, scales_ptr, scale_ld, out_view.data_ptr(),
                                    C._p(bias), x.shape[0], N, K, ld_out, 0, 0, s.gemm_ws.data_ptr(),
                                    s.gemm_ws.numel() * 4, s.gemm_counters.data_ptr(), s.gemm_counters.numel(),
                                    C._stream()), "oxb_gemm_quant")
    return out_view


def linear_quant(x, p, out_view, bias, ld_out):
    n, k = p.shape
    row_bytes = p.data.stride(0) * p.data.element_size()
    whole = k % 256 == 0 and row_bytes % 16 == 0 and p.data.data_ptr() % 16 == 0
    once = decode_once(p.qtype, whole, x.shape[0], n, k, C.sm_count(x.device)) and n * k <= (1 << 28)
    if p.qtype in FUSED_TYPES and k % 64 == 0 and not once:
        return _launch(x, p.data.data_ptr(), FUSED_TYPES[p.qtype], row_bytes, None, 0, out_view, bias, ld_out, n, k)
    buf = C.scratch(x.device).dequant_buf(n * k)[: n * k].view(n, k)
    C.dequant_rows(p, buf, fast=True)
    # The GEMM requests its first weight tiles before it waits for the upstream kernel, which is only safe
    # for weights that no kernel writes.  Here the "weights" were written by the launch just before, so this
    # GEMM is launched without programmatic stream serialization (plain stream order).
    L = C.lib()
    old = L.oxb_set_pdl(0)
    try:
        C.gemm_bf16(x, buf, out_view, bias, ld_out=ld_out)
    finally:
        L.oxb_set_pdl(old)
    return out_view


def linear_fp8(x, p, out_view, bias, ld_out):
    n, k = p.shape
    if p.block != 128 or k % 128 != 0:
        raise ValueError("block-scaled fp8 weights need 128-channel blocks and K % 128 == 0")
    return _launch(x, p.data.data_ptr(), QT_FP8B, k, p.scales.data_ptr(), p.scales.shape[1], out_view, bias, ld_out, n, k)
