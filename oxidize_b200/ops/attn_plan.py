"""Which sequences of a step take the tcgen05 attention kernel (``csrc/attention_prefill.cuh``) and which the mma.sync one.

The first runs 256 (token, query head) rows of a key head to a CTA over the whole visible context, unsplit: it has five to eight
times the other's rate where its CTAs fill the SMs, and leaves most of them idle where a sequence has few rows or heads.  The
other has a CTA for 16 rows and splits contexts.  So the choice goes by estimates of both, made per step from what the host
knows of it, and names sequences: the tail of a long prompt can take one kernel and the prompt next to it the other.

The constants are fits to one B200 (rows 32 to 2048 over contexts up to 32000; 8 to 64 query heads, groups of 1 to 8; windows;
steps of up to 64 sequences), in microseconds; over 791 such steps what the estimates choose is within 0.4 % of the better of
all and none on average, 23 % at worst.  Around the line, at 8 query heads / 1 key head of 128 in bf16: 256 rows over 8000 keys
(8 CTAs) take 168 us here and 86 there, 512 rows 170 and 147, 1024 rows 172 and 279; 8 / 2 heads of 64: 1024 rows 172 and 154,
2048 rows 174 and 266.  At 32 / 8 heads of 128: 64 rows over 8000 keys 168 and 86, 256 rows 174 and 272.  A portion of 500 rows and
a tail of 40 over 12000, 32 / 8 heads: 245 us both here, 242 both there, 103 apart.
"""
from __future__ import annotations

import math
from typing import List, Sequence, Tuple

MIN_ROWS = 32  # shorter portions are the other kernel's
MAX_SEQS = 2048  # ... as are steps of more sequences (its mask of sequences has a bit for each)
# Steps whose portions are all shorter than this are looked at only if their products alone, at 100 TFLOP/s, would take longer in the other
# kernel: for long contexts, that is.  More of them would gain (32 prompts of 33 rows, 32 heads: 20 us here, 61 there), but prompts
# of a hundred rows over q4 pages see little else than their own rows' codes, which the last bits of the layers before decide, and come out up
# to 8 % apart between the kernels (either is up to 19 % from 64 bits).
SHORT = 192
MAX_PAGES_BYTES = 512 << 20  # converted pages of a layer, at most

STEP, STEP_FIXED = 1.27, 6  # 64 keys of a CTA; what starting and ending a CTA costs, in such steps
CONVERT_RATE = 4.2e6  # bytes per us, read and written, of f16 / q8 / q4 pages on their way to bf16
SOURCE_BYTES = {"bf16": 0.0, "f16": 2.0, "q8": 1 + 4 / 32, "q4": 0.5 + 4 / 32}
# the other kernel, by page type: TFLOP/s with two to three CTAs to an SM (heads of 128, of 64), gain when there are many more;
# us that a warp takes for a page; us that a CTA takes beside its products, and one that finds no rows
OTHER_CTA, OTHER_IDLE_CTA = 5.0, 1.8
OTHER = {"bf16": (122, 72, 1.12, 1.5, 0.9), "f16": (60, 41, 1.12, 1.6, 1.5), "q8": (82, 62, 1.25, 1.2, 1.1), "q4": (108, 73, 1.25, 1.15, 0.9)}


def rows_per_cta(group: int) -> int:
    """Tokens of a CTA: 256 rows over the largest power of two that divides the query heads of a key head (128 at most)."""
    gp = 1
    while gp < 128 and group % (2 * gp) == 0:
        gp *= 2
    return 256 // gp


def first_page(rows: int, ctx: int, window: int) -> int:
    """First page that any of the last ``rows`` positions of ``ctx`` sees."""
    return max(0, ctx - rows - window + 1) // 16 if window > 0 else 0


def pages_seen(rows: int, ctx: int, window: int) -> int:
    return (ctx + 15) // 16 - first_page(rows, ctx, window)


def reserve_bytes(spec, max_len: int, max_seqs: int) -> int:
    """What the converted pages of a layer can take in a step over a cache like ``spec`` (``KVCacheSpec``): memory that a server leaves
    free beside its pool."""
    if spec.dtype_name not in SOURCE_BYTES or spec.dtype_name == "bf16" or spec.page_size != 16:
        return 0
    layers = [spec.shape(i) for i in range(spec.n_layers)]
    page = max((heads * 64 * width for heads, planes, width in layers if planes == 2 and width in (64, 128)), default=0)
    return min(MAX_PAGES_BYTES, page * (-(-max_len // 16)) * max_seqs)


def splits(seqs: int, nkv: int, mtiles: int, span: int, sms: int, per_sm: int) -> int:
    """CTA-level KV splits of the mma.sync kernel: as many as keep the grid within ONE wave of ``per_sm`` CTAs per SM (two, or three
    over quantized pages; a partly filled second wave doubles the kernel's time) while each warp of each split still sees a few
    pages."""
    base = max(1, seqs * nkv * mtiles)
    cap = max(1, (span + 15) // 16 // 8)  # >= 2 pages per warp per split
    return max(1, min(max(1, per_sm * sms // base), cap, 16))


def choose(lens: Sequence[Tuple[int, int]], nq: int, nkv: int, hd: int, pages: str, window: int, sms: int,
           most_bytes: int = MAX_PAGES_BYTES) -> List[int]:
    """Indices of the sequences ((rows fed, context length) each) for the tcgen05 kernel."""
    cand = [i for i, (n, c) in enumerate(lens) if n >= MIN_ROWS and c >= n]
    if not cand or len(lens) > MAX_SEQS:
        return []
    group = nq // nkv
    tokens, gp = rows_per_cta(group), 256 // rows_per_cta(group)
    rate128, rate64, many128, many64, page_us = OTHER[pages]
    rate, many = (rate128, many128) if hd > 64 else (rate64, many64)
    page_bytes = nkv * 32 * hd * (SOURCE_BYTES[pages] + 2) if pages != "bf16" else 0

    def work(n, c):  # TFLOP x 1e6 of n rows, each over the keys it sees
        full = c - n / 2
        return 4e-6 * nq * hd * n * (min(full, window) if window > 0 else full)

    if max(lens[i][0] for i in cand) < SHORT:
        waves = -(-sum(-(-lens[i][0] * nq // 256) for i in cand) // sms)
        walk = max(min(c, window + n) if window > 0 else c for n, c in (lens[i] for i in cand)) / 64
        if 1.3 * waves * (walk + STEP_FIXED) + 6 > sum(work(*lens[i]) for i in cand) / 100 + 8:
            return []

    # per sequence, for the tcgen05 kernel: work of its CTAs and of the longest (in steps), bytes of its pages, converted ones
    def alone(n, c):
        top = min(c, window + tokens) if window > 0 else c
        avg = min(c - n / 2, window + tokens) if window > 0 else c - n / 2
        seen = pages_seen(n, c, window)
        return (-(-n // tokens) * (nq // gp) * (avg / 64 + STEP_FIXED), top / 64 + STEP_FIXED, seen * page_bytes,
                seen * nkv * 64 * hd if page_bytes else 0)

    def other(n, c):  # ... and for the mma.sync kernel: rows, keys, tiles of 16 rows, time of its products
        return (n, min(c, window + n) if window > 0 else c, (n * group + 15) // 16 * nkv, work(n, c) * max(1.0, 16 / max(1, n * group)))

    def here(total, longest, conv):
        """us of the tcgen05 kernel: CTAs start longest first."""
        spread = max(longest, total / sms + 0.3 * longest) if total > 0.7 * sms * longest else longest
        return 3 + STEP * spread + (3 + conv / CONVERT_RATE if conv else 0)

    def there(seqs, rows, span, tiles, flops):
        """us of the mma.sync kernel."""
        if not seqs:
            return 0.0
        mtiles = (rows * group + 15) // 16
        sp = splits(seqs, nkv, mtiles, span, sms, 3 if pages in ("q8", "q4") else 2)
        per_sm = 4 if hd <= 64 else 3 if pages in ("q8", "q4") else 2
        around = (OTHER_CTA * tiles * sp + OTHER_IDLE_CTA * (len(lens) * mtiles * nkv - tiles) * sp) / (per_sm * sms)
        r = rate * (many if tiles > 3 * sms else 1.0)
        return 8 + 1.2 * math.log2(max(span / 64, 1)) + max(span / 16 / (4 * sp) * page_us, flops / r + around)

    # sequences join in order of their rows, as those with the most leave the fewest SMs idle; converted pages have to fit
    order, used = [], 0
    for i in sorted(cand, key=lambda i: (-lens[i][0], lens[i][1])):
        need = alone(*lens[i])[3]
        if used + need <= most_bytes:
            used += need
            order.append(i)
    joined = set(order)
    rest = (0, 0, 0, 0, 0.0)  # of the mma.sync kernel: sequences, most rows, most keys, tiles, time of the products

    def add(r, i):
        rows, span, tiles, flops = other(*lens[i])
        return (r[0] + 1, max(r[1], rows), max(r[2], span), r[3] + tiles, r[4] + flops)

    for i in range(len(lens)):
        if i not in joined:
            rest = add(rest, i)
    left = [rest]  # left[k]: with all but the first len(order) - k
    for i in reversed(order):
        left.append(add(left[-1], i))
    best, best_us = 0, there(*left[-1])
    total = longest = conv = 0.0
    for k, i in enumerate(order, 1):
        t, top, c, _ = alone(*lens[i])
        total, longest, conv = total + t, max(longest, top), conv + c
        us = here(total, longest, conv) + there(*left[len(order) - k])
        if us < best_us:
            best, best_us = k, us
    return sorted(order[:best])
