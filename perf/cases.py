"""Model steps as a serving process has them run, on one GPU: what is measured, on which inputs, and how exact it has to be.

A case is one step of a decoder over a paged cache: decoding (one row per running sequence, replayed from a CUDA graph as
the engine does), the verification of drafted tokens (a few rows per sequence) or a portion of prompts (many rows per
sequence).  The shapes are those of the presets that the benchmark and the tests run (``models.config.preset``) with fewer
layers, as every layer runs the same kernels; weights are random numbers in the checkpoint's encoding, the cache holds
earlier rows, contexts and portions are ragged.
"""
from __future__ import annotations

import math

import torch

DEV = "cuda"
PAGE = 16
STD = 0.02  # spread of random weights

#: Widths of the presets: hidden, heads, key / value heads, head width, feed-forward, vocabulary, rotary base, experts (all, per
#: token, their width), norms on q and k; layers run here.
SHAPES = {
    "tiny-llama": dict(h=512, nq=8, nkv=2, hd=64, ffn=1408, vocab=32000, theta=10000.0, E=0, k=0, ef=0, qk=False, layers=8),
    "llama3-8b": dict(h=4096, nq=32, nkv=8, hd=128, ffn=14336, vocab=128256, theta=500000.0, E=0, k=0, ef=0, qk=False, layers=4),
    "llama3-70b": dict(h=8192, nq=64, nkv=8, hd=128, ffn=28672, vocab=128256, theta=500000.0, E=0, k=0, ef=0, qk=False, layers=4),
    "mixtral-8x7b": dict(h=4096, nq=32, nkv=8, hd=128, ffn=14336, vocab=32000, theta=1000000.0, E=8, k=2, ef=14336, qk=False,
                         layers=2),
    "qwen3-30b-a3b": dict(h=2048, nq=32, nkv=4, hd=128, ffn=6144, vocab=151936, theta=1000000.0, E=128, k=8, ef=768, qk=True,
                          layers=4),
}


def _case(name, model, weights, kv, kind, seqs, ctx, rows):
    """``ctx`` and ``rows``: (least, most) of the tokens that a sequence has in the cache and of those that the step feeds it."""
    return {"name": name, "model": model, "weights": weights, "kv": kv, "kind": kind, "seqs": seqs, "ctx_lo": ctx[0], "ctx_hi": ctx[1],
            "rows_lo": rows[0], "rows_hi": rows[1]}


def listed():
    return [
        # a small model for one user: every launch and every latency counts
        _case("tiny q4 decode 1", "tiny-llama", "Q4_K_M", "f16", "decode", 1, (200, 200), (1, 1)),
        # chat with the most common kind of checkpoint: one user
        _case("8b q4 decode 1", "llama3-8b", "Q4_K_M", "q8", "decode", 1, (640, 640), (1, 1)),
        # the same served to 32 users
        _case("8b q4 decode 32", "llama3-8b", "Q4_K_M", "q8", "decode", 32, (513, 767), (1, 1)),
        # and a prompt of it
        _case("8b q4 prefill 512", "llama3-8b", "Q4_K_M", "q8", "prefill", 1, (0, 0), (512, 512)),
        # long documents in a small cache
        _case("8b bf16 q4kv decode 4 long", "llama3-8b", "BF16", "q4", "decode", 4, (20001, 30011), (1, 1)),
        # a portion of a long document
        _case("8b bf16 prefill long", "llama3-8b", "BF16", "bf16", "prefill", 1, (14000, 14000), (2048, 2048)),
        # the benchmark's headline: 64 sequences of a large model
        _case("70b bf16 decode 64", "llama3-70b", "BF16", "bf16", "decode", 64, (256, 2560), (1, 1)),
        # the portions of prompts that the scheduler puts between them: the end of one prompt and others whole
        _case("70b bf16 prefill 3 prompts", "llama3-70b", "BF16", "bf16", "prefill", 3, (0, 1100), (500, 1036)),
        # the large model in four bits
        _case("70b nvfp4 decode 64", "llama3-70b", "NVFP4", "bf16", "decode", 64, (256, 2560), (1, 1)),
        # few large experts in four bits
        _case("mixtral q4 decode 128", "mixtral-8x7b", "Q4_K", "bf16", "decode", 128, (300, 812), (1, 1)),
        _case("mixtral q4 prefill 5 prompts", "mixtral-8x7b", "Q4_K", "bf16", "prefill", 5, (0, 700), (500, 1138)),
        # many small experts; four drafted tokens of 16 sequences are verified
        _case("qwen3moe verify 16x5", "qwen3-30b-a3b", "BF16", "bf16", "verify", 16, (1024, 1280), (5, 5)),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(("tiny-llama", "llama3-8b", "llama3-8b", "llama3-8b", "llama3-70b", "llama3-70b", "mixtral-8x7b", "qwen3-30b-a3b"))
    weights = rng.choice({"tiny-llama": ("Q4_K_M", "BF16"), "llama3-8b": ("Q4_K_M", "BF16", "Q8_0"), "llama3-70b": ("BF16", "NVFP4"),
                          "mixtral-8x7b": ("Q4_K", "BF16"), "qwen3-30b-a3b": ("BF16", "Q4_K")}[model])
    kv = rng.choice(("bf16", "bf16", "f16", "q8", "q4"))
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "verify"))
    if kind == "decode":
        seqs = log_int(1, 128)
        rows = (1, 1)
        most = min(30000, 150000 // seqs)
    elif kind == "verify":
        seqs = log_int(1, 32)
        rows = (rng.randint(2, 6),) * 2
        most = min(8000, 60000 // seqs)
    else:
        seqs = rng.randint(1, 4)
        large = model == "llama3-70b"
        total = log_int(64, 2000 if large else 4000)
        hi = max(2, total // seqs)
        rows = (max(1, int(hi * rng.uniform(0.3, 1.0))), hi)
        most = min(12000, (10000000 if large else 20000000) // total) // seqs
    lo = log_int(32, most)
    ctx = (lo, max(lo, min(most, int(lo * rng.uniform(1.0, 4.0)))))
    if kind == "prefill" and rng.random() < 0.5:
        ctx = (0, 0)  # whole prompts
    c = _case("", model, weights, kv, kind, seqs, ctx, rows)
    del c["name"]
    return c


# ----------------------------------------------------------------------------------------------------------- inputs
def _spread(lo, hi, n):
    """n whole numbers from lo to hi, all over the range, the ends among them (one: the upper end)."""
    if n == 1:
        return [hi]
    return [lo + round((hi - lo) * ((i * 0.6180339887) % 1.0)) if 0 < i < n - 1 else (lo if i == 0 else hi) for i in range(n)]


def _lens(c):
    """[(tokens in the cache, rows of this step)] of the sequences."""
    return list(zip(_spread(c["ctx_lo"], c["ctx_hi"], c["seqs"]), reversed(_spread(c["rows_lo"], c["rows_hi"], c["seqs"]))))


def _matrix_type(weights, name, layer, layers, width):
    """The encoding of a matrix in a checkpoint of kind ``weights``."""
    t = weights
    if weights == "Q4_K_M":
        more = layer >= 7 * layers // 8 or layer < layers // 8 or (layer - layers // 8) % 3 == 2
        t = "Q6_K" if name == "head" or (name in ("v", "down") and more) else "Q4_K"
    return "Q8_0" if t in ("Q4_K", "Q6_K") and width % 256 else t


def _bytes_of(t):
    return {"BF16": 2.0, "Q4_K": 144 / 256, "Q6_K": 210 / 256, "Q8_0": 34 / 32, "NVFP4": 36 / 64}[t]


def _f16_bytes(x):
    return x.to(torch.float16).contiguous().view(torch.uint8)


def _pack(t, w):
    """float32 [n, k] in the encoding ``t``: bf16, or the rows' bytes."""
    n, k = w.shape
    if t == "BF16":
        return w.bfloat16()
    if t == "Q8_0":
        x = w.view(n, k // 32, 32)
        d = (x.abs().amax(-1, keepdim=True) / 127).half().float().clamp_min(1e-7)
        q = torch.round(x / d).clamp(-127, 127).to(torch.int8).view(torch.uint8)
        return torch.cat([_f16_bytes(d), q], -1).view(n, -1)
    if t == "Q4_K":
        x = w.view(n, k // 256, 8, 32)
        m = (-x.amin(-1)).clamp_min(0)
        s = (x.amax(-1) + m) / 15
        d = (s.amax(-1, keepdim=True) / 63).half().float().clamp_min(1e-7)
        dm = (m.amax(-1, keepdim=True) / 63).half().float().clamp_min(1e-7)
        sc, ms = torch.round(s / d).clamp(1, 63), torch.round(m / dm).clamp(0, 63)
        q = torch.round((x + (dm * ms)[..., None]) / (d * sc)[..., None]).clamp(0, 15).to(torch.uint8)
        sc, ms = sc.to(torch.uint8), ms.to(torch.uint8)
        six = torch.cat([sc[..., :4] | (sc[..., 4:] >> 4 << 6), ms[..., :4] | (ms[..., 4:] >> 4 << 6), (sc[..., 4:] & 15) | (ms[..., 4:] & 15) << 4], -1)
        return torch.cat([_f16_bytes(d), _f16_bytes(dm), six, (q[:, :, 0::2] | q[:, :, 1::2] << 4).flatten(2)], -1).view(n, -1)
    if t == "Q6_K":
        x = w.view(n, k // 256, 16, 16)
        s = x.abs().amax(-1) / 31
        d = (s.amax(-1, keepdim=True) / 127).half().float().clamp_min(1e-7)
        sc = torch.round(s / d).clamp(1, 127)
        q = (torch.round(x / (d * sc)[..., None]).clamp(-32, 31) + 32).to(torch.uint8).view(n, k // 256, 2, 4, 32)
        ql = (q[..., :2, :] & 15) | (q[..., 2:, :] & 15) << 4
        qh = q[..., 0, :] >> 4 | q[..., 1, :] >> 4 << 2 | q[..., 2, :] >> 4 << 4 | q[..., 3, :] >> 4 << 6
        return torch.cat([ql.flatten(2), qh.flatten(2), sc.to(torch.int8).view(torch.uint8), _f16_bytes(d)], -1).view(n, -1)
    x = w.view(n, k // 64, 4, 16)  # NVFP4
    s = (x.abs().amax(-1) / 6).clamp_min(2.0 ** -9).to(torch.float8_e4m3fn)
    steps = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=w.device)
    q = torch.bucketize((x / s.float()[..., None]).abs(), steps).to(torch.uint8) | (x < 0).to(torch.uint8) << 3
    return torch.cat([s.view(torch.uint8), (q[..., :8] | q[..., 8:] << 4).flatten(2)], -1).view(n, -1)


def _unpack(t, raw):
    """The values that the encoding stands for, in 64 bits."""
    n = raw.shape[0]
    if t == "BF16":
        return raw.double()
    b = raw.view(n, -1, {"Q8_0": 34, "Q4_K": 144, "Q6_K": 210, "NVFP4": 36}[t])
    half = lambda at: b[..., at : at + 2].contiguous().view(torch.float16).double()  # noqa: E731  [n, blocks, 1]
    if t == "Q8_0":
        return (half(0) * b[..., 2:].contiguous().view(torch.int8).double()).view(n, -1)
    if t == "Q4_K":
        six = b[..., 4:16]
        sc = torch.cat([six[..., :4] & 63, (six[..., 8:] & 15) | six[..., :4] >> 6 << 4], -1).double()
        ms = torch.cat([six[..., 4:8] & 63, six[..., 8:] >> 4 | six[..., 4:8] >> 6 << 4], -1).double()
        q = b[..., 16:].reshape(n, -1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 3).reshape(n, -1, 8, 32).double()
        return (q * (half(0) * sc)[..., None] - (half(2) * ms)[..., None]).view(n, -1)
    if t == "Q6_K":
        ql, qh = b[..., :128].reshape(n, -1, 2, 2, 32), b[..., 128:192].reshape(n, -1, 2, 1, 32)
        hi = torch.cat([qh & 3, qh >> 2 & 3, qh >> 4 & 3, qh >> 6], 3)
        q = (torch.cat([ql & 15, ql >> 4], 3) | hi << 4).reshape(n, -1, 16, 16).double() - 32
        return (q * (half(208) * b[..., 192:208].contiguous().view(torch.int8).double())[..., None]).view(n, -1)
    s = b[..., :4].contiguous().view(torch.float8_e4m3fn).double()
    q = b[..., 4:].reshape(n, -1, 4, 8)
    q = torch.cat([q & 15, q >> 4], -1)
    mag = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device=raw.device)[(q & 7).long()]
    return (torch.where(q > 7, -mag, mag) * s[..., None]).view(n, -1)


class _Inputs:
    """Weights, cached rows and tokens of a case, all from the seed."""

    def __init__(self, c, seed):
        s = SHAPES[c["model"]]
        self.s, self.lens = s, _lens(c)
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(seed)
        L, h, w = s["layers"], s["h"], c["weights"]
        dense = "BF16" if s["E"] and w == "Q4_K" else w  # four-bit experts behind 16-bit attention
        self.layers, routers = [], []
        for i in range(L):
            kind = lambda name, width: _matrix_type(dense, name, i, L, width)  # noqa: E731
            q_rows, k_rows = s["nq"] * s["hd"], s["nkv"] * s["hd"]
            one = {"attn_norm": self.norm(h), "ffn_norm": self.norm(h)}
            if kind("q", h) == kind("v", h):
                one["qkv"] = [self.matrix(kind("q", h), q_rows + 2 * k_rows, h)]
            else:
                one["qkv"] = [self.matrix(kind("q", h), q_rows + k_rows, h), self.matrix(kind("v", h), k_rows, h)]
            one["o"] = self.matrix(kind("o", q_rows), h, q_rows)
            if s["qk"]:
                one["q_norm"], one["k_norm"] = self.norm(s["hd"]), self.norm(s["hd"])
            if s["E"]:
                one["router"] = self.matrix("BF16", s["E"], h)
                routers.append(one["router"][1].float())
                one["up"] = [self.matrix(w, 2 * s["ef"], h) for _ in range(s["E"])]
                one["down"] = [self.matrix(w, h, s["ef"]) for _ in range(s["E"])]
            else:
                one["up"] = self.matrix(kind("up", h), 2 * s["ffn"], h)
                one["down"] = self.matrix(kind("down", s["ffn"]), h, s["ffn"])
            self.layers.append(one)
        embed = torch.randn(s["vocab"], h, generator=self.gen, device=DEV)
        for r in routers:
            # A trained router tells its experts apart.  Random ones nearly tie for many tokens, which 16 bits then decide either
            # way: so that outputs can be compared, every token leans towards a random choice of experts in every layer.
            chosen = torch.rand(s["vocab"], s["E"], generator=self.gen, device=DEV).topk(s["k"], 1).indices
            embed += torch.zeros(s["vocab"], s["E"], device=DEV).scatter_(1, chosen, 6.0 if s["k"] < 4 else 10.0) @ r
        t = _matrix_type(dense, "embed", 0, L, h)
        self.embed = (t, torch.cat([_pack(t, e) for e in embed.split(32768)]))
        del embed
        self.head = self.matrix(_matrix_type(dense, "head", 0, L, h), s["vocab"], h)
        self.out_norm = self.norm(h)
        # pages: those that this step writes come first, then those of earlier rows only; a quantized pool has many more, as a
        # server's has, so that the few codes that close calls decide stay few among all
        need = [(-(-(n + r) // PAGE), n // PAGE) for n, r in self.lens]
        self.written = sum(a - b for a, b in need)
        total = sum(a for a, _ in need)
        quantized = c["kv"] in ("q8", "q4")
        self.blocks = max(total, 64 * self.written) if quantized else total
        order = (torch.randperm(total - self.written, generator=self.gen, device=DEV) + self.written).tolist()
        first, at, self.tables = 0, 0, []
        for a, b in need:
            self.tables.append(order[at : at + b] + list(range(first, first + a - b)))
            first, at = first + a - b, at + b
        self.tokens = torch.randint(0, s["vocab"], (sum(r for _, r in self.lens),), generator=self.gen, device=DEV, dtype=torch.int32)
        self.cache, self.scales = [], []
        shape = (self.blocks, s["nkv"], 2, PAGE)
        for _ in range(L):
            x = torch.empty(*shape, s["hd"], device=DEV, dtype=torch.bfloat16).normal_(generator=self.gen)
            if not quantized:
                self.cache.append(x.to(torch.float16 if c["kv"] == "f16" else torch.bfloat16))
                continue
            top, step = (127, 40.0) if c["kv"] == "q8" else (7, 2.5)
            q = (torch.round(x * step).clamp_(-top, top) + top).to(torch.uint8)
            self.cache.append(q if top == 127 else q[..., 0::2] | q[..., 1::2] << 4)
            self.scales.append((torch.rand(*shape, s["hd"] // 32, generator=self.gen, device=DEV) + 0.5) / step)

    def norm(self, n):
        return 1 + 0.1 * torch.randn(n, generator=self.gen, device=DEV)

    def matrix(self, t, n, k):
        step = max(1, (1 << 27) // k)
        return t, torch.cat([_pack(t, torch.randn(min(step, n - r), k, generator=self.gen, device=DEV) * STD) for r in range(0, n, step)])


def prepare(case, seed):
    from oxidize_b200.models.config import preset
    from oxidize_b200.models.transformer import BatchMeta, Transformer
    from oxidize_b200.models.weights import ExpertWeights, LayerWeights, LinearWeight, ModelWeights, QTensor

    x = _Inputs(case, seed)
    s = x.s

    def q(m):
        t, data = m
        return QTensor(t, data, (data.shape[0], data.shape[1] if t == "BF16" else round(data.shape[1] / _bytes_of(t))))

    def weights(i, one):
        lw = LayerWeights(attn_norm=one["attn_norm"], ffn_norm=one["ffn_norm"], wqkv=LinearWeight([q(m) for m in one["qkv"]]),
                          wo=LinearWeight([q(one["o"])]), q_norm=one.get("q_norm"), k_norm=one.get("k_norm"))
        if s["E"]:
            lw.router, lw.experts = q(one["router"]), ExpertWeights([q(m) for m in one["up"]], [q(m) for m in one["down"]])
            one["up"] = one["down"] = None
            lw.experts.stack()
        else:
            lw.w_gate_up, lw.w_down = LinearWeight([q(one["up"])]), LinearWeight([q(one["down"])])
        x.layers[i] = None  # the model's from here on
        return lw

    longest = max(n + r for n, r in x.lens)
    width = 2 * -(-longest // PAGE)  # a server's limit lies above the sequences that it has
    cfg = preset(case["model"], n_layers=s["layers"])
    layers = [weights(i, one) for i, one in enumerate(x.layers)]
    model = Transformer(ModelWeights(cfg, q(x.embed), layers, x.out_norm, LinearWeight([q(x.head)])), max_context=width * PAGE)
    kv = model.new_cache(x.blocks, PAGE, case["kv"])
    for i in range(s["layers"]):
        kv.data[i].copy_(x.cache[i])
        if x.scales:
            kv.scales[i].copy_(x.scales[i])
    x.cache = x.scales = None

    decode = case["kind"] == "decode"
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    starts = [sum(r for _, r in x.lens[:i]) for i in range(len(x.lens) + 1)]
    positions = [p for n, r in x.lens for p in range(n, n + r)]
    slots = [t[p // PAGE] * PAGE + p % PAGE for t, (n, r) in zip(x.tables, x.lens) for p in range(n, n + r)]
    wanted = [e - 1 for e in starts[1:]] if case["kind"] == "prefill" else list(range(starts[-1]))
    meta = BatchMeta(token_ids=x.tokens, positions=ints(positions), slot_mapping=ints(slots), query_start=ints(starts),
                     seq_lens=ints([n + r for n, r in x.lens]), block_tables=ints([t + [0] * (width - len(t)) for t in x.tables]),
                     logits_indices=ints(wanted), max_query_len=max(r for _, r in x.lens),
                     max_seq_len=width * PAGE if decode else longest, num_seqs=len(x.lens), logits_all=decode)
    state = {"model": model, "kv": kv, "meta": meta, "graph": None,
             "pages": [d if kv.scales[0] is not None else d[: x.written] for d in kv.data]}
    if decode:  # a server captures its decode step once and replays it
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                model.forward(meta, kv)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["logits"] = model.forward(meta, kv)
    else:
        meta.host_lens = [(r, n + r) for n, r in x.lens]
    return state


def run(state):
    """The logits that the step is there for, and the pages that it writes."""
    if state["graph"] is not None:
        state["graph"].replay()
        logits = state["logits"]
    else:
        logits = state["model"].forward(state["meta"], state["kv"])
    scales = state["kv"].scales if state["kv"].scales[0] is not None else []
    return {"logits": logits, "pages": state["pages"], "scales": scales}


def work(case):
    s, lens = SHAPES[case["model"]], _lens(case)
    h, hd, L, w = s["h"], s["hd"], s["layers"], case["weights"]
    dense = "BF16" if s["E"] and w == "Q4_K" else w
    T = sum(r for _, r in lens)
    out_rows = len(lens) if case["kind"] == "prefill" else T
    row = 2 * s["nkv"] * hd * {"bf16": 2.0, "f16": 2.0, "q8": 1 + 4 / 32, "q4": 0.5 + 4 / 32}[case["kv"]]
    kind = lambda name, i, k: _bytes_of(_matrix_type(dense, name, i, L, k))  # noqa: E731
    bytes_ = s["vocab"] * h * kind("head", 0, h) + T * h * kind("embed", 0, h) + out_rows * s["vocab"] * 4
    flops = 2.0 * out_rows * s["vocab"] * h
    for i in range(L):
        q_rows, k_rows = s["nq"] * hd, s["nkv"] * hd
        bytes_ += h * ((q_rows + k_rows) * kind("q", i, h) + k_rows * kind("v", i, h)) + h * q_rows * kind("o", i, q_rows)
        flops += 2.0 * T * h * (2 * q_rows + 2 * k_rows)
        if s["E"]:
            touched = s["E"] * (1 - (1 - s["k"] / s["E"]) ** T)
            bytes_ += touched * 3 * h * s["ef"] * _bytes_of(w) + s["E"] * h * 2
            flops += 2.0 * T * h * (s["E"] + 3 * s["k"] * s["ef"])
        else:
            bytes_ += h * s["ffn"] * (2 * kind("up", i, h) + kind("down", i, s["ffn"]))
            flops += 6.0 * T * h * s["ffn"]
        bytes_ += sum(n + r for n, r in lens) * row
        flops += sum(4.0 * q_rows * (r * n + r * (r + 1) / 2) for n, r in lens)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # Activations are rounded to 16 bits between the operators, a packed matrix's scales too (and activations to 8 bits ahead of
    # its products for one or two tokens): logits are 0.5 to 2.4 % off the statement in 64 bits, and two implementations that
    # round elsewhere are as far from one another.  Quantized pages differ in codes where a value lies between two of them.
    return {"rel": 0.03, "max": 0.5, "differ": 0.01}


# ------------------------------------------------------------------------------------------------------ plain statement
def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w.double()


def _rotate(x, pos, theta):
    half = x.shape[-1] // 2
    ang = pos.double()[:, None] * theta ** (-torch.arange(half, device=DEV, dtype=torch.float64) / half)
    cos, sin, a, b = ang.cos()[:, None], ang.sin()[:, None], x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _times(x, m):
    t, raw = m
    return torch.cat([x @ _unpack(t, r).t() for r in raw.split(16384)], -1)


def _through_codes(x, kv):
    """What a quantized cache keeps of rows: whole multiples of a scale for every 32 values."""
    top = 127 if kv == "q8" else 7
    scale = x.unflatten(-1, (-1, 32)).abs().amax(-1, keepdim=True) / top
    return (torch.round(x.unflatten(-1, (-1, 32)) / scale) * scale).flatten(-2)


def exact(case, seed):
    x = _Inputs(case, seed)
    s, lens = x.s, x.lens
    nq, nkv, hd = s["nq"], s["nkv"], s["hd"]
    quantized = bool(x.scales)
    pos = torch.cat([torch.arange(n, n + r, device=DEV) for n, r in lens])
    seq_of = [slice(sum(r for _, r in lens[:i]), sum(r for _, r in lens[: i + 1])) for i in range(len(lens))]
    hidden = _unpack(x.embed[0], x.embed[1][x.tokens.long()])
    pages = []
    for i, one in enumerate(x.layers):
        a = _rms(hidden, one["attn_norm"])
        z = torch.cat([_times(a, m) for m in one["qkv"]], -1).view(len(a), nq + 2 * nkv, hd)
        q, k, v = (part.clone() for part in z.split([nq, nkv, nkv], 1))
        if s["qk"]:
            q, k = _rms(q, one["q_norm"]), _rms(k, one["k_norm"])
        q, k = _rotate(q, pos, s["theta"]), _rotate(k, pos, s["theta"])
        cache = x.cache[i]
        kept = None if quantized else cache[: x.written].double()
        att = torch.empty_like(q)
        for table, (n, r), rows in zip(x.tables, lens, seq_of):
            blocks = torch.tensor(table, device=DEV)
            old = cache[blocks]
            if quantized:
                k[rows], v[rows] = _through_codes(k[rows], case["kv"]), _through_codes(v[rows], case["kv"])
                if case["kv"] == "q4":
                    old = torch.stack([old & 15, old >> 4], -1).flatten(-2)
                old = old.double().unflatten(-1, (-1, 32)) - (127 if case["kv"] == "q8" else 7)
                old = (old * x.scales[i][blocks][..., None]).flatten(-2)
            old = old.permute(2, 0, 3, 1, 4).reshape(2, -1, nkv, hd)[:, :n].double()
            keys, values = torch.cat([old[0], k[rows]]), torch.cat([old[1], v[rows]])
            seen = torch.arange(n + r, device=DEV)[None] <= pos[rows][:, None]
            for g in range(nkv):
                heads = slice(g * nq // nkv, (g + 1) * nq // nkv)
                for part in range(rows.start, rows.stop, 512):
                    some = slice(part, min(part + 512, rows.stop))
                    score = torch.einsum("rhd,kd->hrk", q[some, heads], keys[:, g]) / math.sqrt(hd)
                    score.masked_fill_(~seen[some.start - rows.start : some.stop - rows.start][None], -math.inf)
                    att[some, heads] = torch.einsum("hrk,kd->rhd", score.softmax(-1), values[:, g])
            if kept is not None:
                at = pos[rows]
                kept[blocks[at // PAGE], :, 0, at % PAGE], kept[blocks[at // PAGE], :, 1, at % PAGE] = k[rows], v[rows]
        pages.append(kept)
        hidden = hidden + _times(att.flatten(1), one["o"])
        a = _rms(hidden, one["ffn_norm"])

        def block(y, up, down):
            gate, up = _times(y, up).chunk(2, -1)
            return _times(torch.nn.functional.silu(gate) * up, down)

        if s["E"]:
            top, ids = _times(a, one["router"]).topk(s["k"], -1)
            top, out = top.softmax(-1), torch.zeros_like(hidden)
            for e in range(s["E"]):
                row, which = (ids == e).nonzero(as_tuple=True)
                if len(row):
                    out.index_add_(0, row, block(a[row], one["up"][e], one["down"][e]) * top[row, which][:, None])
            hidden = hidden + out
        else:
            hidden = hidden + block(a, one["up"], one["down"])
    if case["kind"] == "prefill":
        hidden = hidden[[r.stop - 1 for r in seq_of]]
    return {"logits": _times(_rms(hidden, x.out_norm), x.head), "pages": pages, "scales": [None] * len(x.scales)}
