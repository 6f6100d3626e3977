"""Kernels whose tiles follow the size of a call, at the edges of those tiles, against plain statements of the same op."""
import pytest
import torch

from oxidize_b200 import ops
from oxidize_b200.engine.kv_pool import KVCache, KVCacheSpec
from oxidize_b200.models.transformer import BatchMeta
from oxidize_b200.models.weights import qtensor_from_dense
from oxidize_b200.ops import ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from oxidize_b200.ops import cuda as C

    C.lib()
    return C


def _off(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm())


def _check_status(C):
    torch.cuda.synchronize()
    assert C.status() == (0, 0, 0)


# ------------------------------------------------------------------------------------------------- attention
def _step(kvd, hd, nq, nkv, lens, seed=0):
    """Cache (pages in random order, a page past each sequence's own), step and queries of (rows fed, context) sequences."""
    gen = torch.Generator().manual_seed(seed)
    need = [(c + 15) // 16 for _, c in lens]
    cpu = KVCache(KVCacheSpec(1, nkv, hd, 16, kvd), sum(need) + 2, torch.device("cpu"))
    order = torch.randperm(sum(need) + 2, generator=gen).tolist()
    tables, at = [], 0
    for n, (_, c) in zip(need, lens):
        tables.append(order[at : at + n] + [0] * (max(need) + 1 - n))
        at += n
        slots = torch.tensor([tables[-1][p // 16] * 16 + p % 16 for p in range(c)], dtype=torch.int32)
        k, v = (torch.randn(c, nkv, hd, generator=gen).bfloat16().float() for _ in range(2))
        ref.kv_write(cpu, 0, k, v, slots)
    starts = [sum(n for n, _ in lens[:i]) for i in range(len(lens) + 1)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    meta = BatchMeta(None, None, None, ints(starts), ints([c for _, c in lens]), ints(tables), None, max(n for n, _ in lens),
                     max(c for _, c in lens), len(lens))
    gpu = KVCache(cpu.spec, cpu.num_blocks, torch.device("cuda"))
    gpu.data = [d.cuda() for d in cpu.data]
    gpu.scales = [None if s is None else s.cuda() for s in cpu.scales]
    on_gpu = BatchMeta(None, None, None, meta.query_start.cuda(), meta.seq_lens.cuda(), meta.block_tables.cuda(), None, meta.max_query_len,
                       meta.max_seq_len, len(lens), host_lens=list(lens))
    q = torch.randn(starts[-1], nq, hd, generator=gen).bfloat16()
    return cpu, meta, gpu, on_gpu, q


LONG = [(200, 200), (64, 300), (1, 70), (33, 33), (3, 18), (257, 450)]  # long ones, and short ones that the other kernel takes


@pytest.mark.parametrize("kvd,hd,nq,nkv,lens,window", [
    ("bf16", 128, 8, 2, LONG, 0), ("bf16", 64, 4, 4, LONG, 0), ("bf16", 128, 7, 1, LONG, 0), ("bf16", 128, 12, 2, [(192, 193)], 0),
    ("bf16", 128, 16, 1, [(224, 1000)], 0), ("bf16", 128, 8, 2, LONG, 50), ("bf16", 64, 4, 2, [(200, 400)], 200),
    ("f16", 128, 8, 2, LONG, 0), ("q8", 128, 8, 2, LONG, 0), ("q4", 128, 8, 2, LONG, 0), ("q8", 64, 4, 1, LONG, 90), ("q4", 64, 4, 2, LONG, 0)])
def test_long_portions(C, kvd, hd, nq, nkv, lens, window):
    cpu, meta, gpu, on_gpu, q = _step(kvd, hd, nq, nkv, lens)
    got = C.paged_attention(q.cuda(), gpu, 0, on_gpu, hd ** -0.5, window)
    _check_status(C)
    want = ref.paged_attention(q.float(), cpu, 0, meta, hd ** -0.5, window)
    # outputs are rounded to bf16 (2e-3 at most), and f16 and quantized rows on their way in (as much again, keys and values)
    assert _off(got, want) < (2.5e-3 if kvd == "bf16" else 6e-3)
    assert torch.isfinite(got.float()).all()


def test_long_portion_with_sink_gate_and_a_wider_output(C):
    cpu, meta, gpu, on_gpu, q = _step("bf16", 128, 8, 2, LONG)
    T = q.shape[0]
    sink, gate = torch.randn(8), torch.randn(T, 8 * 128).bfloat16()
    wide = torch.full((T, 8 * 128 + 10), 7.0, dtype=torch.bfloat16, device="cuda")
    C.paged_attention(q.cuda(), gpu, 0, on_gpu, 128 ** -0.5, sink=sink.cuda(), out=wide[:, 2 : 2 + 8 * 128], gate=gate.cuda(),
                      gate_per_value=True)
    other = C.paged_attention(q.cuda(), gpu, 0, on_gpu, 128 ** -0.5, splits=1, sink=sink.cuda(), gate=gate.cuda(), gate_per_value=True)
    _check_status(C)
    assert _off(wide[:, 2 : 2 + 8 * 128], other.reshape(T, -1)) < 6e-3  # (two roundings to bf16, probabilities of the other's to bf16 too)
    assert (wide[:, :2] == 7).all() and (wide[:, 2 + 8 * 128 :] == 7).all()


@pytest.mark.parametrize("kvd", ["q8", "q4"])
@pytest.mark.parametrize("hd,nq,nkv,lens", [(128, 8, 2, [(1, 1), (1, 16), (1, 17), (5, 333), (1, 2000)]), (64, 7, 7, [(1, 40), (3, 3)]),
                                            (64, 32, 2, [(1, 500), (4, 64)])])
def test_quantized_pages_in_fragments(C, kvd, hd, nq, nkv, lens):
    cpu, meta, gpu, on_gpu, q = _step(kvd, hd, nq, nkv, lens)
    want = ref.paged_attention(q.float(), cpu, 0, meta, hd ** -0.5, 0)
    for splits in (None, 1, 3):
        got = C.paged_attention(q.cuda(), gpu, 0, on_gpu, hd ** -0.5, splits=splits)
        _check_status(C)
        # codes are exact; the output and the scaled probabilities are rounded to bf16
        assert _off(got, want) < 4e-3


@pytest.mark.parametrize("kvd", ["bf16", "f16", "q8", "q4"])
@pytest.mark.parametrize("hd,rot,pairing,norm", [(64, 64, "split_half", True), (64, 32, "adjacent", False), (128, 128, "adjacent", True),
                                                 (128, 96, "split_half", False), (256, 64, "split_half", True), (256, 256, "adjacent", False),
                                                 (128, 20, "split_half", True), (96, 96, "split_half", False)])
def test_rotation_and_cache_rows_of_a_warp_to_a_head(C, kvd, hd, rot, pairing, norm):
    """Widths and rotations that a warp per head takes (the last two: that it does not), a token count that fills no CTA."""
    from types import SimpleNamespace

    gen = torch.Generator().manual_seed(hd + rot)
    T, nq, nkv = 11, 3, 2
    qkv = torch.randn(T, (nq + 2 * nkv) * hd, generator=gen).bfloat16()
    pos = torch.tensor([0, 1, 2, 40, 41, 7, 100, 3000, 5, 6, 9], dtype=torch.int32)
    slots = torch.tensor([0, 1, 2, 56, 57, 23, -1, 90, 21, 22, 127], dtype=torch.int32)
    norms = [torch.rand(hd, generator=gen) + 0.5 if norm else None for _ in range(2)]
    caches, queries = [], []
    for dev in ("cpu", "cuda"):
        kv = KVCache(KVCacheSpec(1, nkv, hd, 16, kvd), 8, torch.device(dev))
        rope = SimpleNamespace(inv_freq=ref.rope_inv_freq(rot, 10000.0, None, device=dev), pairing=pairing, mscale=1.0, n_heads=nq,
                               n_kv_heads=nkv, head_dim=hd, max_pos=0)
        x = qkv.float() if dev == "cpu" else qkv.cuda()
        queries.append(ops.qk_rope_kv_write(x, pos.to(dev), slots.to(dev), kv, 0, rope,
                                            *[None if n is None else n.to(dev) for n in norms], 1e-6))
        caches.append(kv)
    _check_status(C)
    assert _off(queries[1], queries[0]) < 3e-3  # rounded to bf16
    back = KVCache(caches[0].spec, 8, torch.device("cpu"))
    back.data, back.scales = [d.cpu() for d in caches[1].data], [None if s is None else s.cpu() for s in caches[1].scales]
    table = torch.arange(8, dtype=torch.int32)
    for got, want in zip(ref.kv_gather(back, 0, table, 128), ref.kv_gather(caches[0], 0, table, 128)):
        # (quantized: a code may fall to the other side where a value lies between two; one step of 32 values' largest)
        assert _off(got, want) < {"bf16": 3e-3, "f16": 1e-3, "q8": 2e-3, "q4": 3e-2}[kvd]


# ------------------------------------------------------------------------------------------- packed GEMM
@pytest.mark.parametrize("qtype", ["Q4_K", "Q6_K", "Q8_0", "NVFP4", "Q4_0"])
@pytest.mark.parametrize("T,N,K", [(1, 300, 320), (17, 130, 1280), (64, 128, 256), (129, 260, 2816), (256, 20000, 256), (257, 19100, 512),
                                   (600, 520, 768)])
def test_packed_gemm_tiles(C, qtype, T, N, K):
    if qtype in ("Q4_K", "Q6_K") and K % 256:
        pytest.skip("blocks of 256 values")
    gen = torch.Generator(device="cuda").manual_seed(T + N)
    w = qtensor_from_dense((torch.randn(N, K, generator=gen, device="cuda") * 0.05).cpu(), qtype, device="cuda")
    x = torch.randn(T, K, generator=gen, device="cuda").bfloat16()
    x[0, : K // 2] = 0
    C.configure(C.KernelOptions(gemv_max_tokens=0, mmq_max_tokens=0))
    try:
        got = C.linear(x, [w])
        again = C.linear(x, [w])
    finally:
        C.configure(C.KernelOptions())
    _check_status(C)
    want = x.double() @ C.dequant_rows(w).double().t()  # (decoded value by value, to bf16)
    assert _off(got, want) < 8e-3  # output, and for the k-quants scales and offsets, rounded to bf16
    assert torch.equal(got, again)


@pytest.mark.parametrize("qtype,N,K", [("BF16", 200, 128), ("Q4_K", 256, 512)])
@pytest.mark.parametrize("rows", [[0] * 39 + [5], [1] * 40, [0, 300, 0, 17] + [0] * 30 + [16, 33, 1, 0, 128, 129], [2, 700] + [3] * 38])
def test_grouped_rows_lists(C, qtype, N, K, rows):
    """Groups with no rows, with rows for several tiles, and more of them than a warp has lanes."""
    from oxidize_b200.ops import cuda_moe

    E, R = len(rows), sum(rows)
    gen = torch.Generator(device="cuda").manual_seed(R)
    dense = torch.randn(E * N, K, generator=gen, device="cuda") * 0.05
    w = qtensor_from_dense(dense.cpu(), qtype, device="cuda")
    x = torch.randn(R + 9, K, generator=gen, device="cuda").bfloat16()  # rows past the last group are not touched
    off = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32, device="cuda")
    got = cuda_moe.gemm_grouped_rows(x, w, off, E, max(rows))
    _check_status(C)
    full = (w.data if qtype == "BF16" else C.dequant_rows(w)).double().view(E, N, K)
    want = torch.cat([x[a:b].double() @ full[e].t() for e, (a, b) in enumerate(zip(off[:-1].tolist(), off[1:].tolist()))])
    assert _off(got[:R], want) < 8e-3


def _worst(got, want):
    """Largest distance of a row and of a column, each over the root mean square row's or column's norm: a lost edge shows."""
    d, w = (got.double() - want).cpu(), want.cpu()
    return max(float(d.norm(dim=i).max() / w.norm(dim=i).square().mean().sqrt()) for i in (0, 1))


@pytest.mark.parametrize("qtype", ["BF16", "Q4_K"])
@pytest.mark.parametrize("N,K,rows", [(260, 2624, [300, 130, 0, 257]), (260, 2304, [150] * 5), (18961, 256, [0, 70, 5, 33, 1]), (300, 2560, [1] * 200 + [40])])
def test_grouped_rows_wide_tiles_and_orders(C, qtype, N, K, rows):
    """Tiles of 256 rows over rows long enough that every ring wraps, more weight tiles than SMs (group by group), groups by the hundred."""
    from oxidize_b200.ops import cuda_moe

    if qtype == "Q4_K" and K % 256:
        K = 2560
    E, R = len(rows), sum(rows)
    gen = torch.Generator(device="cuda").manual_seed(R)
    w = qtensor_from_dense((torch.randn(E * N, K, generator=gen, device="cuda") * 0.05).cpu(), qtype, device="cuda")
    x = torch.randn(R + 9, K, generator=gen, device="cuda").bfloat16()
    off = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32, device="cuda")
    got = cuda_moe.gemm_grouped_rows(x, w, off, E, max(rows))
    _check_status(C)
    full = (w.data if qtype == "BF16" else C.dequant_rows(w)).double().view(E, N, K)
    want = torch.cat([x[a:b].double() @ full[e].t() for e, (a, b) in enumerate(zip(off[:-1].tolist(), off[1:].tolist()))])
    assert _off(got[:R], want) < 8e-3  # (as test_grouped_rows_lists)
    assert _worst(got[:R], want) < 3e-2  # roundings alone: a row or column of 260 values or more is within a few times the whole


@pytest.mark.parametrize("qtype,rows,expected,groups,most,N,K,tn,splits", [
    ("Q4_K", 800, 0, 8, 400, 28672, 4096, 128, 1),   # 100 rows to a group: a tile of 256 would be emptier
    ("BF16", 800, 0, 8, 400, 4096, 14336, 128, 1),   # ... and not split along K
    ("Q4_K", 1200, 0, 8, 600, 28672, 4096, 256, 1),
    ("Q4_K", 400, 100, 2, 200, 28672, 4096, 128, 1),  # one rank of four: its experts get a quarter of the step's rows
    ("BF16", 2, 0, 8, 1, 28672, 4096, 16, 1),        # one token, short rows: not split
    ("Q4_K", 1024, 0, 128, 128, 2048, 768, 32, 1)])  # many experts in four bits: 32 tokens at least
def test_grouped_rows_plans(C, qtype, rows, expected, groups, most, N, K, tn, splits):
    import ctypes

    out = (ctypes.c_int * 4)()
    assert C.lib().oxb_gemm_grouped_rows_plan(rows, C.QTYPE_CODE[qtype], groups, most, expected, N, K, out) == 0
    assert (out[0], out[3]) == (tn, splits)


@pytest.mark.parametrize("kvd", ["bf16", "q8"])
@pytest.mark.parametrize("lens,window", [([(200, 1000), (33, 500)], 50), ([(256, 600), (1, 300)], 100), ([(300, 700)], 17)])
def test_long_portions_read_no_page_below_the_window(C, kvd, lens, window):
    """Table entries of pages that no row sees may be anything, and the pages hold anything: here ids out of range."""
    cpu, meta, gpu, on_gpu, q = _step(kvd, 128, 8, 2, lens)
    want = ref.paged_attention(q.float(), cpu, 0, meta, 128 ** -0.5, window)
    for b, (n, c) in enumerate(lens):
        on_gpu.block_tables[b, : max(0, c - n - window + 1) // 16] = -1 - b
    got = C.paged_attention(q.cuda(), gpu, 0, on_gpu, 128 ** -0.5, window)
    _check_status(C)
    assert _off(got, want) < (2.5e-3 if kvd == "bf16" else 6e-3)  # (as test_long_portions)


@pytest.mark.parametrize("kvd", ["bf16", "q8"])
@pytest.mark.parametrize("offset,scale", [(2, 0.09), (6, 0.09), (0, 0.0), (0, -0.09), (8, 0.09)])
def test_long_portions_of_queries_on_any_boundary_and_with_any_scale(C, kvd, offset, scale):
    """The tcgen05 kernel copies queries from 16-byte boundaries and takes the maximum before it scales: others are served all the same."""
    cpu, meta, gpu, on_gpu, q = _step(kvd, 128, 8, 2, LONG)
    room = torch.zeros(q.numel() + 8, dtype=torch.bfloat16, device="cuda")
    at = room[offset : offset + q.numel()].view(q.shape)
    at.copy_(q)
    got = C.paged_attention(at, gpu, 0, on_gpu, scale, 0)
    _check_status(C)
    want = ref.paged_attention(q.float(), cpu, 0, meta, scale, 0)
    assert _off(got, want) < (2.5e-3 if kvd == "bf16" else 6e-3)  # (as test_long_portions)


@pytest.mark.parametrize("qtype", ["Q4_K", "Q6_K", "Q8_0", "NVFP4", "Q4_0", "FP8B"])
@pytest.mark.parametrize("T,N,K", [(200, 9601, 2560), (500, 9601, 2560), (256, 9700, 2432), (255, 10000, 2944)])
def test_packed_gemm_tiles_of_256(C, qtype, T, N, K):
    """Every ring wraps several times (ten super-blocks and more, or an odd number of k-blocks); rows and columns one by one; nothing
    but the output is written."""
    import ctypes

    from oxidize_b200.ops import cuda_quant

    if K % 256 and qtype in ("Q4_K", "Q6_K"):
        K = 2816
    plan = (ctypes.c_int * 4)()
    assert C.lib().oxb_gemm_quant_plan(T, N, K, plan) == 0 and plan[0] == 256 and plan[3] == 1
    gen = torch.Generator(device="cuda").manual_seed(T + K)
    some = 1201  # distinct rows, repeated: no whole number of tiles
    w = qtensor_from_dense((torch.randn(some, K, generator=gen, device="cuda") * 0.05).cpu(), qtype, device="cuda")
    dense = w.to("cpu").dense_cache().double().cuda()
    again = -(-N // some)
    w.data = w.data.repeat(again, 1)[:N].contiguous()
    w.scales = None if w.scales is None else w.scales.repeat(again, 1)[:N].contiguous()
    w.shape, w._dense = (N, K), None
    x = torch.randn(T, K, generator=gen, device="cuda").bfloat16()
    bias = torch.randn(N, generator=gen, device="cuda")
    room = torch.full((T + 4, N + 27), 7.0, dtype=torch.bfloat16, device="cuda")
    out = room[2 : T + 2, 8 : N + 8]
    C.configure(C.KernelOptions(gemv_max_tokens=0, mmq_max_tokens=0))
    try:
        (cuda_quant.linear_fp8 if qtype == "FP8B" else cuda_quant.linear_quant)(x, w, out, bias, room.stride(0))
    finally:
        C.configure(C.KernelOptions())
    _check_status(C)
    want = (x.double() @ dense.t()).repeat(1, again)[:, :N] + bias.double()
    assert _off(out, want) < 8e-3  # (as test_packed_gemm_tiles)
    assert _worst(out, want) < 3e-2  # roundings alone: a row or column of 200 values or more is within a few times the whole
    out.fill_(7.0)
    assert (room == 7.0).all()


def _take(monkeypatch, C, which):
    """Which sequences the tcgen05 kernel takes, whatever the estimates say."""
    monkeypatch.setattr(C, "_long_portions", lambda q, kv, layer, meta, *a: [i for i, (n, _) in enumerate(meta.host_lens) if which(i, n)])


@pytest.mark.parametrize("kvd,hd,nq,nkv,lens,window", [
    ("bf16", 128, 8, 2, LONG, 0), ("bf16", 64, 4, 4, LONG, 0), ("bf16", 128, 7, 1, LONG, 50), ("q8", 64, 4, 1, LONG, 90), ("q4", 128, 8, 2, LONG, 0),
    ("f16", 128, 8, 2, [(40, 400), (1, 30), (64, 64), (33, 1200)], 0), ("q8", 128, 8, 8, [(40, 400), (1, 30), (64, 64), (33, 1200)], 300),
    ("bf16", 64, 4, 2, [(33 + i % 5, 40 + 3 * i) if i % 9 else (1 + i % 3, 20 + i) for i in range(90)], 0),
    ("q8", 64, 4, 2, [(33 + i % 5, 40 + 3 * i) if i % 9 else (1 + i % 3, 20 + i) for i in range(90)], 70)])
@pytest.mark.parametrize("some", [False, True])
def test_steps_between_the_two_kernels(C, monkeypatch, kvd, hd, nq, nkv, lens, window, some):
    """All long portions, or every other one, among short ones; more of them than a launch lists, more sequences than a mask word holds."""
    _take(monkeypatch, C, lambda i, n: n >= 32 and not (some and i % 2))
    cpu, meta, gpu, on_gpu, q = _step(kvd, hd, nq, nkv, lens)
    got = C.paged_attention(q.cuda(), gpu, 0, on_gpu, hd ** -0.5, window)
    _check_status(C)
    want = ref.paged_attention(q.float(), cpu, 0, meta, hd ** -0.5, window)
    assert _off(got, want) < (2.5e-3 if kvd == "bf16" else 6e-3)  # (as test_long_portions)
    off, at = (got.double().cpu() - want.double()).flatten(1), 0
    for n, _ in lens:  # no sequence is left out
        assert off[at : at + n].norm() / want[at : at + n].double().norm() < 8e-3
        at += n


@pytest.mark.parametrize("kvd", ["bf16", "q8"])
@pytest.mark.parametrize("gates", [None, "head", "value"])
@pytest.mark.parametrize("sinks", [False, True])
def test_long_portions_with_sinks_and_gates(C, monkeypatch, kvd, gates, sinks):
    """Against the plain statement: a logit per head in the denominator, a gate per head or per value, a factor on all."""
    from types import SimpleNamespace

    _take(monkeypatch, C, lambda i, n: n >= 32)
    cpu, meta, gpu, on_gpu, q = _step(kvd, 128, 8, 2, LONG)
    gen = torch.Generator().manual_seed(5)
    sink = torch.randn(8, generator=gen) * 2 if sinks else None
    gate = None if gates is None else torch.randn(q.shape[0], 8 if gates == "head" else 1024, generator=gen).bfloat16()
    got = C.paged_attention(q.cuda(), gpu, 0, on_gpu, 128 ** -0.5, sink=None if sink is None else sink.cuda(), out_scale=0.5,
                            gate=None if gate is None else gate.cuda(), gate_per_value=gates == "value")
    _check_status(C)
    want = ref.paged_attention(q.float(), cpu, 0, meta, 128 ** -0.5, sink=sink) * 0.5
    if gates is not None:
        want = ref.head_gate(want, gate, SimpleNamespace(heads=8, width=128, gate=gates))
    assert _off(got, want) < (2.5e-3 if kvd == "bf16" else 6e-3)  # (as test_long_portions)


@pytest.mark.parametrize("kvd", ["q8", "q4", "f16"])
def test_long_portions_without_room_for_converted_pages(C, monkeypatch, kvd):
    """An allocation that fails sends the step to the kernel that needs none."""
    _take(monkeypatch, C, lambda i, n: n >= 32)
    cpu, meta, gpu, on_gpu, q = _step(kvd, 128, 8, 2, LONG)
    asked = []

    def none_left(*size, **more):
        if more.get("dtype") is torch.bfloat16:
            asked.append(size)
            raise torch.OutOfMemoryError("no room")
        return torch.empty(*size, **more)

    with monkeypatch.context() as m:
        m.setattr(C, "torch", _Without(torch, empty=none_left))
        m.setattr(C.scratch(torch.device("cuda")), "guards", None)
        got = C.paged_attention(q.cuda(), gpu, 0, on_gpu, 128 ** -0.5, splits=None, out=torch.zeros_like(q.cuda()))
    _check_status(C)
    assert len(asked) == 1
    assert _off(got, ref.paged_attention(q.float(), cpu, 0, meta, 128 ** -0.5)) < 6e-3  # (as test_long_portions)


class _Without:
    """A module with some of its names replaced."""

    def __init__(self, module, **names):
        self.__dict__.update(names)
        self._module = module

    def __getattr__(self, name):
        return getattr(self._module, name)


@pytest.mark.parametrize("qtype,K", [("Q8_0", 512), ("Q8_0", 1536), ("Q8_0", 3584), ("Q6_K", 1024), ("Q6_K", 3072), ("Q6_K", 2048), ("Q4_K", 2048),
                                     ("Q4_K", 6144)])
@pytest.mark.parametrize("T,N", [(1, 1), (2, 33), (1, 4737), (2, 9473)])
def test_packed_gemv_stream(C, qtype, K, T, N):
    """Rows that end inside a segment, rings that wrap and that do not fill, rows that are no pairs or one for every warp and one more;
    against the same activations in 8 bits, so that only sums and the output are rounded."""
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    some = 257
    w = qtensor_from_dense((torch.randn(some, K, generator=gen, device="cuda") * 0.05).cpu(), qtype, device="cuda")
    dense = w.to("cpu").dense_cache().double().cuda()
    again = -(-N // some)
    w.data, w.shape, w._dense = w.data.repeat(again, 1)[:N].contiguous(), (N, K), None
    x = torch.randn(T, K, generator=gen, device="cuda").bfloat16()
    x[0, : K // 4] = 0
    codes = x.float().view(T, -1, 32)
    step = codes.abs().amax(-1, keepdim=True) / 127
    codes = (torch.round(torch.where(step > 0, codes / step, 0)).double() * step.double()).view(T, K)
    room = torch.full((T + 2, N + 3), 7.0, dtype=torch.bfloat16, device="cuda")
    from oxidize_b200.ops import cuda_quant

    C.configure(C.KernelOptions(gemv_wide=True))
    try:
        cuda_quant.linear_quant(x, w, room[1 : T + 1, 1 : N + 1], None, room.stride(0))
    finally:
        C.configure(C.KernelOptions())
    _check_status(C)
    got, want = room[1 : T + 1, 1 : N + 1].double(), (codes @ dense.t()).repeat(1, again)[:, :N]
    # the output to bf16 (2^-9); a code of 8 bits may fall to the other side where a value lies between two (1 / 254 of 32 values' largest)
    assert ((got - want).abs() <= want.abs() * 2 ** -8 + 0.01 * want.square().mean().sqrt()).all()
    room[1 : T + 1, 1 : N + 1] = 7.0
    assert (room == 7.0).all()


@pytest.mark.parametrize("kvd", ["bf16", "f32", "q8", "q4"])
@pytest.mark.parametrize("hd,pairing,norm", [(64, "split_half", False), (64, "adjacent", True), (128, "split_half", True), (128, "adjacent", False),
                                             (256, "split_half", True), (256, "adjacent", True)])
def test_both_rotation_kernels_write_the_same_bits(C, kvd, hd, pairing, norm):
    """Queries on an 8-byte boundary take the kernel of one value to a thread, the same on a 16-byte one a warp to a head."""
    from types import SimpleNamespace

    gen = torch.Generator().manual_seed(hd)
    T, nq, nkv = 77, 5, 2
    qkv = torch.randn(T, (nq + 2 * nkv) * hd, generator=gen).bfloat16()
    norms = [(torch.rand(hd, generator=gen) + 0.5).cuda() if norm else None for _ in range(2)]
    pos, slots = (torch.arange(T, dtype=torch.int32, device="cuda") * 31, torch.arange(T, dtype=torch.int32, device="cuda"))
    rope = SimpleNamespace(inv_freq=ref.rope_inv_freq(hd, 10000.0, None, device="cuda"), pairing=pairing, mscale=1.0, n_heads=nq,
                           n_kv_heads=nkv, head_dim=hd, max_pos=0)
    seen = []
    for offset in (0, 4):
        room = torch.empty(qkv.numel() + 4, dtype=torch.bfloat16, device="cuda")
        at = room[offset : offset + qkv.numel()].view(qkv.shape)
        at.copy_(qkv)
        kv = KVCache(KVCacheSpec(1, nkv, hd, 16, kvd), 8, torch.device("cuda"))
        for d in kv.data + [s for s in kv.scales if s is not None]:
            d.zero_()
        q = C.qk_rope_kv_write(at, pos, slots, kv, 0, rope, *norms, 1e-6)
        seen.append([q, kv.data[0]] + ([] if kv.scales[0] is None else [kv.scales[0]]))
    _check_status(C)
    assert all(torch.equal(a, b) for a, b in zip(*seen))


@pytest.mark.parametrize("kvd", ["bf16", "q8"])
def test_long_portions_as_they_are_dispatched(C, kvd):
    """A prompt that fills the SMs takes the tcgen05 kernel, the tail of a long one beside it does not; a step that is built anew on the
    same object is looked at anew."""
    lens = [(40, 12000), (500, 500)]
    cpu, meta, gpu, on_gpu, q = _step(kvd, 128, 32, 8, lens)
    q = q.cuda()
    assert C._long_portions(q, gpu, 0, on_gpu, 0.09, 0) == [1]
    got = C.paged_attention(q, gpu, 0, on_gpu, 0.09)
    _check_status(C)
    want = ref.paged_attention(q.float().cpu(), cpu, 0, meta, 0.09)
    assert _off(got, want) < (2.5e-3 if kvd == "bf16" else 6e-3)  # (as test_long_portions)
    assert C._long_portions(q, gpu, 0, on_gpu, 0.09, 0) == [1]
    on_gpu.host_lens = [(600, 700), (5, 60)]
    assert C._long_portions(q, gpu, 0, on_gpu, 0.09, 0) == [0]
    on_gpu.host_lens = None
    assert C._long_portions(q, gpu, 0, on_gpu, 0.09, 0) == []
