"""Decode-time kernels and the inference engine against fp32 PyTorch references."""
import pytest
import torch

from scirust_b200.models import GQADecoder, SciAgentConfig
from scirust_b200.models.infer import InferenceEngine, reference_generate
from scirust_b200 import ops
from scirust_b200.ops import _lib, decode as D, gemm as _g

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _r(shape, seed, scale=0.5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(BF)


@pytest.mark.parametrize("M,K,N", [(1, 1024, 1536), (3, 4096, 512), (8, 2816, 1024), (13, 1024, 264),
                                   (8, 14336, 520), (2, 40, 8), (1, 4096, 6144), (16, 4096, 1024), (27, 2816, 520),
                                   (32, 14336, 256), (45, 1024, 512)])
def test_gemv_bf16(M, K, N):
    x, w, r = _r((M, K), 1), _r((K, N), 2), _r((M, N), 3)
    y = D.gemv(x, w, residual=r)
    ref = x.float() @ w.float() + r.float()
    assert (y.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    assert torch.equal(y, D.gemv(x, w, residual=r))
    f = torch.empty((M, N), dtype=torch.float32, device="cuda")
    D.gemv(x, w, out_f32=f)
    assert (f - x.float() @ w.float()).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("M,K,N", [(1, 1024, 1536), (5, 4096, 512), (8, 1024, 2048), (7, 14336, 528)])
def test_gemv_int8_and_quantize(M, K, N):
    x, w = _r((M, K), 4), _r((K, N), 5)
    qw = D.quantize_per_channel(w)
    qc = D.quantize_per_channel(w.cpu())
    assert torch.allclose(qw.scale.cpu(), qc.scale, rtol=1e-6)
    assert (qw.q.cpu().int() - qc.q.int()).abs().max().item() <= 1   # bf16 half-way cases may round either way
    y = D.gemv(x, qw)
    ref = x.float() @ (qw.q.float() * qw.scale[None, :])
    assert (y.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    assert (qw.dequantize().float() - qw.q.float() * qw.scale[None, :]).abs().max().item() <= 1e-2


@pytest.mark.parametrize("quant", [False, True])
def test_gemv_of_no_rows_is_empty(quant):
    """As on the CPU: an empty result and no launch."""
    w = _r((256, 512), 2)
    w = D.quantize_per_channel(w) if quant else w
    launched = _g.launch_count
    assert tuple(D.gemv(_r((0, 256), 1), w, residual=_r((0, 512), 3)).shape) == (0, 512)
    assert tuple(D.gemv(_r((0, 512), 1), w, swiglu=True).shape) == (0, 512)
    f = torch.empty((0, 512), device="cuda")
    assert D.gemv(_r((0, 256), 1), w, out_f32=f, rms_weight=_r((256,), 4)) is f
    assert _g.launch_count == launched


@pytest.mark.parametrize("dh,H,Hkv", [(64, 16, 4), (128, 32, 8), (128, 4, 4), (64, 16, 2), (128, 16, 1)])
def test_paged_decode_attention(dh, H, Hkv):
    B, page, max_seq = 3, 16, 700
    max_blocks = (max_seq + page - 1) // page
    n_blocks = B * max_blocks
    pool = torch.zeros((n_blocks, 2, Hkv, page, dh), dtype=BF, device="cuda")
    perm = torch.randperm(n_blocks, generator=torch.Generator().manual_seed(0)).int()
    table = perm.reshape(B, max_blocks).cuda()          # scattered physical pages
    lens = torch.tensor([1, 257, 700], dtype=torch.int32, device="cuda")
    ld = (H + 2 * Hkv) * dh
    for b in range(B):
        L = int(lens[b])
        rows = _r((L, ld), 10 + b)
        D.kv_append(rows, H, Hkv, dh, pool, table, page, torch.full((L,), b, dtype=torch.int32, device="cuda"),
                    torch.arange(L, dtype=torch.int32, device="cuda"))
    q = _r((B, ld), 20)
    out = D.decode_attention(q, pool, table, page, lens, H, Hkv, dh, n_splits=5)
    ref = D.decode_attention_ref(q, pool, table, page, lens, H, Hkv, dh)
    assert (out.float() - ref).abs().max().item() < 2e-2
    one = D.decode_attention(q, pool, table, page, lens, H, Hkv, dh, n_splits=1)
    assert (one.float() - ref).abs().max().item() < 2e-2
    assert torch.equal(out, D.decode_attention(q, pool, table, page, lens, H, Hkv, dh, n_splits=5))


def test_argmax_tie_and_nan_rules():
    V = 10000
    lg = torch.randn(8, V, device="cuda")
    lg[0, 77] = 50.0
    lg[0, 9000] = 50.0          # tie -> lower id
    lg[1, 5] = float("nan")     # a NaN past column 0 is skipped
    lg[1, 4100] = 60.0
    lg[2] = -5.0
    lg[2, 8191] = -4.0
    lg[4, 0] = float("nan")     # NaN in column 0: the greedy loop starts from it and nothing compares greater
    lg[4, 300] = 99.0
    lg[5, 4096] = float("nan")  # first element of the second slab
    lg[5, 4097] = 70.0
    lg[6] = float("nan")        # no number at all
    lg[7, 4096] = float("nan")  # the maximum sits in the first slab, the second slab starts with a NaN
    lg[7, 17] = 80.0
    tok = D.argmax_rows(lg).tolist()
    assert tok[:3] == [77, 4100, 8191]
    assert tok[3] == int(torch.argmax(lg[3]))
    assert tok[4:] == [0, 4097, 0, 17]
    # the host statement of the same rule agrees row by row
    assert D.argmax_rows(lg.cpu()).tolist() == tok


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("M,K,N,splits", [(1, 1024, 50272, 1), (5, 2048, 4112, 4), (8, 512, 1024, None)])
def test_lm_head_fused_with_argmax_equals_gemv_then_argmax(quant, M, K, N, splits):
    """One launch (GEMV + in-kernel arg-max) gives the tokens and the logits of the three-launch path, including the
    NaN rules: weights with NaN columns make NaN logits in column 0 (row wins token 0), column 7 (skipped)."""
    g = torch.Generator(device="cuda").manual_seed(M * 31 + K)
    x = (torch.randn(M, K, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    w = (torch.randn(K, N, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    gain = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16)
    w[:, N - 3] = w[:, 40]                          # a tie between two columns when x.w is the row maximum
    cases = [w]
    if not quant:
        wn = w.clone(); wn[0, 7] = float("nan"); cases.append(wn)           # NaN logits in column 7: skipped
        w0 = w.clone(); w0[0, 0] = float("nan"); cases.append(w0)           # NaN logits in column 0: token 0
    for wc in cases:
        wt = D.quantize_per_channel(wc) if quant else wc
        lg = torch.empty(M, N, dtype=torch.float32, device="cuda")
        D.gemv(x, wt, out_f32=lg, rms_weight=gain, splits=splits)
        want = D.argmax_rows(lg)
        lg2 = torch.zeros_like(lg)
        got = D.gemv_argmax(x, wt, rms_weight=gain, logits=lg2, splits=splits)
        nolog = D.gemv_argmax(x, wt, rms_weight=gain, splits=splits)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(nolog, want)
        nan = torch.isnan(lg)
        assert torch.equal(torch.isnan(lg2), nan) and torch.equal(lg2[~nan], lg[~nan])
    if not quant:
        assert got.tolist() == [0] * M
    _lib.check_status(torch.device("cuda"))


@pytest.mark.parametrize("quant", [None, "int8"])
def test_engine_cached_equals_naive_and_graph(quant):
    cfg = SciAgentConfig(vocab_size=1024, d_model=256, n_layers=2, n_heads=4, n_kv_heads=2, d_ff=512,
                         max_seq_len=512, rope_theta=10000.0)
    model = GQADecoder(cfg, device="cuda", seed=5, init_std=0.08)
    prompts = torch.randint(1, 1024, (2, 128), generator=torch.Generator().manual_seed(1)).cuda()
    eager = InferenceEngine(model, quant=quant, max_batch=2, max_seq=256, page=16, use_graph=False)
    graph = InferenceEngine(model, quant=quant, max_batch=2, max_seq=256, page=16, use_graph=True)
    a = eager.generate(prompts, 8)
    b = graph.generate(prompts, 8)
    _lib.check_status()
    assert torch.equal(a, b)
    if quant is None:
        naive = reference_generate(model, prompts, 8)
        assert torch.equal(a, naive), (a.tolist(), naive.tolist())


@pytest.mark.parametrize("M,K,N", [(16, 1024, 512), (64, 4096, 1536), (200, 1000, 272), (2048, 1024, 2816)])
def test_dequant_fused_gemm(M, K, N):
    x, w, r = _r((M, K), 6), _r((K, N), 7), _r((M, N), 8)
    qw = D.quantize_per_channel(w)
    ref = x.float() @ (qw.q.float() * qw.scale[None, :]) + r.float()
    y = D.matmul_w8(x, qw, residual=r)
    _lib.check_status()
    assert (y.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    y2 = D.matmul_w8(x, qw, residual=r, splits=4)
    _lib.check_status()
    assert (y2.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    assert torch.equal(y2, D.matmul_w8(x, qw, residual=r, splits=4))


@pytest.mark.parametrize("M,K,N,splits", [(16, 4096, 1024, None), (64, 512, 768, 1), (200, 1040, 264, 3), (9, 128, 8, None)])
def test_w8a8_gemm_on_integer_tensor_cores_is_exact(M, K, N, splits):
    """tcgen05.mma.kind::i8: int8 x int8 -> int32 is exact, so the kernel must reproduce the host statement of the
    reference's quantised linear layer (dynamic row scales, int64 accumulation, one rescale) to the last bf16 bit,
    whatever the split-K factor; and it stays close to the unquantised product."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = (torch.randn(M, K, generator=g, device="cuda") * 0.7).to(torch.bfloat16)
    w = (torch.randn(K, N, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    r = (torch.randn(M, N, generator=g, device="cuda") * 0.3).to(torch.bfloat16)
    wq = D.quantize_per_channel(w)
    xq, sx = D.quantize_rows(x)
    xq_ref, sx_ref = D.quantize_rows(x.cpu())
    assert torch.equal(xq.cpu(), xq_ref) and torch.equal(sx.cpu(), sx_ref)
    acc = xq.cpu().to(torch.int64) @ wq.q.cpu().to(torch.int64)
    want = (acc.float() * (sx_ref[:, None] * wq.scale.cpu()[None, :]) + r.cpu().float()).to(torch.bfloat16)
    got = D.matmul_w8a8(x, wq, residual=r, splits=splits)
    torch.cuda.synchronize()
    assert torch.equal(got.cpu(), want)
    again = D.matmul_w8a8(x, wq, residual=r, splits=2 if K >= 256 else 1)
    assert torch.equal(again, got)                        # split-K adds integers: same bits
    full = x.float() @ w.float() + r.float()
    assert (got.float() - full).abs().max().item() <= 0.04 * full.abs().max().item()
    _lib.check_status(torch.device("cuda"))


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("M,K,N,splits", [(16, 4096, 1024, 0), (9, 320, 264, 1), (33, 1040, 4104, 3), (64, 512, 128, 0),
                                          (12, 128, 19200, 0)])
def test_skinny_weight_streaming_gemm_matches_reference(quant, M, K, N, splits):
    """9..64 rows on the swapped-operand tcgen05 kernel (weights as the 128-row operand, C^T in tensor memory):
    bf16 against the fp32 product, int8 (W8A8) bit for bit against the integer statement; ragged N and K, one and
    several work items per CTA, explicit and automatic split-K; two runs agree bit for bit."""
    if quant and K % 16:
        K = (K + 15) // 16 * 16
    g = torch.Generator(device="cuda").manual_seed(M * 7 + K)
    x = (torch.randn(M, K, generator=g, device="cuda") * 0.7).to(torch.bfloat16)
    w = (torch.randn(K, N, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    r = (torch.randn(M, N, generator=g, device="cuda") * 0.3).to(torch.bfloat16)
    if quant:
        wq = D.quantize_per_channel(w)
        xq, sx = D.quantize_rows(x.cpu())
        acc = xq.to(torch.int64) @ wq.q.cpu().to(torch.int64)
        want = (acc.float() * (sx[:, None] * wq.scale.cpu()[None, :]) + r.cpu().float()).to(torch.bfloat16)
        got = D.matmul_skinny(x, wq, residual=r, splits=splits)
        torch.cuda.synchronize()
        assert torch.equal(got.cpu(), want)
        assert torch.equal(D.matmul_skinny(x, wq, residual=r, splits=splits), got)
    else:
        ref = x.float() @ w.float() + r.float()
        got = D.matmul_skinny(x, w, residual=r, splits=splits)
        torch.cuda.synchronize()
        err = (got.float() - ref).abs()
        tol = ref.abs() * 2.0 ** -7 + 2.0 ** -14 * 0.035 * 0.8 * K + 1e-3
        assert bool((err <= tol).all()), float((err - tol).max())
        assert torch.equal(D.matmul_skinny(x, w, residual=r, splits=splits), got)
        plain = D.matmul_skinny(x, w, splits=1)
        assert (plain.float() - x.float() @ w.float()).abs().max().item() <= 0.02 * max(1.0, (x.float() @ w.float()).abs().max().item())
    _lib.check_status(torch.device("cuda"))


def test_driver_smoke_entry_runs_training_decode_and_batched_decode():
    """The entry point the round-end driver calls: a few training steps, a cached decode, and 12-sequence decodes with
    bf16 and int8 weights (the weight-streaming GEMM and its W8A8 form)."""
    import __graft_entry__ as entry
    entry.smoke()


@pytest.mark.parametrize("K,N", [(1, 8), (7, 24), (8, 2048), (65, 4104), (9, 20), (33, 13)])
def test_dequantize_is_the_rounded_product(K, N):
    """Whole 8-byte words (one thread per eight columns, eight rows at a time) and rows that are not: the same bits as
    bf16(code * scale)."""
    g = torch.Generator(device="cuda").manual_seed(K + N)
    q = torch.randint(-128, 128, (K, N), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    scale = torch.rand(N, generator=g, device="cuda") * 0.01 + 1e-4
    want = (q.float() * scale[None, :]).to(BF)
    assert torch.equal(D.QuantWeight(q, scale).dequantize(), want)


@pytest.mark.parametrize("dh,H,Hkv", [(128, 32, 8), (128, 16, 1), (128, 3, 3), (128, 8, 1)])
@pytest.mark.parametrize("page", [8, 16, 32, 64, 192])
def test_paged_decode_attention_stream(dh, H, Hkv, page, monkeypatch):
    """The balanced tile stream (no explicit split count): ragged lengths around the 64-position tile, an empty and a
    one-position sequence, jobs inside one CTA and across many, several page sizes; positions past the end and pages of
    nobody hold NaN and must not be seen."""
    monkeypatch.setattr(D, "_stream_wins", lambda *a: True)
    for lens in ([0, 1, 63, 64, 65, 700], [1500], [200] * 40):
        B, longest = len(lens), max(lens)
        max_blocks = (longest + page - 1) // page
        n_blocks = B * max_blocks + 3
        pool = torch.full((n_blocks, 2, Hkv, page, dh), float("nan"), dtype=BF, device="cuda")
        table = torch.randperm(n_blocks, generator=torch.Generator().manual_seed(page))[:B * max_blocks].int()
        table = table.reshape(B, max_blocks).cuda()
        ld = (H + 2 * Hkv) * dh
        for b, L in enumerate(lens):
            if L:
                D.kv_append(_r((L, ld), 10 + b), H, Hkv, dh, pool, table, page,
                            torch.full((L,), b, dtype=torch.int32, device="cuda"),
                            torch.arange(L, dtype=torch.int32, device="cuda"))
        ln = torch.tensor(lens, dtype=torch.int32, device="cuda")
        q = _r((B, ld), 20)
        out = D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, max_len=longest)
        ref = D.decode_attention_ref(q, pool.nan_to_num(0.0), table, page, ln.clamp(min=1), H, Hkv, dh)
        ref[ln == 0] = 0.0
        assert (out.float() - ref).abs().max().item() < 2e-2
        assert torch.equal(out, D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, max_len=longest))
        one = D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, n_splits=1)
        assert (out.float() - one.float()).abs().max().item() < 2e-2
    _lib.check_status(torch.device("cuda"))


@pytest.mark.parametrize("H,Hkv", [(4, 1), (5, 1), (14, 2), (16, 1)])
def test_decode_attention_stream_of_jobs_that_share_a_cta(H, Hkv):
    """Two tiles to a CTA and lengths that differ, so that CTAs end one job and begin the next: with more than four query heads the
    consumers help to merge the last piece, and the job of the first may be put off behind it. Whichever CTA comes last, the sums are the same."""
    dh, page = 128, 64
    g = torch.Generator().manual_seed(H)
    for B, longest in ((2, 2048), (3, 1500), (9, 300), (2, 700)):
        max_blocks = (longest + page - 1) // page
        pool = _r((B * max_blocks, 2, Hkv, page, dh), 3)
        table = torch.randperm(B * max_blocks, generator=g).int().reshape(B, max_blocks).cuda()
        q = _r((B, (H + 2 * Hkv) * dh), 20)
        for _ in range(4):
            lens = torch.randint(1, longest + 1, (B,), generator=g).int().cuda()
            out, *again = (D.decode_attention(q, pool, table, page, lens, H, Hkv, dh, max_len=longest, stream=True) for _ in range(6))
            assert all(torch.equal(out, o) for o in again)
            ref = D.decode_attention_ref(q, pool, table, page, lens, H, Hkv, dh)
            assert (out.float() - ref).abs().max().item() < 2e-2
    _lib.check_status(torch.device("cuda"))


def test_decode_attention_stream_repeats_under_load(monkeypatch):
    """The ring of the streamed attention refills a stage only after all eight consumer warps have passed its fill: many
    repetitions over long sequences give the same bits, and no bounded wait runs out."""
    monkeypatch.setattr(D, "_stream_wins", lambda *a: True)
    B, L, H, Hkv, dh, page = 48, 1600, 32, 8, 128, 64
    nb = L // page
    pool = _r((B * nb, 2, Hkv, page, dh), 1)
    table = torch.randperm(B * nb, generator=torch.Generator().manual_seed(2)).int().reshape(B, nb).cuda()
    ln = torch.randint(L // 2, L + 1, (B,), generator=torch.Generator().manual_seed(3)).int().cuda()
    q = _r((B, (H + 2 * Hkv) * dh), 4)
    first = D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, max_len=L)
    for _ in range(300):
        last = D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, max_len=L)
    assert torch.equal(first, last)
    _lib.check_status(torch.device("cuda"))


@pytest.mark.parametrize("graph", [True, False])
def test_generation_chooses_attention_by_what_the_cache_holds(graph, monkeypatch):
    """The engine asks for the streamed kernel once the sequences are long enough, whatever they may grow to: a generation
    that crosses the line runs the split kernel before it and the stream after it, replayed or not, and one that ends soon
    after the line keeps its kernel."""
    torch.manual_seed(0)
    model = GQADecoder(SciAgentConfig(512, 512, 2, 4, 1, 512, 256, 1e4), device="cuda")
    prompts = torch.randint(0, 512, (3, 20), generator=torch.Generator().manual_seed(1))
    monkeypatch.setattr(D, "_stream_wins", lambda L, *a: L >= 30)
    asked = []
    real = D.decode_attention
    monkeypatch.setattr(D, "decode_attention", lambda *a, **k: (asked.append(k["stream"]), real(*a, **k))[1])
    out = {}
    for recapture in (8, 100):
        eng = InferenceEngine(model, max_batch=3, max_seq=128, page=64, use_graph=graph)
        eng.RECAPTURE_STEPS = recapture
        asked.clear()
        out[recapture] = eng.generate(prompts, 40).cpu()
        # two layers a step; a graph runs each kernel eagerly once and records it once
        per = {False: 4, True: 4} if graph else {False: 9 * 2, True: 30 * 2}
        want = per if recapture == 8 else {False: 4 if graph else 39 * 2, True: 0}
        assert {r: asked.count(r) for r in (False, True)} == want
    a = InferenceEngine(model, max_batch=3, max_seq=128, page=64, use_graph=not graph)
    a.RECAPTURE_STEPS = 8
    assert torch.equal(a.generate(prompts, 40).cpu(), out[8])
    assert (out[8] == out[100]).float().mean().item() > 0.5      # the kernels differ by roundings, which may flip a near-tie


def test_decode_attention_stream_without_weight_is_zero():
    """A sequence whose scores are all NaN has no weight: zeros, as from the split kernel, also where its values are NaN
    and its tiles are spread over many CTAs."""
    H, Hkv, dh, page = 8, 2, 128, 64
    lens = [1500, 40, 300]
    nb = (max(lens) + page - 1) // page
    pool = _r((3 * nb, 2, Hkv, page, dh), 1)
    table = torch.arange(3 * nb, dtype=torch.int32, device="cuda").reshape(3, nb)
    pool[table[0].long()] = float("nan")
    pool[table[1].long()] = float("nan")
    ln = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = _r((3, (H + 2 * Hkv) * dh), 2)
    out = D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, stream=True)
    one = D.decode_attention(q, pool, table, page, ln, H, Hkv, dh, stream=False)
    assert (one[:2] == 0).all() and (out[:2] == 0).all()
    assert (out[2].float() - one[2].float()).abs().max().item() < 2e-2


@pytest.mark.parametrize("rows,quant", [(1, False), (8, True), (9, False), (33, True), (64, False)])
def test_dependent_launches_read_what_their_predecessor_wrote(rows, quant):
    """A row norm, a product whose weights a copy has just written, and SwiGLU give, launch for launch, the bits of plain stream
    order. (The copies are not launched dependently; the chains of the next test have none.)"""
    K, N = 1024, 1536
    g = torch.Generator(device="cuda").manual_seed(rows)
    gain = torch.ones(K, dtype=torch.bfloat16, device="cuda")
    xs = [torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4)]
    ws = [(torch.randn(K, N, generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(4)]
    qs = [D.quantize_per_channel(w) for w in ws]
    for q in qs:
        q.transposed()

    def chain():
        w = D.QuantWeight(qs[0].q.clone(), qs[0].scale.clone()) if quant else ws[0].clone()
        if quant:
            w.transposed()
        out = []
        for i in range(12):
            x = ops.rmsnorm_fwd(xs[i % 4], gain, 1e-5, want_inv=False)[0]
            if quant:
                w.scale.copy_(qs[i % 4].scale)
                w.q.copy_(qs[i % 4].q)
                w.transposed().copy_(qs[i % 4].transposed())
            else:
                w.copy_(ws[i % 4])
            y = D.gemv(x, w, rms_weight=gain) if rows <= 8 else D.matmul_skinny(x, w)
            out.append(ops.swiglu_fwd(y))
        return torch.stack(out)

    got = chain()
    _lib.call("sb_set_pdl", 0)
    try:
        want = chain()
    finally:
        _lib.call("sb_set_pdl", 1)
    assert torch.equal(got, want)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("rows,quant,stream", [(1, False, False), (8, True, True), (9, False, True), (16, True, False),
                                               (64, False, False), (64, True, True)])
def test_chains_of_dependent_launches_give_the_bits_of_plain_stream_order(rows, quant, stream, graph):
    """Decoder layers fed back into themselves, without any other kernel between: every kernel reads what the one right before it
    has just written, at addresses that held another step's values before (product -> rotation and append -> attention -> product
    -> norm -> product with split sums in memory -> SwiGLU -> product -> norm)."""
    d, H, Hkv, dh, ff, page, past, steps = 1024, 8, 2, 128, 3072, 64, 300, 8
    ws = [_r(s, 10 + i, 0.05) for i, s in enumerate([(d, (H + 2 * Hkv) * dh), (d, d), (d, 2 * ff), (ff, d)])]
    if quant:
        ws = [D.quantize_per_channel(w) for w in ws]
        for w in ws:
            w.transposed()
    gain, x0 = _r((d,), 1) + 1, _r((rows, d), 2)
    cos, sin = ops.rope_table(512, dh, 1e4, torch.device("cuda"))
    nb = (past + steps + page - 1) // page
    table = torch.arange(rows * nb, dtype=torch.int32, device="cuda").reshape(rows, nb)
    pool0 = _r((rows * nb, 2, Hkv, page, dh), 3)
    seq_of = torch.arange(rows, dtype=torch.int32, device="cuda")
    pos = [torch.full((rows,), past + i, dtype=torch.int32, device="cuda") for i in range(steps)]
    lens = [p + 1 for p in pos]
    if rows > 8 and not quant:
        assert D._skinny_launches(x0.device, rows, 2 * ff, d, False, 3) == 2       # clusters of three for 48 tiles do not fit

    def linear(x, w):
        return D.gemv(x, w) if rows <= 8 else D.matmul_skinny(x, w)

    def chain():
        pool, x, out = pool0.clone(), x0, []
        for i in range(steps):
            qkv = linear(x, ws[0])
            D.rope_kv_append(qkv, H, Hkv, dh, cos, sin, pool, table, page, seq_of, pos[i])
            a = D.decode_attention(qkv, pool, table, page, lens[i], H, Hkv, dh, stream=stream)
            h = ops.rmsnorm_fwd(linear(a, ws[1]), gain, 1e-5, want_inv=False)[0]
            x = ops.rmsnorm_fwd(linear(ops.swiglu_fwd(linear(h, ws[2])), ws[3]), gain, 1e-5, want_inv=False)[0]
            out.append(x)
        return torch.stack(out), pool

    def run():
        if not graph:
            return chain()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            chain()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                out = chain()
        torch.cuda.current_stream().wait_stream(side)
        g.replay()
        g.replay()
        return [t.clone() for t in out]

    got = run()
    _lib.call("sb_set_pdl", 0)
    try:
        want = run()
    finally:
        _lib.call("sb_set_pdl", 1)
    _lib.check_status()
    assert got[0].isfinite().all() and len({bytes(t.view(torch.uint8).cpu().numpy().tobytes()) for t in got[0]}) == steps
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("M,K,N,splits", [(1, 1024, 264 + 8, 8), (8, 992, 1552, 8), (3, 4096, 4096, 8), (5, 200, 16, 3),
                                          (1, 2816, 1024, 8), (8, 14336, 4096, 8), (2, 4096, 22016, 3), (7, 4096, 28672, 5),
                                          # clusters of half blocks that do not fit at once, of whole blocks that do not
                                          (1, 1024, 4608, 8), (2, 512, 9728, 8), (5, 512, 24576, 8)])
def test_splits_that_finish_in_a_cluster_give_the_bits_of_the_finish_through_memory(quant, M, K, N, splits):
    """Grids of narrow and of wide column blocks, ragged last blocks, k ranges that end inside a tile: the fused LM head keeps
    the finish through memory, adds in the same order and so has the same logits; an output and a residual at odd addresses
    give the bits of aligned ones."""
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    x = (torch.randn(M, K, generator=g, device="cuda") * 0.5).to(BF)
    w = (torch.randn(K, N, generator=g, device="cuda") * 0.05).to(BF)
    wt = D.quantize_per_channel(w) if quant else w
    lg, lg2 = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    D.gemv(x, wt, out_f32=lg, splits=splits)
    D.gemv_argmax(x, wt, logits=lg2, splits=splits)
    assert torch.equal(lg, lg2)
    ref = x.double() @ (wt.q.double() * wt.scale.double() if quant else w.double())
    assert ((lg.double() - ref).norm() / ref.norm()).item() < 1e-5       # fp32 sums of exact products
    r = torch.randn(M, N + 1, generator=g, device="cuda").to(BF)
    wide = torch.empty(M, N + 3, dtype=BF, device="cuda")
    D.gemv(x, wt, residual=r[:, 1:], out=wide[:, 1:N + 1], splits=splits)
    assert torch.equal(wide[:, 1:N + 1], D.gemv(x, wt, residual=r[:, 1:].contiguous(), splits=splits))


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("M,K,N,splits", [(9, 1040, 8, 2), (33, 1040, 136, 3), (64, 4096, 4096, 4), (17, 2816, 1544, 5), (64, 4096, 1032, 6),
                                          (48, 4096, 6144, 3)])
def test_skinny_splits_in_a_cluster(quant, M, K, N, splits):
    """Splits that finish inside a cluster (and 48 tiles of three, which do not all fit and finish through memory): int8 sums
    are exact, so any split has the bits of none; bf16 sums against float64. Residual and output at odd addresses."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(BF)
    w = (torch.randn(K, N, generator=g, device="cuda") * 0.05).to(BF)
    r = torch.randn(M, N + 1, generator=g, device="cuda").to(BF)[:, 1:]
    wide = torch.zeros(M, N + 3, dtype=BF, device="cuda")
    wt = D.quantize_per_channel(w) if quant else w
    D.matmul_skinny(x, wt, residual=r, out=wide[:, 1:N + 1], splits=splits)
    got = D.matmul_skinny(x, wt, residual=r.contiguous(), splits=splits)
    assert torch.equal(wide[:, 1:N + 1], got) and not wide[:, 0].any() and not wide[:, N + 1:].any()
    if quant:
        assert torch.equal(got, D.matmul_skinny(x, wt, residual=r, splits=1))
    else:
        ref = x.double() @ w.double() + r.double()
        assert ((got.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8      # one rounding to bf16


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("M,K,N", [(1, 4096, 4096), (8, 2816, 1024), (1, 14336, 4096), (4, 11008, 4096), (1, 4096, 6144)])
def test_sums_of_long_k_ranges_keep_the_precision_of_short_ones(quant, M, K, N):
    """A tensor core cuts its running sum off, so the error of one accumulation grows with its length (1.8e-6 over 1792 rows of k,
    2.4e-7 over 256); accumulations of 128 rows joined by rounded additions stay at that of 128 rows, 1.5e-7 (8e-8 for the 8-bit
    weights of an fp16 product), whatever the splits. The limit leaves a third."""
    g = torch.Generator(device="cuda").manual_seed(K + M)
    x = torch.randn(M, K, generator=g, device="cuda").to(BF)
    w = (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(BF)
    wt = D.quantize_per_channel(w) if quant else w
    out = torch.empty(M, N, device="cuda")
    D.gemv(x, wt, out_f32=out)
    ref = x.double() @ (wt.q.double() * wt.scale.double() if quant else w.double())
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2e-7


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("M,K,N,splits", [(16, 4096, 4096, 0), (64, 4096, 6144, 0), (33, 4096, 22016, 0), (9, 1024, 1536, 0),
                                          (16, 2048, 1024, 7), (16, 100 * 16, 1024, 3)])
def test_launches_of_the_weight_streaming_gemm_are_counted_as_they_are(quant, M, K, N, splits):
    """Partial sums reach the workspace exactly where a second kernel adds them up."""
    x, w = _r((M, K), 1), _r((K, N), 2)
    w = D.quantize_per_channel(w) if quant else w
    D.matmul_skinny(x, w, splits=splits)                       # the workspace and the transposed codes are there
    ws = D._workspace(1, x.device)
    ws.fill_(float("nan"))
    before = _g.launch_count
    D.matmul_skinny(x, w, splits=splits)
    counted = _g.launch_count - before - (1 if quant else 0)   # the row quantiser is one
    assert counted == (1 if ws.isnan().all() else 2)


@pytest.mark.parametrize("M,K", [(3, 8), (16, 1000), (16, 4096), (149, 4096), (9, 4104), (2, 8192), (16, 14336), (148, 4096), (32, 8192),
                                 (33, 8192), (512, 2048), (511, 2048), (1025, 8192)])
def test_row_quantiser_is_the_division_rounded(M, K):
    """Bit for bit the host statement on rows of halfway values, of one size, tiny, huge, denormal and with no number in them: the
    product by 1 / scale decides only where the division would decide the same."""
    g = torch.Generator().manual_seed(K)
    for size in (1.0, 1e-30, 1e-38, 3e-39, 1e-40, 3e38):
        x = (torch.randn((M, K), generator=g).clamp(-1, 1) * size).to(BF)
        x[0] = (torch.arange(K) % 255 - 127).to(BF) * 0.5 * (size if size < 1e30 else 1e30)
        x[0, 0] = 127.0 * (size if size < 1e30 else 1e30)
        x[1] = x[1].abs().max()
        q, s = D.quantize_rows(x.cuda())
        qr, sr = D.quantize_rows(x)
        assert torch.equal(q.cpu(), qr) and torch.equal(s.cpu(), sr)
    x[0], x[1, 0] = float("nan"), float("inf")            # as the division has it: -128 where there is no number
    q, s = D.quantize_rows(x.cuda())
    assert bool((q[0] == -128).all()) and int(q[1, 0]) == -128 and bool((q[1, 1:] == 0).all())
