"""tcgen05 GEMM against a plain fp32 PyTorch reference, all operand forms."""
import pytest
import torch

from scirust_b200 import ops
from scirust_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _mk(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * 0.5).to(torch.bfloat16)


def _check(y, ref, K):
    """Per-element bound: one bf16 rounding of the result (relative 2^-8, taken with a factor two) plus the fp32
    accumulation slack, which grows with sum |a||b| ~ 0.16 K for the N(0, 0.5^2) operands of these tests. A kernel
    that drops one 64-deep k-step is off by ~2 per element and fails this at any K; a bound on max|ref| would not."""
    _lib.check_status()
    err = (y.float() - ref).abs()
    tol = ref.abs() * 2.0 ** -7 + 2.0 ** -14 * 0.16 * K
    bad = err > tol
    assert not bool(bad.any()), f"{int(bad.sum())} elements off, worst {float((err - tol).max()):.4g} over its bound"


def _ints(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2, 3, shape, generator=g, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("M,N", [(256, 256), (384, 520)])
def test_small_integer_operands_are_exact_in_every_form(pair, M, N, monkeypatch):
    """K = 64 with operands in {-2..2} (and all ones): every product and partial sum is an integer below 256,
    exact in fp32 and in bf16, so each operand form must return the integers themselves."""
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "PAIR_MODE", pair)
    K = 64
    for mk in (_ints, lambda shape, seed: torch.ones(shape, dtype=torch.bfloat16, device="cuda")):
        a, b, at, bt = mk((M, K), 1), mk((K, N), 2), mk((K, M), 3), mk((N, K), 4)
        assert torch.equal(ops.matmul_nn(a, b).float(), a.float() @ b.float())
        assert torch.equal(ops.matmul_nt(a, bt).float(), a.float() @ bt.float().t())
        assert torch.equal(ops.matmul_tn(at, b, splits=1).float(), at.float().t() @ b.float())
        assert torch.equal(ops.matmul_tt_a(at, bt).float(), at.float().t() @ bt.float().t())
    _lib.check_status()


SHAPES = [(128, 128, 64), (256, 256, 256), (384, 512, 1024), (200, 264, 136), (2048, 1536, 1024), (1000, 5632, 1024)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_nn(M, N, K):
    x, w = _mk((M, K), 1), _mk((K, N), 2)
    _check(ops.matmul_nn(x, w), x.float() @ w.float(), K)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_nt(M, N, K):
    a, b = _mk((M, K), 3), _mk((N, K), 4)
    _check(ops.matmul_nt(a, b), a.float() @ b.float().t(), K)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_tn(M, N, K):
    a, b = _mk((K, M), 5), _mk((K, N), 6)
    _check(ops.matmul_tn(a, b, splits=1), a.float().t() @ b.float(), K)


@pytest.mark.parametrize("M,N,K", SHAPES[:4])
def test_tt_a(M, N, K):
    a, b = _mk((K, M), 7), _mk((N, K), 8)
    _check(ops.matmul_tt_a(a, b), a.float().t() @ b.float().t(), K)


def test_residual_and_bn128():
    x, w, r = _mk((512, 1024), 1), _mk((1024, 1024), 2), _mk((512, 1024), 9)
    ref = x.float() @ w.float() + r.float()
    _check(ops.matmul_nn(x, w, residual=r), ref, 1024)
    _check(ops.matmul_nn(x, w, residual=r, bn=128), ref, 1024)


def test_splitk_fixed_order_is_repeatable():
    a, b, r = _mk((8192, 1024), 5), _mk((8192, 1536), 6), _mk((1024, 1536), 3)
    ref = a.float().t() @ b.float() + r.float()
    y1 = ops.matmul_tn(a, b, residual=r, splits=8)
    y2 = ops.matmul_tn(a, b, residual=r, splits=8)
    _check(y1, ref, 8192)
    assert torch.equal(y1, y2)
    y3 = ops.matmul_tn(a, b, residual=r)  # heuristic split
    _check(y3, ref, 8192)


@pytest.mark.parametrize("splits", [2, 3, 4, 8, 9, 10])
def test_splitk_adds_every_part_once(splits):
    """Numbers of parts around what the sum has on its way at once. Operands in {-2..2} over 640 of k: sums are integers, exact in fp32,
    and in bf16 up to 256, which they stay below by ten deviations."""
    x, w, r = _ints((136, 640), 1), _ints((640, 264), 2), _ints((136, 264), 3)
    want = x.float() @ w.float()
    assert want.abs().max() < 250
    assert torch.equal(ops.matmul_nn(x, w, splits=splits).float(), want)
    assert torch.equal(ops.matmul_nn(x, w, residual=r, splits=splits).float(), want + r.float())
    _lib.check_status()


def test_strided_views():
    big = _mk((512, 3072), 11)
    x = big[:, 1024:2048]  # pitch 3072, offset 2048 bytes
    w = _mk((1024, 256), 12)
    out = torch.zeros((512, 1024), dtype=torch.bfloat16, device="cuda")
    ops.matmul_nn(x, w, out=out[:, 512:768])
    _lib.check_status()
    ref = x.float() @ w.float()
    assert (out[:, 512:768].float() - ref).abs().max().item() < 0.3
    assert out[:, :512].abs().max().item() == 0 and out[:, 768:].abs().max().item() == 0


PAIR_SHAPES = [(256, 256, 64), (512, 768, 512), (304, 264, 1000), (4096, 1536, 1024), (2176, 2816, 520)]


@pytest.mark.parametrize("M,N,K", PAIR_SHAPES)
@pytest.mark.parametrize("form", ["nn", "nt", "tn", "tt"])
def test_cta_pair_kernel_all_forms(M, N, K, form, monkeypatch):
    """The cta_group::2 kernel (256 x 256 tiles over two SMs) against fp32, same answers as the
    single-CTA kernel's contract; odd sizes exercise the zero-filled edges of both CTAs."""
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "PAIR_MODE", "1")
    r = _mk((M, N), 11)
    if form == "nn":
        a, b = _mk((M, K), 1), _mk((K, N), 2)
        y, ref = ops.matmul_nn(a, b, residual=r), a.float() @ b.float()
    elif form == "nt":
        a, b = _mk((M, K), 3), _mk((N, K), 4)
        y, ref = ops.matmul_nt(a, b, residual=r), a.float() @ b.float().t()
    elif form == "tn":
        a, b = _mk((K, M), 5), _mk((K, N), 6)
        y, ref = ops.matmul_tn(a, b, residual=r, splits=1), a.float().t() @ b.float()
    else:
        a, b = _mk((K, M), 7), _mk((N, K), 8)
        y, ref = ops.matmul_tt_a(a, b, residual=r), a.float().t() @ b.float().t()
    _check(y, ref + r.float(), K)


def test_cta_pair_kernel_is_bitwise_repeatable_and_matches_single_cta(monkeypatch):
    from scirust_b200.ops import gemm
    x, w = _mk((4096, 1024), 1), _mk((1024, 2816), 2)
    monkeypatch.setattr(gemm, "BALANCED", False)
    monkeypatch.setattr(gemm, "PAIR_MODE", "1")
    y1 = ops.matmul_nn(x, w)
    y2 = ops.matmul_nn(x, w)
    monkeypatch.setattr(gemm, "PAIR_MODE", "0")
    y0 = ops.matmul_nn(x, w)
    _lib.check_status()
    assert torch.equal(y1, y2)
    # same K order and fp32 accumulation in both kernels: identical results
    assert torch.equal(y1, y0)


@pytest.mark.parametrize("M,N,K", [(16384, 1024, 1024), (1024, 1536, 16384), (2816, 1024, 8192), (200, 264, 136),
                                   (19072, 256, 512), (16, 6144, 4096)])
def test_balanced_schedule_matches_plain_schedule_bitwise(M, N, K, monkeypatch):
    """Whole waves one tile per CTA, the last partial wave dealt out in k-blocks and summed by the
    fix-up pass in k order: fp32 partial sums are added in a fixed order, so two runs agree bit for
    bit, and the result matches fp32 within bf16 rounding for every operand form."""
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "PAIR_MODE", "0")
    monkeypatch.setattr(gemm, "BALANCED", True)
    monkeypatch.setattr(gemm, "_BALANCED_MIN_K", 0)
    x, w, r = _mk((M, K), 1), _mk((K, N), 2), _mk((M, N), 3)
    y1 = ops.matmul_nn(x, w, residual=r)
    y2 = ops.matmul_nn(x, w, residual=r)
    assert torch.equal(y1, y2)
    _check(y1, x.float() @ w.float() + r.float(), K)
    a, b = _mk((K, M), 5), _mk((K, N), 6)
    _check(ops.matmul_tn(a, b), a.float().t() @ b.float(), K)
    bt = _mk((N, K), 7)
    _check(ops.matmul_nt(x, bt), x.float() @ bt.float().t(), K)


@pytest.mark.parametrize("M,N,K", [(1024, 1536, 16384), (2816, 1024, 8192), (5632, 1024, 4096), (300, 520, 704)])
def test_cta_pair_kernel_with_balanced_schedule(M, N, K, monkeypatch):
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "PAIR_MODE", "1")
    monkeypatch.setattr(gemm, "BALANCED", True)
    monkeypatch.setattr(gemm, "_BALANCED_MIN_K", 0)
    Mt = (M + 7) // 8 * 8
    a, b, r = _mk((K, Mt), 5), _mk((K, N), 6), _mk((Mt, N), 3)
    y1 = ops.matmul_tn(a, b, residual=r)
    y2 = ops.matmul_tn(a, b, residual=r)
    assert torch.equal(y1, y2)
    _check(y1, a.float().t() @ b.float() + r.float(), K)
    x, w = _mk((M, K), 1), _mk((K, N), 2)
    _check(ops.matmul_nn(x, w), x.float() @ w.float(), K)


@pytest.mark.parametrize("pair", ["0", "1"])
def test_bias_epilogue(pair, monkeypatch):
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "PAIR_MODE", pair)
    x, w, b = _mk((640, 512), 1), _mk((512, 768), 2), _mk((768,), 3)
    _check(ops.matmul_nn(x, w, bias=b), x.float() @ w.float() + b.float()[None, :], 512)
    wt = _mk((768, 512), 4)
    _check(ops.matmul_nt(x, wt, bias=b), x.float() @ wt.float().t() + b.float()[None, :], 512)
    with pytest.raises(ValueError):
        ops.matmul_nn(x, w, bias=b, residual=_mk((640, 768), 5))


@pytest.mark.parametrize("M,K,ff", [(512, 256, 128), (4096, 1024, 2816), (1000, 512, 264)])
def test_swiglu_epilogue_is_bitwise_the_unfused_path(M, K, ff, monkeypatch):
    from scirust_b200.ops import basic, gemm
    monkeypatch.setattr(gemm, "FUSE_SWIGLU", True)
    x, wgu = _mk((M, K), 1), _mk((K, 2 * ff), 2)
    gu, act = ops.matmul_nn_swiglu(x, wgu)
    _lib.check_status()
    monkeypatch.setattr(gemm, "PAIR_MODE", "0")
    monkeypatch.setattr(gemm, "BALANCED", False)
    gu0 = ops.matmul_nn(x, wgu)
    act0 = basic.swiglu_fwd(gu0)
    assert torch.equal(gu, gu0)
    assert torch.equal(act, act0)
    _check(gu, x.float() @ wgu.float(), K)


@pytest.mark.parametrize("M,K,ff", [(256, 64, 8), (257, 128, 72), (1000, 512, 264), (2048, 1024, 4736)])
def test_swiglu_epilogue_without_the_product(M, K, ff, monkeypatch):
    """act alone, the same bits as with the product kept: one row past a tile, slabs of 64 columns that end inside (and would
    reach into the up columns), more tiles than CTA pairs. The product keeps its gate and up columns apart."""
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "FUSE_SWIGLU", True)
    x, wgu = _mk((M, K), 1), _mk((K, 2 * ff), 2)
    gu, act = ops.matmul_nn_swiglu(x, wgu)
    only = ops.matmul_nn_swiglu_act(x, wgu)
    _lib.check_status()
    assert torch.equal(act, only)
    assert torch.equal(act, ops.swiglu_fwd(gu))
    _check(gu, x.float() @ wgu.float(), K)


@pytest.mark.parametrize("fuse", [True, False])
def test_swiglu_product_looks_at_the_buffers_it_is_given(fuse, monkeypatch):
    """What does not hold the result is refused before anything is launched, whichever kernels would run; a matrix with rows of its
    own pitch and a buffer of as many elements are filled, and nothing beside them."""
    from scirust_b200.ops import gemm
    monkeypatch.setattr(gemm, "FUSE_SWIGLU", fuse)
    M, K, ff = 300, 128, 264
    x, wgu = _mk((M, K), 1), _mk((K, 2 * ff), 2)
    gu, act = ops.matmul_nn_swiglu(x, wgu)

    def buf(*shape, dtype=torch.bfloat16):
        return torch.full(shape, 7.0, dtype=dtype, device="cuda")

    launched = gemm.launch_count
    for out in (buf(M - 1, 2 * ff), buf(M, ff), buf(M, 2 * ff, dtype=torch.float32), buf(2 * ff, M).t(), buf(M * 2 * ff)):
        with pytest.raises(ValueError):
            ops.matmul_nn_swiglu(x, wgu, out=out)
    for a in (buf(M - 1, ff), buf(M, ff, dtype=torch.float32), buf(ff, M).t(), buf(M, 2 * ff)[:, ::2], buf(1, ff).expand(M, ff)):
        with pytest.raises(ValueError):
            ops.matmul_nn_swiglu(x, wgu, act=a)
    assert gemm.launch_count == launched
    wide_out, wide_act = buf(M, 2 * ff + 8), buf(M, ff + 16)
    got, a = ops.matmul_nn_swiglu(x, wgu, out=wide_out[:, :2 * ff], act=wide_act[:, :ff])
    assert torch.equal(got, gu) and torch.equal(a, act)
    assert bool((wide_out[:, 2 * ff:] == 7.0).all()) and bool((wide_act[:, ff:] == 7.0).all())
    for shape in ((M * ff,), (3, M // 3, ff), (M + 1, ff)):
        a = buf(*shape)
        assert ops.matmul_nn_swiglu(x, wgu, act=a)[1] is a
        assert torch.equal(a.view(-1)[:M * ff].view(M, ff), act) and bool((a.view(-1)[M * ff:] == 7.0).all())
    _lib.check_status()


@pytest.mark.parametrize("quant", [None, "int8"])
def test_prefill_with_the_swiglu_in_the_product(quant, monkeypatch):
    """The engine's feed-forward with and without it: the same logits and cache to the bit."""
    from scirust_b200.models.infer import InferenceEngine
    from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig
    from scirust_b200.ops import gemm
    cfg = SciAgentConfig(512, 256, 2, 4, 2, 512, 2048, 1e4)
    model = GQADecoder(cfg, device="cuda", seed=3)
    tokens = torch.randint(0, 512, (2, 600), generator=torch.Generator().manual_seed(1)).cuda()
    got = []
    for fuse in (True, False):
        monkeypatch.setattr(gemm, "FUSE_SWIGLU", fuse)
        eng = InferenceEngine(model, quant=quant, max_batch=2, max_seq=640)
        got.append((eng.prefill(tokens).clone(), *eng.cache.pools))
    _lib.check_status()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("how", ["_linear", "_proj_out", "instance"])
def test_prefill_takes_every_product_of_a_subclass(how, monkeypatch):
    """An engine with products of its own (an adapter, another quantisation) has all of them taken in a prefill, gate/up among
    them, at sizes where the base class takes that one through its epilogue."""
    from scirust_b200.models.infer import InferenceEngine
    from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig
    from scirust_b200.ops import gemm

    class Adapted(InferenceEngine):
        pass

    def linear(self, x, w, residual=None):
        seen.append(tuple(w.shape))
        return InferenceEngine._linear(self, x, w, residual) * 1.5

    def proj_out(self, a, w, x, swiglu=False, site="attn"):
        seen.append((site, swiglu))
        return InferenceEngine._proj_out(self, a, w, x, swiglu, site)

    if how != "instance":
        setattr(Adapted, how, {"_linear": linear, "_proj_out": proj_out}[how])
    cfg = SciAgentConfig(512, 256, 2, 4, 2, 512, 2048, 1e4)
    model = GQADecoder(cfg, device="cuda", seed=3)
    tokens = torch.randint(0, 512, (2, 600), generator=torch.Generator().manual_seed(1)).cuda()
    got = []
    for fuse in (True, False):
        monkeypatch.setattr(gemm, "FUSE_SWIGLU", fuse)
        seen = []
        eng = Adapted(model, max_batch=2, max_seq=640)
        if how == "instance":
            eng._linear = lambda x, w, residual=None: linear(eng, x, w, residual)
        got.append((eng.prefill(tokens).clone(), *eng.cache.pools))
        want = ([("attn", False), ("mlp", True)] if how == "_proj_out" else
                [(256, 512), (256, 256), (256, 1024), (512, 256)])
        assert [s for s in seen if s in want] == want * 2
    _lib.check_status()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,d,ff", [(512, 256, 128), (4096, 1024, 2816), (1000, 512, 264)])
def test_swiglu_backward_epilogue_is_bitwise_the_unfused_path(M, d, ff, monkeypatch):
    from scirust_b200.ops import basic, gemm
    monkeypatch.setattr(gemm, "FUSE_SWIGLU", True)
    dy, wd, gu = _mk((M, d), 1), _mk((ff, d), 2), _mk((M, 2 * ff), 3)
    dgu = ops.matmul_nt_swiglu_bwd(dy, wd, gu)
    _lib.check_status()
    monkeypatch.setattr(gemm, "PAIR_MODE", "0")
    monkeypatch.setattr(gemm, "BALANCED", False)
    ref = basic.swiglu_bwd(gu, ops.matmul_nt(dy, wd))
    assert torch.equal(dgu, ref)


@pytest.mark.parametrize("M,N,K,form", [(300, 520, 128, "plain"), (1100, 2816, 1024, "residual"), (2560, 2304, 4096, "balanced"),
                                        (1100, 5632, 1024, "swiglu")])
def test_product_widens_int8_matrices_beside_itself(M, N, K, form, monkeypatch):
    """The product's bits are those without the expansion, the matrices' those of ``dequantize``; ragged units of rows and columns, few
    CTAs and all of them, and nothing is written behind a matrix."""
    from scirust_b200.ops import decode as D, gemm
    monkeypatch.setattr(gemm, "PAIR_MODE", "1")
    monkeypatch.setattr(gemm, "FUSE_SWIGLU", form == "swiglu")
    g = torch.Generator(device="cuda").manual_seed(5)
    sizes = [(13, 16), (2056, 1040), (70, 528)]
    jobs, want, tails = [], [], []
    for k, n in sizes:
        q = torch.randint(-128, 128, (k, n), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
        scale = torch.rand(n, generator=g, device="cuda") * 0.1
        buf = torch.full((k * n + 512,), 7.0, dtype=torch.bfloat16, device="cuda")
        jobs.append((q, scale, buf[:k * n].view(k, n)))
        want.append(D.QuantWeight(q, scale).dequantize())
        tails.append(buf[k * n:])
    x, w = _mk((M, K), 1), _mk((K, N), 2)
    res = _mk((M, N), 3) if form == "residual" else None
    if form == "swiglu":
        alone, y = ops.matmul_nn_swiglu_act(x, w), ops.matmul_nn_swiglu_act(x, w, widen=jobs)
    else:
        alone, y = ops.matmul_nn(x, w, residual=res), gemm.matmul_nn_beside(x, w, res, jobs)
    _lib.check_status()
    assert torch.equal(alone, y)
    for (_, _, got), right, tail in zip(jobs, want, tails):
        assert torch.equal(got, right)
        assert bool((tail == 7.0).all())
    with pytest.raises((ValueError, RuntimeError)):            # a width that the expansion does not take
        gemm.matmul_nn_beside(x, w, None, [(jobs[0][0].view(16, 13), jobs[0][1][:13].clone(), jobs[0][2].view(16, 13))])
    (q, scale, out), launched = jobs[0], gemm.launch_count
    for bad in ((q, scale, out[:12]), (q, scale, out.float()), (q, scale[:8], out), (q, scale.double(), out), (q.int(), scale, out),
                (q, scale, torch.empty(16, 13, dtype=torch.bfloat16, device="cuda").t()), (q.cpu(), scale, out), (q, scale, out.view(-1))):
        with pytest.raises(ValueError):                        # buffers that would be read or written past their ends
            gemm.matmul_nn_beside(x, w, None, [bad])
    assert gemm.launch_count == launched


@pytest.mark.parametrize("batch,seq,ff", [(1, 1100, 2816), (3, 683, 2824)])
def test_prefill_that_widens_ahead(batch, seq, ff, monkeypatch):
    """Logits and cache as from an engine that expands each matrix before its product (ff 2824: two matrices are not wide enough by
    whole 16-byte words and are left to that)."""
    from scirust_b200.models.infer import InferenceEngine, _WidenAhead
    from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig

    class Before(InferenceEngine):
        def _linear(self, x, w, residual=None):
            return InferenceEngine._linear(self, x, w, residual)

        def _proj_out(self, a, w, x, swiglu=False, site="attn"):
            return InferenceEngine._linear(self, ops.swiglu_fwd(a) if swiglu else a, w, residual=x)

    monkeypatch.setattr(_WidenAhead, "WORK", 0)
    cfg = SciAgentConfig(512, 1024, 3, 16, 4, ff, 2048, 1e4)
    model = GQADecoder(cfg, device="cuda", seed=3)
    tokens = torch.randint(0, 512, (batch, seq), generator=torch.Generator().manual_seed(1)).cuda()
    got = []
    for cls in (InferenceEngine, Before):
        eng = cls(model, quant="int8", max_batch=batch, max_seq=seq + 20)
        got.append((eng.prefill(tokens).clone(), *eng.cache.pools))
    _lib.check_status()
    for a, b in zip(*got):
        assert torch.equal(a, b)
    plan = _WidenAhead(eng.layers, batch * seq)
    taken = [len(plan.product(l[k])[1].get("widen", ())) for l in eng.layers for k in ("wqkv", "wo", "wgu", "wd")]
    assert sum(taken) >= 3 and max(taken) <= 3
    monkeypatch.undo()
    plan = _WidenAhead(eng.layers, batch * seq)            # too little work for the host to plan
    assert all(plan.product(l[k]) == (l[k], {}) for l in eng.layers for k in ("wqkv", "wo", "wgu", "wd"))


def test_prefill_expands_a_kind_of_weight_of_its_own_by_its_own_method(monkeypatch):
    """A subclass of the int8 weight with another meaning of its codes is not expanded beside a product."""
    from scirust_b200.models import infer
    from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig
    from scirust_b200.ops import decode as D

    class Doubled(D.QuantWeight):
        def dequantize(self):
            return super().dequantize() * 2

    cfg = SciAgentConfig(512, 1024, 2, 16, 4, 2816, 2048, 1e4)
    model = GQADecoder(cfg, device="cuda", seed=3)
    tokens = torch.randint(0, 512, (1, 1100), generator=torch.Generator().manual_seed(1)).cuda()
    got = []
    for work in (0, 1 << 60):
        monkeypatch.setattr(infer._WidenAhead, "WORK", work)
        eng = infer.InferenceEngine(model, quant="int8", max_batch=1, max_seq=1200)
        for l in eng.layers:
            l["wd"] = Doubled(l["wd"].q, l["wd"].scale)
        got.append((eng.prefill(tokens).clone(), *eng.cache.pools))
    _lib.check_status()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("where", ["attention_fwd", "swiglu_fwd", "rmsnorm_fwd"])
def test_prefill_gives_matrices_back_when_memory_runs_out(where, monkeypatch):
    """An allocation that fails while matrices expanded ahead are held (here by exception, on the host): the piece of the layer is run
    again without them, with the same logits and cache, and prompts of as many rows expand nothing ahead from then on."""
    from scirust_b200.models import infer
    from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig
    from scirust_b200.ops import gemm
    monkeypatch.setattr(infer._WidenAhead, "WORK", 0)
    monkeypatch.setattr(gemm, "FUSE_SWIGLU", False)
    cfg = SciAgentConfig(512, 1024, 3, 16, 4, 2816, 2048, 1e4)
    model = GQADecoder(cfg, device="cuda", seed=3)
    tokens = torch.randint(0, 512, (1, 1100), generator=torch.Generator().manual_seed(1)).cuda()
    plans, product = [], infer._WidenAhead.product

    def watched(self, w):
        if self not in plans:
            plans.append(self)
        return product(self, w)

    monkeypatch.setattr(infer._WidenAhead, "product", watched)
    eng = infer.InferenceEngine(model, quant="int8", max_batch=1, max_seq=1200)

    def prefill():                                             # logits, and the cache in the order of the sequence
        for p in eng.cache.pools:
            p.zero_()
        logits = eng.prefill(tokens).clone()
        _lib.check_status()
        return [logits, *(p[eng.cache.block_table[0, :18].long()] for p in eng.cache.pools)]

    want = prefill()
    assert plans[0].taken > 3 and not plans[0].ran_out
    module = infer.att if where == "attention_fwd" else infer.ops
    real, failed = getattr(module, where), []

    def short_of_memory(*args, **kw):
        if plans[-1].wide and len(plans) == 2 and not failed:
            failed.append(1)
            raise torch.OutOfMemoryError("no memory")
        return real(*args, **kw)

    monkeypatch.setattr(module, where, short_of_memory)
    for _ in range(2):
        for a, b in zip(want, prefill()):
            assert torch.equal(a, b)
    assert failed and plans[1].ran_out and not plans[1].order and not plans[2].taken and not plans[2].ran_out
    monkeypatch.setattr(module, where, real)
    eng.prefill(tokens[:, :1050])                              # fewer rows may again
    assert plans[3].taken > 3
