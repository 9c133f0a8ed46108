"""Bandwidth-bound kernels against the fp32 PyTorch statement of the same op (the CPU path of
each op in scirust_b200.ops.basic is that statement)."""
import pytest
import torch

from scirust_b200 import ops

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _r(shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(BF)


def _close(a, b, tol=2e-2):
    a, b = a.float().cpu(), b.float().cpu()
    err = (a - b).abs().max().item()
    lim = tol * max(1.0, b.abs().max().item())
    assert err <= lim, f"max err {err} > {lim}"


@pytest.mark.parametrize("rows,cols", [(7, 256), (1000, 1024), (33, 4096), (5, 264)])
def test_rmsnorm_fwd_bwd(rows, cols):
    x, w, dy, dres = _r((rows, cols), 1), _r((cols,), 2), _r((rows, cols), 3), _r((rows, cols), 4)
    y_ref, inv_ref = ops.rmsnorm_fwd(x, w)
    y, inv = ops.rmsnorm_fwd(x.cuda(), w.cuda())
    _close(y, y_ref)
    assert torch.allclose(inv.cpu(), inv_ref, rtol=1e-4, atol=1e-6)
    dx_ref, dw_ref = ops.rmsnorm_bwd(dy, x, w, inv_ref, dres=dres)
    dx, dw = ops.rmsnorm_bwd(dy.cuda(), x.cuda(), w.cuda(), inv, dres=dres.cuda())
    _close(dx, dx_ref)
    assert torch.allclose(dw.cpu(), dw_ref, rtol=2e-3, atol=2e-2 * max(1.0, dw_ref.abs().max().item()) * 0.05)
    dx2, dw2 = ops.rmsnorm_bwd(dy.cuda(), x.cuda(), w.cuda(), inv, dres=dres.cuda())
    assert torch.equal(dw, dw2) and torch.equal(dx, dx2)


@pytest.mark.parametrize("rows,cols", [(1, 512), (9, 1024), (2368, 512), (2369, 1024), (5000, 1024)])
@pytest.mark.parametrize("res,out", [(True, torch.float32), (False, torch.bfloat16), (True, torch.bfloat16)])
def test_rmsnorm_bwd_in_one_pass(rows, cols, res, out):
    """Both gradients from one pass (rows of 512 and 1024): a single row, a last CTA with one row, a grid that is exactly full and
    one row more, several rows a warp. dx has one rounding to bf16 (2^-8) of terms of size one; dw sums rows fp32 terms."""
    x, w, dy, dres = _r((rows, cols), 1), _r((cols,), 2), _r((rows, cols), 3), _r((rows, cols), 4)
    inv = ops.rmsnorm_fwd(x, w)[1]
    dx_ref, dw_ref = ops.rmsnorm_bwd(dy, x, w, inv, dres=dres if res else None)
    dw_out = torch.full((cols,), float("nan"), dtype=out, device="cuda")
    dx, dw = ops.rmsnorm_bwd(dy.cuda(), x.cuda(), w.cuda(), inv.cuda(), dres=dres.cuda() if res else None, dw_out=dw_out)
    assert dw is dw_out
    _close(dx, dx_ref, 2 ** -7)
    terms = (dy.float() * x.float() * inv[:, None]).abs().sum(0).max().item()
    lim = terms * (rows * 2.0 ** -24 if out == torch.float32 else 2.0 ** -8) + 1e-6
    assert (dw.float().cpu() - dw_ref).abs().max().item() <= lim


@pytest.mark.parametrize("rows,cols", [(999, 512), (16384, 1024)])
@pytest.mark.parametrize("res", [True, False])
def test_rmsnorm_bwd_rounds_alike_with_and_without_the_gain(rows, cols, res):
    """dx of the pass that takes both gradients against the kernel of dx alone: the same operations on the same roundings, so the same
    bits. Enough elements that another contraction of r (g - x k) + d shows in a few of them."""
    x, w, dy, dres = (_r(s, i).cuda() for i, s in enumerate([(rows, cols), (cols,), (rows, cols), (rows, cols)], 1))
    inv = ops.rmsnorm_fwd(x, w)[1]
    one, two = (ops.rmsnorm_bwd(dy, x, w, inv, dres=dres if res else None, want_dw=want)[0] for want in (True, False))
    assert torch.equal(one, two)


@pytest.mark.parametrize("rows,cols", [(999, 512), (5000, 1024)])
def test_rmsnorm_gain_gradient_does_not_depend_on_the_device(rows, cols, monkeypatch):
    """The order of its sum follows from rows and columns: the same bits where the device says that it has other numbers of SMs."""
    from scirust_b200.ops import basic
    x, w, dy = (_r(s, i).cuda() for i, s in enumerate([(rows, cols), (cols,), (rows, cols)], 1))
    inv = ops.rmsnorm_fwd(x, w)[1]
    got = []
    for sms in (148, 132, 20):
        monkeypatch.setattr(basic._g, "num_sms", lambda device=None: sms)
        got.append(ops.rmsnorm_bwd(dy, x, w, inv)[1])
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("dh", [64, 128])
def test_rope_roundtrip_and_reference(dh):
    rows, heads, kv = 96, 4, 2
    ld = (heads + 2 * kv) * dh
    x = _r((rows, ld), 5)
    cos_t, sin_t = ops.rope_table(64, dh, 10000.0, "cpu")
    ref = ops.rope_(x.clone(), heads + kv, dh, 32, cos_t, sin_t, offset=3)
    xg = x.cuda()
    cg, sg = ops.rope_table(64, dh, 10000.0, "cuda")
    ops.rope_(xg, heads + kv, dh, 32, cg, sg, offset=3)
    _close(xg, ref, 1e-2)
    assert torch.equal(xg[:, (heads + kv) * dh:].cpu(), x[:, (heads + kv) * dh:])  # v untouched
    ops.rope_(xg, heads + kv, dh, 32, cg, sg, offset=3, backward=True)
    _close(xg, x, 2e-2)
    pos = torch.randint(0, 64, (rows,), dtype=torch.int32)
    ref2 = ops.rope_(x.clone(), heads, dh, 32, cos_t, sin_t, positions=pos)
    x2 = x.cuda()
    ops.rope_(x2, heads, dh, 32, cg, sg, positions=pos.cuda())
    _close(x2, ref2, 1e-2)


def test_swiglu_and_add():
    gu, dh = _r((130, 2 * 2816), 6), _r((130, 2816), 7)
    _close(ops.swiglu_fwd(gu.cuda()), ops.swiglu_fwd(gu))
    _close(ops.swiglu_bwd(gu.cuda(), dh.cuda()), ops.swiglu_bwd(gu, dh))
    a, b = _r((64, 1024), 8), _r((64, 1024), 9)
    _close(ops.add(a.cuda(), b.cuda()), ops.add(a, b), 1e-2)


def test_embedding_fwd_bwd_deterministic():
    V, d, n = 500, 256, 4096
    table = _r((V, d), 10)
    tok = torch.randint(0, V, (n,), generator=torch.Generator().manual_seed(0))
    tok[:100] = 7  # a long segment
    out = ops.embed_fwd(table.cuda(), tok.cuda())
    assert torch.equal(out.cpu(), table[tok])
    dy = _r((n, d), 11, 0.1)
    base = _r((V, d), 12, 0.1)
    ref = ops.embed_bwd(dy, tok, base.clone())
    g1 = ops.embed_bwd(dy.cuda(), tok.cuda(), base.clone().cuda())
    g2 = ops.embed_bwd(dy.cuda(), tok.cuda(), base.clone().cuda())
    assert torch.equal(g1, g2)
    _close(g1, ref, 2e-2)


@pytest.mark.parametrize("n,V,d,repeat", [
    (1, 1, 8, 0), (300, 7, 1032, 0),             # every chain longer than a warp ranks; a second slab of 8 columns
    (2500, 4000, 64, 32), (2500, 4000, 64, 33),  # the longest ranked chain, the shortest that the tokens are read for
    (2050, 50, 4096, 1500), (40, 1000, 2048, 2)])
@pytest.mark.parametrize("accumulate", [True, False])
def test_embedding_bwd_adds_in_ascending_order(n, V, d, repeat, accumulate):
    """Rows of one token are added in fp32 in the order of their positions, whatever order the chains were built in: the same bits
    as a loop. Ids outside the table count for its first and last row."""
    tok = torch.randint(0, V, (n,), generator=torch.Generator().manual_seed(n))
    if n > 4 and V > 7:
        tok[tok == 3] = 4
        tok[torch.randperm(n, generator=torch.Generator().manual_seed(1))[:repeat]] = 3
        tok[1], tok[n - 1] = -5, V + 9
    dy, base = _r((n, d), 11, 0.1), _r((V, d), 12, 0.1)
    want = base.float() if accumulate else torch.zeros(V, d)
    for i in range(n):
        want[tok[i].clamp(0, V - 1)] += dy[i].float()
    got = ops.embed_bwd(dy.cuda(), tok.cuda(), base.clone().cuda(), accumulate=accumulate)
    assert torch.equal(got.cpu(), want.to(torch.bfloat16))


@pytest.mark.parametrize("rows,cols", [(64, 32000), (17, 1000), (9, 128256)])
def test_cross_entropy(rows, cols):
    logits = _r((rows, cols), 13, 2.0)
    tgt = torch.randint(0, cols, (rows,), generator=torch.Generator().manual_seed(1))
    tgt[0] = cols + 5  # clamps
    tgt[1] = -1        # ignored
    loss_ref, d_ref = ops.ce_fwd_bwd(logits.clone(), tgt, 1.0 / rows)
    lg = logits.cuda()
    loss, d = ops.ce_fwd_bwd(lg, tgt.cuda(), 1.0 / rows)
    assert d.data_ptr() == lg.data_ptr()
    assert torch.allclose(loss.cpu(), loss_ref, rtol=1e-3, atol=1e-3)
    assert (d.float().cpu() - d_ref.float()).abs().max().item() <= 1e-2 / rows + 1e-6
    assert torch.allclose(ops.ce_loss_only(logits.cuda(), tgt.cuda()).cpu(), loss_ref, rtol=1e-3, atol=1e-3)


def test_sumsq_and_optimizer():
    n = 1_000_003
    g = _r((n,), 14, 0.01)
    s = ops.sumsq(g.cuda())
    assert abs(s.item() - g.float().pow(2).sum().item()) <= 1e-3 * s.item()
    assert torch.equal(s, ops.sumsq(g.cuda()))
    for mode in ("adamw", "adam", "sgd"):
        p = torch.randn(n, generator=torch.Generator().manual_seed(3))
        m, v = torch.zeros(n), torch.zeros(n)
        pg, mg, vg = p.cuda(), m.cuda(), v.cuda()
        pb = torch.empty(n, dtype=BF, device="cuda")
        for step in (1, 2):
            kw = dict(lr=1e-2, weight_decay=0.1, step=step, decay_end=n // 2, max_grad_norm=0.5, mode=mode)
            ops.optim_step(p, m, v, g, None, grad_sumsq=g.float().pow(2).sum().reshape(1), **kw)
            ops.optim_step(pg, mg, vg, g.cuda(), pb, grad_sumsq=s, **kw)
        assert torch.allclose(pg.cpu(), p, rtol=1e-4, atol=1e-5), mode
        assert torch.equal(pb.cpu(), pg.cpu().to(BF))
    # non-finite gradient norm skips the update
    before = pg.clone()
    ops.optim_step(pg, mg, vg, g.cuda(), pb, lr=1e-2, grad_sumsq=torch.tensor([float("nan")], device="cuda"))
    assert torch.equal(before, pg)


def test_deferred_status_raises_collective_timeout_one_poll_late():
    """A bounded wait that runs out leaves a code in the status word; the non-blocking reader used by the
    trainers turns it into CollectiveTimeout on the following poll, and the word is cleared."""
    import ctypes as C
    from scirust_b200.ops import _lib
    _lib.register("sb_wait_probe", [_lib.vp, _lib.i32, C.c_uint32, _lib.i32, _lib.vp, _lib.vp])
    dev = torch.device("cuda", 0)
    ds = _lib.DeferredStatus(dev)
    ds.poll()
    ds.poll()                                   # nothing recorded: no error
    flags = torch.zeros(16, dtype=torch.int32, device=dev)
    st = _lib.status_word(dev)
    _lib.call("sb_wait_probe", flags.data_ptr(), 2, 7, 50, st.data_ptr(), _lib.stream())   # waits 50 ms for nothing
    ds.poll()                                   # queues the copy behind the probe
    with pytest.raises(_lib.CollectiveTimeout):
        ds.poll()
    assert int(st.item()) == 0
    ds.poll()
    ds.poll()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 32768 + 5, 1000003])
@pytest.mark.parametrize("offset", [0, 1])
def test_sumsq_edges(dtype, n, offset):
    """Whole and partial blocks of 4096, 16-byte aligned buffers and others, against float64: fp32 sums of up to 4096 + n / 4096
    terms in a tree, 1e-5 relative; accumulation adds to what is there."""
    g = _r((n + offset,), n).cuda().to(dtype)[offset:]
    want = g.double().square().sum().item()
    out = ops.sumsq(g)
    assert abs(out.item() - want) <= 1e-5 * want
    ops.sumsq(g, out=out, accumulate=True)
    assert abs(out.item() - 2 * want) <= 2e-5 * want


@pytest.mark.parametrize("cols", [8, 600, 1024, 2056, 8192, 9000])
def test_rmsnorm_few_rows_are_the_bits_of_many(cols):
    """A CTA per row for few rows (up to 296, or up to 1184 of twice as many columns), a warp per row beyond: the same
    association, so the same bits on both sides of every line; rows longer than what a thread keeps are read again."""
    x, w = _r((1185, cols), 1).cuda(), _r((cols,), 2).cuda()
    many, inv_many = ops.rmsnorm_fwd(x, w)
    for n in (7, 296, 297, min(1184, cols // 2)):
        few, inv_few = ops.rmsnorm_fwd(x[:n], w)
        assert torch.equal(few, many[:n]) and torch.equal(inv_few, inv_many[:n])


@pytest.mark.parametrize("M,K", [(1, 8), (3, 4096), (3, 8184), (3, 8192), (1025, 8192), (2, 16384), (2, 16392), (5, 24)])
def test_quantize_rows_edges(M, K):
    """Rows that fit a CTA's registers and rows that do not, a zero row: the host statement bit for bit."""
    from scirust_b200.ops import decode
    x = _r((M, K), K).cuda()
    x[0] = 0
    q, s = decode.quantize_rows(x)
    qc, sc = decode.quantize_rows(x.cpu())
    assert torch.equal(s.cpu(), sc) and torch.equal(q.cpu(), qc)


@pytest.mark.parametrize("cols", [8, 4096, 32760, 32768, 32776])
def test_cross_entropy_row_kept_in_registers(cols):
    """Both sides of the 32768-column line, ignored and clamped targets, the gradient over the logits or beside them: the
    loss does not depend on where the gradient goes, and a repeated call gives the same bits."""
    rows = 37
    lg = _r((rows, cols), 11).cuda() * 3
    lg[4] = float("-inf")
    lg[4, 5] = 1.0
    tg = torch.randint(0, cols, (rows,), generator=torch.Generator().manual_seed(1)).cuda()
    tg[0], tg[1], tg[4] = -1, cols + 7, 5
    loss, d = ops.ce_fwd_bwd(lg.clone(), tg, 0.25, in_place=False)
    loss_only = ops.ce_loss_only(lg, tg)
    inp = lg.clone()
    loss2, d2 = ops.ce_fwd_bwd(inp, tg, 0.25)
    assert d2.data_ptr() == inp.data_ptr()
    assert torch.equal(loss, loss2) and torch.equal(d, d2) and torch.equal(loss, loss_only)
    _check_cross_entropy(lg, tg, 0.25, loss, d)


def _check_cross_entropy(lg, tg, scale, loss, d):
    """Against the float64 statement. The loss: exponentials to 2^-21, sums of positive terms and a difference rounded to
    fp32, 1e-5 in all. The gradient is rounded to bf16 (2^-9) after a probability good to 1e-5 (2^-8 covers both; the
    target's entry p - 1 carries p's absolute error; results below 1e-36 may be flushed), so a row's sum is zero to 2^-9 of
    the sum of magnitudes, 2 * scale."""
    x, cols = lg.double(), lg.shape[1]
    ignored = tg < 0
    at = tg.clamp(0, cols - 1)[:, None]
    p = torch.softmax(x, -1)
    # the target's loss relative to the maximum: the difference of two large logits is exact, their logsumexp is not
    m = x.max(-1, keepdim=True).values
    want_loss = (torch.exp(x - m).sum(-1).log() - (x.gather(1, at) - m)[:, 0]).masked_fill(ignored, 0.0)
    want = p.scatter_add(1, at, -torch.ones_like(at, dtype=torch.float64)) * scale
    want[ignored] = 0.0
    lim = 2 ** -8 * want.abs() + 1e-36
    lim.scatter_add_(1, at, torch.full_like(at, 1e-5 * scale, dtype=torch.float64))
    assert ((loss.double() - want_loss).abs() <= 1e-5 * want_loss.abs().clamp(min=1.0)).all()
    assert ((d.double() - want).abs() <= lim).all()
    assert (d.double().sum(-1).abs() <= 2 ** -8 * 2 * scale).all()
    assert (d[ignored] == 0).all()


@pytest.mark.parametrize("cols", [8, 4096, 32768, 32776])
def test_cross_entropy_of_large_logits(cols):
    """Rows far from zero, down to the type's lowest value, on both sides of the 32768-column line: the result depends on
    the distances from the row's maximum, whatever the offset. Each row holds its offset and values up to three bf16 steps
    below it. Ignored rows give zeros, also where the logits are not numbers."""
    offsets = [0.0, 1e3, -1e3, 1e5, -1e7, 1e9, -1e30, 2.5e38, -3.0e38, torch.finfo(torch.bfloat16).min]
    g = torch.Generator().manual_seed(cols)
    base = torch.tensor(offsets).to(torch.bfloat16)[:, None].expand(-1, cols)
    steps = torch.randint(0, 4, base.shape, generator=g) * (base[:, :1].float().abs() * 2 ** -8).clamp(min=1.0)
    lg = (base.float() - steps).clamp(min=torch.finfo(torch.bfloat16).min).to(torch.bfloat16)
    lg[:, 3] = base[:, 3]
    lg = torch.cat((lg, lg, torch.full((2, cols), float("nan"), dtype=torch.bfloat16))).cuda()
    lg[-1] = float("-inf")
    n = len(offsets)
    tg = torch.randint(0, cols, (2 * n + 2,), generator=g)
    tg[:n:2], tg[n:] = 3, -1
    tg = tg.cuda()
    loss, d = ops.ce_fwd_bwd(lg.clone(), tg, 0.25, in_place=False)
    assert (loss[n:] == 0).all() and (d[n:] == 0).all()
    _check_cross_entropy(lg[:n], tg[:n], 0.25, loss[:n], d[:n])
    assert torch.equal(loss, ops.ce_loss_only(lg, tg))


@pytest.mark.parametrize("n,V,d", [(1, 1, 8), (32, 1, 1032), (33, 1, 2056), (97, 1, 64), (1000, 7, 4096), (2500, 4000, 1024), (32769, 3000, 64)])
@pytest.mark.parametrize("accumulate", [True, False])
def test_embedding_bwd_of_many_tokens(n, V, d, accumulate, monkeypatch):
    """Sorted tokens, which many take, against tokens as they are: rows in ascending order either way, so the same bits. Runs of 32
    places and of one more, runs that begin on a multiple of 32 and beside one, several slabs of columns. Ids outside the table come
    before and behind the others in the order: its first and last row, summed in another order."""
    from scirust_b200.ops import basic
    tok = torch.randint(0, V, (n,), generator=torch.Generator().manual_seed(n))
    outside = n > 1000
    if outside:
        tok[::5] = 3
        tok[torch.randperm(n)[:64]] = 2                       # with one id below, runs of 63 to 65 from the second place on
        tok[1], tok[n - 1] = -5, V + 9
    dy, base = _r((n, d), 11, 0.1).cuda(), _r((V, d), 12, 0.1).cuda()
    got = []
    for line in (n, n - 1):
        monkeypatch.setattr(basic, "EMBED_CHAIN_TOKENS", line)
        got.append(ops.embed_bwd(dy, tok.cuda(), base.clone(), accumulate=accumulate))
    one, two = (g[1:-1] if outside else g for g in got)
    assert torch.equal(one, two)
    _close(*got, tol=2 ** -7)


@pytest.mark.parametrize("n,V,d", [(1, 1, 8), (300, 7, 1032), (2500, 4000, 64)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_embedding_bwd_of_sorted_tokens_by_the_c_abi(n, V, d, accumulate):
    """The entry that takes tokens sorted by the caller: rows of a token in the order of their positions, the same bits as the form
    that takes tokens as they are."""
    from scirust_b200.ops import _lib
    tok = torch.randint(0, V, (n,), generator=torch.Generator().manual_seed(n)).cuda()
    dy, base = _r((n, d), 11, 0.1).cuda(), _r((V, d), 12, 0.1).cuda()
    order, perm = torch.sort(tok, stable=True)
    got = base.clone() if accumulate else torch.zeros_like(base)
    _lib.call("sb_embed_bwd", dy.data_ptr(), order.data_ptr(), perm.data_ptr(), got.data_ptr(), n, d, V, accumulate, _lib.stream())
    assert torch.equal(got, ops.embed_bwd(dy, tok, base.clone(), accumulate=bool(accumulate)))


@pytest.mark.parametrize("rows,heads,dh", [(1, 1, 8), (33, 3, 24), (4736, 8, 64), (4737, 8, 64), (40000, 1, 64), (20000, 5, 24), (2400, 5, 256)])
@pytest.mark.parametrize("backward", [False, True])
def test_rope_by_words_and_by_heads(rows, heads, dh, backward):
    """Both kernels around the line between them (a thread of the GPU's 148 x 2048 for each word of 16 bytes), one head, narrow heads. The rows
    of a call one by one are its bits: rotations have no sums over rows."""
    cos_t, sin_t = ops.rope_table(256, dh, 10000.0, "cuda")
    x = _r((rows, (heads + 1) * dh), 5).cuda()
    got = ops.rope_(x.clone(), heads, dh, 100, cos_t, sin_t, offset=7, backward=backward)
    _close(got, ops.rope_(x.cpu(), heads, dh, 100, cos_t.cpu(), sin_t.cpu(), offset=7, backward=backward), 2 ** -8)
    assert torch.equal(got[:, heads * dh:], x[:, heads * dh:])
    part = x[rows // 2:][:50].clone()
    pos = (torch.arange(rows)[rows // 2:][:50] % 100 + 7).int().cuda()
    ops.rope_(part, heads, dh, 100, cos_t, sin_t, positions=pos, backward=backward)
    assert torch.equal(part, got[rows // 2:][:50])


@pytest.mark.parametrize("rows,H,Hkv,dh,page", [(129, 3, 1, 64, 16), (300, 4, 2, 128, 64), (257, 5, 1, 24, 8), (1000, 2, 2, 8, 64)])
def test_rope_by_rows_fills_the_cache(rows, H, Hkv, dh, page):
    """A prompt's rotation with the copy to the cache (by rows, past 128 tokens) against the rotation and the copy by themselves: heads
    that do not fill a thread's four, rows that do not fill a block, head dimensions that do not divide it. The same bits; and the
    rotation against its fp32 statement."""
    from scirust_b200.ops import decode as D
    ld = (H + 2 * Hkv) * dh
    x = _r((rows, ld), 21).cuda()
    cos_t, sin_t = ops.rope_table(rows, dh, 10000.0, "cuda")
    blocks = (rows + page - 1) // page
    table = torch.randperm(blocks, generator=torch.Generator().manual_seed(2)).int().reshape(1, blocks).cuda()
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    seq_of = torch.zeros(rows, dtype=torch.int32, device="cuda")
    pools = [torch.zeros(blocks, 2, Hkv, page, dh, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    one, two = x.clone(), x.clone()
    D.rope_kv_append(one, H, Hkv, dh, cos_t, sin_t, pools[0], table, page, seq_of, pos)
    ops.rope_(two, H + Hkv, dh, rows, cos_t, sin_t)
    D.kv_append(two, H, Hkv, dh, pools[1], table, page, seq_of, pos)
    assert torch.equal(one, two) and torch.equal(pools[0], pools[1])
    ref = ops.rope_(x.cpu(), H + Hkv, dh, rows, *(t.cpu() for t in (cos_t, sin_t)))
    _close(two, ref, 2 ** -8)
    back = ops.rope_(two.clone(), H + Hkv, dh, rows, cos_t, sin_t, backward=True)
    _close(back, x, 2 ** -7)
