"""tcgen05 flash attention against the dense fp32 PyTorch reference."""
import pytest
import torch

from scirust_b200.ops import _lib, attention as A

pytestmark = pytest.mark.gpu


def _qkv(B, S, H, Hkv, dh, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(B * S, (H + 2 * Hkv) * dh, generator=g, device="cuda").to(torch.bfloat16)


CASES = [(1, 128, 1, 1, 64), (2, 256, 4, 2, 64), (1, 1000, 4, 1, 64), (2, 2048, 16, 4, 64), (1, 384, 4, 2, 128),
         (1, 200, 2, 2, 128)]


@pytest.mark.parametrize("B,S,H,Hkv,dh", CASES)
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("two_tiles", [True, False])
def test_forward(B, S, H, Hkv, dh, causal, two_tiles, monkeypatch):
    # two_tiles: the kernel with two query tiles per CTA, also where the rule on sizes would not choose it
    monkeypatch.setattr(A, "FWD_TWO_TILES", two_tiles)
    monkeypatch.setattr(A, "_two_tiles_win", lambda *a: True)
    qkv = _qkv(B, S, H, Hkv, dh)
    o, lse = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    _lib.check_status()
    o_ref, lse_ref = A.attention_ref(qkv, B, S, H, Hkv, dh, causal=causal)
    assert (o.float() - o_ref).abs().max().item() < 3e-2
    assert (lse - lse_ref).abs().max().item() < 2e-2
    o2, _ = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    assert torch.equal(o, o2)


@pytest.mark.parametrize("causal", [True, False])
def test_forward_growing_maxima(causal, monkeypatch):
    # keys grow along the sequence, so row maxima rise by more than 2^8 from block to block and the
    # output accumulator in tensor memory is rescaled many times
    monkeypatch.setattr(A, "FWD_TWO_TILES", True)
    monkeypatch.setattr(A, "_two_tiles_win", lambda *a: True)
    B, S, H, Hkv, dh = 2, 1024, 4, 2, 64
    qkv = _qkv(B, S, H, Hkv, dh, seed=5).float().reshape(B, S, H + 2 * Hkv, dh)
    ramp = (1.0 + 6.0 * torch.arange(S, device="cuda") / S).reshape(1, S, 1, 1)
    qkv[:, :, H:H + Hkv] *= ramp
    qkv = qkv.reshape(B * S, -1).to(torch.bfloat16)
    o, lse = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    _lib.check_status()
    o_ref, lse_ref = A.attention_ref(qkv, B, S, H, Hkv, dh, causal=causal)
    assert (o.float() - o_ref).abs().max().item() < 3e-2
    assert (lse - lse_ref).abs().max().item() < 2e-2
    monkeypatch.setattr(A, "FWD_TWO_TILES", False)
    o1, lse1 = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    assert (o.float() - o1.float()).abs().max().item() < 2e-2 and (lse - lse1).abs().max().item() < 1e-3


@pytest.mark.parametrize("scale", [0.0, -0.1])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H,Hkv,dh", [(2, 300, 4, 2, 64), (1, 300, 2, 1, 128), (1, 513, 2, 2, 128)])
@pytest.mark.parametrize("two_tiles", [True, False])
def test_forward_takes_any_scale(two_tiles, B, S, H, Hkv, dh, causal, scale, monkeypatch):
    # a masked weight is zero whatever the scale makes of its score: at zero every visible key weighs the same
    monkeypatch.setattr(A, "FWD_TWO_TILES", two_tiles)
    monkeypatch.setattr(A, "_two_tiles_win", lambda *a: True)
    qkv = _qkv(B, S, H, Hkv, dh, seed=11)
    o, lse = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal, scale=scale)
    _lib.check_status()
    o_ref, lse_ref = A.attention_ref(qkv, B, S, H, Hkv, dh, causal=causal, scale=scale)
    # weights and output are rounded to bf16 once each (2^-9 of values of up to 5); sums are fp32
    assert (o.float() - o_ref).abs().max().item() < 3e-2
    assert (lse - lse_ref).abs().max().item() < 1e-3


@pytest.mark.parametrize("B,S,H,Hkv,dh", CASES)
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("spill", [True, False])
def test_backward(B, S, H, Hkv, dh, causal, spill, monkeypatch):
    # spill: dQ streams the dS tiles stored by the dK/dV kernel; otherwise it recomputes the scores
    monkeypatch.setattr(A, "DS_SCRATCH_LIMIT_BYTES", (4 << 30) if spill else 0)
    qkv = _qkv(B, S, H, Hkv, dh, seed=1)
    g = torch.Generator(device="cuda").manual_seed(2)
    do = torch.randn(B * S, H * dh, generator=g, device="cuda").to(torch.bfloat16)
    o, lse = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    d = A.attention_bwd(qkv, o, lse, do, B, S, H, Hkv, dh, causal=causal)
    _lib.check_status()
    ref = A.attention_bwd_ref(qkv, do, B, S, H, Hkv, dh, causal=causal)
    err = (d.float() - ref).abs().max().item()
    assert err < 3e-2 * max(1.0, ref.abs().max().item()), err
    d2 = A.attention_bwd(qkv, o, lse, do, B, S, H, Hkv, dh, causal=causal)
    assert torch.equal(d, d2)


@pytest.mark.parametrize("B,S,H,Hkv", [(1, 1, 1, 1), (2, 127, 2, 1), (1, 129, 2, 2), (3, 256, 4, 1), (1, 257, 2, 1),
                                       (2, 1000, 4, 2), (1, 2048, 8, 2)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dh", [64, 128])
def test_forward_two_tiles_at_tile_edges(B, S, H, Hkv, causal, dh, monkeypatch):
    """Tile edges of the two-tile kernel (second tile empty, one row, full; at 128 K in two stages, V in half tiles)
    against the dense statement and, with growing keys (the accumulator is rescaled), the one-tile kernel: both keep P in
    bf16 (2^-8 of each term), so they agree to 2^-7 of the largest value."""
    qkv = _qkv(B, S, H, Hkv, dh, seed=S).float().reshape(B, S, H + 2 * Hkv, dh)
    qkv[:, :, H:H + Hkv] *= (1.0 + 4.0 * torch.arange(S, device="cuda") / S).reshape(1, S, 1, 1)
    qkv = qkv.reshape(B * S, -1).to(torch.bfloat16)
    monkeypatch.setattr(A, "FWD_TWO_TILES", True)
    monkeypatch.setattr(A, "_two_tiles_win", lambda *a: True)
    o, lse = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    again, _ = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    monkeypatch.setattr(A, "FWD_TWO_TILES", False)
    o1, lse1 = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    _lib.check_status()
    o_ref, lse_ref = A.attention_ref(qkv, B, S, H, Hkv, dh, causal=causal)
    assert torch.equal(o, again)
    assert (o.float() - o_ref).abs().max().item() < 3e-2
    assert (lse - lse_ref).abs().max().item() < 2e-2
    assert (o.float() - o1.float()).abs().max().item() <= 2 ** -7 * o_ref.abs().max().item()


@pytest.mark.parametrize("B,S,H,Hkv,dh", [(1, 1, 1, 1, 128), (1, 129, 4, 1, 128), (2, 640, 8, 2, 128), (1, 640, 6, 2, 64),
                                          (3, 255, 2, 2, 64)])
@pytest.mark.parametrize("causal", [True, False])
def test_backward_pipeline_edges(B, S, H, Hkv, dh, causal):
    """One iteration, an odd and an even number, several heads per kv head: the dK / dV pipeline with its single P buffer
    (and, at 128, single dO and dS) against the fp32 statement, twice with the same bits."""
    qkv = _qkv(B, S, H, Hkv, dh, seed=7)
    do = torch.randn(B * S, H * dh, generator=torch.Generator(device="cuda").manual_seed(8), device="cuda").to(torch.bfloat16)
    o, lse = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
    d = A.attention_bwd(qkv, o, lse, do, B, S, H, Hkv, dh, causal=causal)
    assert torch.equal(d, A.attention_bwd(qkv, o, lse, do, B, S, H, Hkv, dh, causal=causal))
    _lib.check_status()
    ref = A.attention_bwd_ref(qkv, do, B, S, H, Hkv, dh, causal=causal)
    assert (d.float() - ref).abs().max().item() < 3e-2 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("causal,scale", [(True, 1.0), (True, 2.0), (False, 3.0)])
def test_two_tiles_at_128_are_as_exact_as_one(causal, scale, monkeypatch):
    """Against float64, on scores of growing spread: the two-tile kernel refers P to the running maximum, as the one-tile
    kernel does, so the largest weight of a row is exactly 1 in bf16 in both. What is left between them is the order of
    the fp32 sums, far below the 2^-9 of P and of the output: a thousandth of the error, where a reference that lags the
    maximum costs 2 % (unit scores) to 20 %."""
    B, S, H, Hkv, dh = 1, 1500, 4, 1, 128
    qkv = _qkv(B, S, H, Hkv, dh, seed=21).float()
    qkv[:, :(H + Hkv) * dh] *= scale
    qkv = qkv.to(torch.bfloat16)
    x = qkv.double().reshape(S, H + 2 * Hkv, dh)
    sc = torch.einsum("qhd,kd->hqk", x[:, :H], x[:, H]) / dh ** 0.5
    if causal:
        sc = sc.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = torch.einsum("hqk,kd->qhd", torch.softmax(sc, -1), x[:, H + Hkv]).reshape(S, H * dh)
    err = []
    for two in (False, True):
        monkeypatch.setattr(A, "_two_tiles_win", lambda *a: two)
        o, _ = A.attention_fwd(qkv, B, S, H, Hkv, dh, causal=causal)
        err.append(((o.double() - ref).norm() / ref.norm()).item())
    _lib.check_status()
    assert err[1] <= err[0] * 1.001, err


@pytest.mark.parametrize("B,S,H,Hkv,dh", [(2, 200, 4, 2, 64), (1, 333, 2, 1, 128)])
def test_backward_of_rows_with_a_pitch(B, S, H, Hkv, dh):
    """qkv as columns of a wider matrix: the gradient has that row pitch too, of memory that is its own, and the bits of the dense one."""
    ld = (H + 2 * Hkv) * dh
    g = torch.Generator(device="cuda").manual_seed(1)
    wide = torch.randn(B * S, ld + 64, generator=g, device="cuda").to(torch.bfloat16)
    do = torch.randn(B * S, H * dh, generator=g, device="cuda").to(torch.bfloat16)
    qkv, dense = wide[:, :ld], wide[:, :ld].contiguous()
    o, lse = A.attention_fwd(dense, B, S, H, Hkv, dh)
    want = A.attention_bwd(dense, o, lse, do, B, S, H, Hkv, dh)
    got = A.attention_bwd(qkv, o, lse, do, B, S, H, Hkv, dh)
    _lib.check_status()
    assert want.is_contiguous() and got.stride() == qkv.stride() and torch.equal(got, want)
    assert got.untyped_storage().nbytes() >= B * S * (ld + 64) * 2


def test_backward_scratch_belongs_to_a_stream():
    """The dS tiles of two passes that may run at once lie in buffers of their own; a pass after another on its stream takes the same."""
    device = torch.device("cuda", torch.cuda.current_device())
    first = A._scratch(1, 64, 2, device)
    with torch.cuda.stream(torch.cuda.Stream()):
        other = A._scratch(1, 64, 2, device)
        assert A._scratch(1, 64, 2, device) is other
    assert A._scratch(1, 64, 2, device) is first and other.data_ptr() != first.data_ptr()
