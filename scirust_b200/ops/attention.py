"""GQA flash attention (prefill / training) on the tcgen05 kernels in csrc/attention_*_tcgen05.cu.

The activation layout is the fused projection output ``qkv [B*S, (H + 2*Hkv) * dh]`` (q heads, k heads,
v heads; RoPE already applied to q and k), so no per-head slicing copies exist (the reference slices and
re-concatenates per head: scirust-sciagent/src/cuda_model.rs:796-869).
"""
from __future__ import annotations

import math
import os

import torch

from . import _lib
from . import gemm as _g

_lib.register("sb_attention_fwd", [_lib.vp, _lib.vp, _lib.vp, _lib.i32, _lib.i32, _lib.i32, _lib.i32, _lib.i32,
                                   _lib.i32, _lib.i32, _lib.f32, _lib.i32, _lib.vp, _lib.vp])
_lib.register("sb_attention_fwd_pp", [_lib.vp, _lib.vp, _lib.vp, _lib.i32, _lib.i32, _lib.i32, _lib.i32, _lib.i32,
                                      _lib.i32, _lib.i32, _lib.f32, _lib.i32, _lib.vp, _lib.vp])
_lib.register("sb_attention_bwd", [_lib.vp, _lib.vp, _lib.vp, _lib.vp, _lib.vp, _lib.vp, _lib.vp, _lib.i32, _lib.i32,
                                   _lib.i32, _lib.i32, _lib.i32, _lib.i32, _lib.i32, _lib.i32, _lib.f32,
                                   _lib.i32, _lib.vp, _lib.vp])

# The forward pass has a kernel with two query tiles per CTA, whose output accumulator stays in tensor memory, and one with one;
# sizes choose (_two_tiles_win). SB_ATT_FWD=single selects the one-tile kernel throughout.
FWD_TWO_TILES = os.environ.get("SB_ATT_FWD", "pair") != "single"


def _two_tiles_win(B, S, H, dh, causal, device) -> bool:
    """Which of the two kernels runs, by the CTAs that each of them starts.

    Head dimension 128 (one CTA per SM in both): a CTA of two tiles took about 1.7 times as long as one of a single
    tile when these lines were drawn, so while its grid fits the GPU at once one tile runs, and beyond that two must save
    waves: sequences of up to 256 rows need more than 1.5 times fewer, up to 384 (the second CTA of a head has one tile)
    1.5 times, longer ones always do. The two-tile kernel has become the faster by more since, and the lines lie too far
    out by up to a third. Causal, 32 heads, us, one tile / two: taken as two 1 x 1300 43.0 / 29.2, 2 x 1000 49.2 / 32.8,
    9 x 256 28.9 / 20.8; as one 1 x 128 6.5 / 6.7, 2 x 256 8.9 / 10.3, 3 x 333 17.4 / 18.7, and, where two would be faster,
    1 x 1000 25.1 / 23.4, 2 x 512 18.9 / 15.3, 4 x 256 15.0 / 11.0, 5 x 333 30.1 / 27.6, 12 x 333 63.1 / 53.3.

    Head dimension 64 (two CTAs per SM with one tile, one with two), 16 heads: while the two-tile grid fits the GPU at
    once one tile runs for causal sequences, but past 512 rows for an even number of tiles only (the longest tile
    of an odd number runs alone in its CTA): 1 x 512 10.7 / 11.6, 1 x 1000 17.8 / 18.8, but 3 x 600 13.9 / 12.2; without
    the mask up to 384 rows only: 3 x 333 9.6 / 11.6, but 2 x 1000 22.2 / 21.2. Off the faster side by now: causal 3 x 333
    9.1 / 8.1 (one runs), 16 x 100 7.4 / 10.3 (two run), without the mask 1 x 512 10.6 / 12.8 (two run)."""
    sms, tiles = _g.num_sms(device), (S + 127) // 128
    one, two = B * H * tiles, B * H * ((S + 255) // 256)
    if dh == 64:
        fewer = (S <= 512 or tiles % 2 == 0) if causal else S <= 384
        return two > sms or not fewer
    if two <= sms or S <= 128:
        return False
    one, two = -(-one // sms), -(-two // sms)          # waves
    return S > 384 or (2 * one >= 3 * two if S > 256 else 2 * one > 3 * two)


# The backward pass spills its dS tiles (bf16 [B*H, S, S]) to a scratch buffer so that dQ is a streamed
# product instead of a second pass over scores and exponentials; above this size it recomputes instead.
DS_SCRATCH_LIMIT_BYTES = int(os.environ.get("SB_ATT_DS_SCRATCH_MB", "4096")) << 20
_ds_scratch: dict = {}


def _scratch(B, S, H, device):
    n = B * H * S * ((S + 63) // 64 * 64)
    if n * 2 > DS_SCRATCH_LIMIT_BYTES:
        return None
    key = str(device)
    t = _ds_scratch.get(key)
    if t is None or t.numel() < n:
        t = _lib.empty(n, torch.bfloat16, device)
        _ds_scratch[key] = t
    return t


def attention_ref(qkv, B, S, H, Hkv, dh, causal=True, scale=None):
    """fp32 dense reference: returns (O [B*S, H*dh] fp32, LSE [B,H,S] fp32)."""
    scale = 1.0 / math.sqrt(dh) if scale is None else scale
    x = qkv.float().reshape(B, S, H + 2 * Hkv, dh)
    q = x[:, :, :H].permute(0, 2, 1, 3)
    k = x[:, :, H:H + Hkv].permute(0, 2, 1, 3).repeat_interleave(H // Hkv, 1)
    v = x[:, :, H + Hkv:].permute(0, 2, 1, 3).repeat_interleave(H // Hkv, 1)
    s = torch.matmul(q, k.transpose(-1, -2)) * scale
    if causal:
        mask = torch.triu(torch.ones(S, S, dtype=torch.bool, device=qkv.device), 1)
        s = s.masked_fill(mask, float("-inf"))
    lse = torch.logsumexp(s, -1)
    o = torch.matmul(torch.softmax(s, -1), v)
    return o.permute(0, 2, 1, 3).reshape(B * S, H * dh), lse


def attention_fwd(qkv, B, S, H, Hkv, dh, causal=True, scale=None, want_lse=True):
    scale = 1.0 / math.sqrt(dh) if scale is None else scale
    if not qkv.is_cuda:
        o, lse = attention_ref(qkv, B, S, H, Hkv, dh, causal, scale)
        return o.to(qkv.dtype), lse
    if qkv.dim() != 2 or qkv.stride(1) != 1 or qkv.dtype != torch.bfloat16:
        raise ValueError("qkv must be a 2-D bf16 matrix with unit inner stride")
    out = _lib.empty((B * S, H * dh), torch.bfloat16, qkv.device)
    lse = _lib.empty((B, H, S), torch.float32, qkv.device) if want_lse else None
    entry = "sb_attention_fwd_pp" if FWD_TWO_TILES and _two_tiles_win(B, S, H, dh, causal, qkv.device) else "sb_attention_fwd"
    _lib.call(entry, qkv.data_ptr(), out.data_ptr(), _lib.ptr(lse), B, S, H, Hkv, dh, qkv.stride(0),
              out.stride(0), float(scale), int(causal), _lib.status_word(qkv.device).data_ptr(), _lib.stream())
    _g.launch_count += 1
    return out, lse


def attention_bwd_ref(qkv, do, B, S, H, Hkv, dh, causal=True, scale=None):
    with torch.enable_grad():
        x = qkv.detach().float().requires_grad_(True)
        o, _ = attention_ref(x, B, S, H, Hkv, dh, causal, scale)
        (g,) = torch.autograd.grad(o, x, do.float())
    return g


def attention_bwd_flash_ref(qkv, o, lse, do, B, S, H, Hkv, dh, causal=True, scale=None):
    """fp32 statement of the flash backward, written on the SAVED normaliser and output like the kernels:
    P = exp(S - lse), delta = rowsum(dO * O), dS = P * (dP - delta). With the block's own (o, lse) it equals
    ``attention_bwd_ref``; with the merged (o, lse) of a ring of KV blocks it is that block's share of the gradient,
    which is what context parallelism needs."""
    scale = 1.0 / math.sqrt(dh) if scale is None else scale
    rep = H // Hkv
    x = qkv.float().reshape(B, S, H + 2 * Hkv, dh)
    q = x[:, :, :H].permute(0, 2, 1, 3)
    k = x[:, :, H:H + Hkv].permute(0, 2, 1, 3).repeat_interleave(rep, 1)
    v = x[:, :, H + Hkv:].permute(0, 2, 1, 3).repeat_interleave(rep, 1)
    dof = do.float().reshape(B, S, H, dh).permute(0, 2, 1, 3)
    of = o.float().reshape(B, S, H, dh).permute(0, 2, 1, 3)
    s = torch.matmul(q, k.transpose(-1, -2)) * scale
    p = torch.exp(s - lse.float()[..., None])
    if causal:
        p = p.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=qkv.device), 1), 0.0)
    p = torch.nan_to_num(p, nan=0.0)                       # rows with lse = -inf (no visible key) contribute nothing
    dv = torch.matmul(p.transpose(-1, -2), dof)
    dp = torch.matmul(dof, v.transpose(-1, -2))
    delta = (dof * of).sum(-1, keepdim=True)
    ds = p * (dp - delta)
    dq = torch.matmul(ds, k) * scale
    dk = torch.matmul(ds.transpose(-1, -2), q) * scale
    dk = dk.reshape(B, Hkv, rep, S, dh).sum(2)
    dv = dv.reshape(B, Hkv, rep, S, dh).sum(2)
    g = torch.cat([dq.permute(0, 2, 1, 3), dk.permute(0, 2, 1, 3), dv.permute(0, 2, 1, 3)], 2)
    return g.reshape(B * S, (H + 2 * Hkv) * dh)


def attention_bwd(qkv, o, lse, do, B, S, H, Hkv, dh, causal=True, scale=None):
    """Gradient w.r.t. the fused qkv matrix (same layout), deterministic (no atomics)."""
    scale = 1.0 / math.sqrt(dh) if scale is None else scale
    if not qkv.is_cuda:
        return attention_bwd_flash_ref(qkv, o, lse, do, B, S, H, Hkv, dh, causal, scale).to(qkv.dtype)
    dqkv = torch.empty_like(qkv)
    delta = _lib.empty((B, H, S, 2), torch.float32, qkv.device)
    ds = _scratch(B, S, H, qkv.device)
    _lib.call("sb_attention_bwd", qkv.data_ptr(), o.data_ptr(), lse.data_ptr(), do.data_ptr(), dqkv.data_ptr(),
              delta.data_ptr(), _lib.ptr(ds), B, S, H, Hkv, dh, qkv.stride(0), o.stride(0), do.stride(0), float(scale),
              int(causal), _lib.status_word(qkv.device).data_ptr(), _lib.stream())
    _g.launch_count += 3
    return dqkv
