"""Convolutional ops on NHWC bf16 activations (csrc/conv.cu + the tcgen05 GEMM): convolution as implicit
GEMMs whose patch operand is fetched by TMA (forward, weight gradient, stride-1 input gradient), or with an explicit
patch matrix where the shape does not tile (im2col -> GEMM, col2im for the input gradient), max pooling, BatchNorm2d with optional fused ReLU. Activations are ``[B*H*W, C]``
matrices; ``ConvGeom`` carries the spatial shape. CPU tensors run the fp32 PyTorch statement
(``torch.nn.functional``), which is also the oracle of the GPU tests."""
from __future__ import annotations

from dataclasses import dataclass

import torch
import torch.nn.functional as F

from . import _lib
from . import gemm as G

BF = torch.bfloat16
vp, i32, f32, sz = _lib.vp, _lib.i32, _lib.f32, _lib.sz
_lib.register("sb_im2col_nhwc", [vp, vp] + [i32] * 11 + [vp])
_lib.register("sb_col2im_nhwc", [vp, vp] + [i32] * 11 + [vp])
_lib.register("sb_maxpool_fwd", [vp, vp, vp] + [i32] * 8 + [vp])
_lib.register("sb_maxpool_bwd", [vp, vp, vp] + [i32] * 8 + [vp])
_lib.register("sb_bn_layer_fwd", [vp] * 10 + [i32, i32, f32, f32, i32, vp])
_lib.register("sb_bn_layer_bwd", [vp] * 11 + [i32, i32, vp])
_lib.register("sb_bias_act", [vp, vp, vp, sz, i32, i32, vp])


@dataclass(frozen=True)
class ConvGeom:
    B: int
    H: int
    W: int
    C: int

    @property
    def rows(self):
        return self.B * self.H * self.W


def _pad8(n):
    return (n + 7) // 8 * 8


def nchw_to_rows(x4: torch.Tensor):
    B, C, H, W = x4.shape
    return x4.permute(0, 2, 3, 1).reshape(B * H * W, C).contiguous(), ConvGeom(B, H, W, C)


def rows_to_nchw(x: torch.Tensor, g: ConvGeom):
    return x.reshape(g.B, g.H, g.W, g.C).permute(0, 3, 1, 2).contiguous()


def pack_conv_weight(w_ref: torch.Tensor, in_c: int, k: int) -> torch.Tensor:
    """Reference layout ``(out_c, in_c*k*k)`` with (c, kh, kw) order -> ``[out_c, pad8(k*k*in_c)]`` with
    (kh, kw, c) order, the column order of the NHWC patches."""
    oc = w_ref.shape[0]
    w = w_ref.reshape(oc, in_c, k, k).permute(0, 2, 3, 1).reshape(oc, k * k * in_c)
    out = torch.zeros((oc, _pad8(k * k * in_c)), dtype=w_ref.dtype, device=w_ref.device)
    out[:, : k * k * in_c] = w
    return out


def unpack_conv_weight(wp: torch.Tensor, in_c: int, k: int) -> torch.Tensor:
    oc = wp.shape[0]
    return wp[:, : k * k * in_c].reshape(oc, k, k, in_c).permute(0, 3, 1, 2).reshape(oc, in_c * k * k)


_lib.register("sb_conv_gemm", [i32, vp, vp, vp] + [i32] * 11 + [vp, vp, vp])
_lib.register("sb_conv_fprop_keep", [vp, vp, vp, vp] + [i32] * 11 + [vp, vp, vp])
_FPROP, _WGRAD, _DGRAD, _WGRAD_F32 = 1, 2, 3, 4


def _rows_tile(oh: int, ow: int, box: int) -> bool:
    """Whether ``box`` consecutive pixels of an oh x ow grid are whole rows of one image or whole images."""
    if oh < 1 or ow < 1 or ow > box or box % ow:
        return False
    rows = box // ow
    return oh % rows == 0 if rows <= oh else rows % oh == 0


def implicit_ok(geom: ConvGeom, oc: int, k: int, stride: int, pad: int) -> bool:
    """Whether a convolution runs without a patch matrix (csrc/gemm_tcgen05.cu: ``sb_conv_gemm``): channels in whole
    64-wide blocks and output rows that tile the 128-pixel operand (and the weight gradient's 64-pixel one). Others
    (an RGB stem, odd image sizes) gather their patches first, and so do those without a pixel, which the native call refuses."""
    oh, ow = (geom.H + 2 * pad - k) // stride + 1, (geom.W + 2 * pad - k) // stride + 1
    return (geom.B > 0 and geom.C % 64 == 0 and oc % 64 == 0 and stride <= 8 and _rows_tile(oh, ow, 128) and _rows_tile(oh, ow, 64)
            and (ow - 1) * stride < 256 and (128 // ow - 1) * stride < 256)


def _conv_gemm(mode, a, b, geom, oc, k, stride, pad, OH, OW, keep=None, f32=False):
    pix_o, pix_i, kp = geom.B * OH * OW, geom.rows, k * k * geom.C
    M, N, K = ((pix_o, oc, kp) if mode == _FPROP else (oc, kp, pix_o) if mode == _WGRAD else (pix_i, geom.C, k * k * oc))
    # one wave of work items, at least eight 64-deep k-blocks each (a weight gradient has K = pixels and few tiles)
    tiles = ((M + 127) // 128) * ((N + 255) // 256)
    splits = max(1, min(G.num_sms(a.device) // tiles, (K + 63) // 64 // 8, 64))
    if f32 and splits > 1:                              # the sum of the splits is written as it is
        mode, dtype = _WGRAD_F32, torch.float32
    else:
        dtype = BF
    out = _lib.empty((M, N), dtype, a.device)
    ws = G._workspace(splits * M * N, a.device) if splits > 1 else None
    rest = (geom.B, geom.H, geom.W, geom.C, oc, k, stride, pad, OH, OW, splits, _lib.ptr(ws),
            _lib.status_word(a.device).data_ptr(), _lib.stream())
    if keep is None:
        _lib.call("sb_conv_gemm", mode, a.data_ptr(), b.data_ptr(), out.data_ptr(), *rest)
    else:
        _lib.call("sb_conv_fprop_keep", a.data_ptr(), b.data_ptr(), out.data_ptr(), keep.data_ptr(), *rest)
    G.launch_count += 2 if splits > 1 else 1
    return out.float() if f32 and dtype == BF else out


class _Conv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, wp, geom, k, stride, pad, want_dw, master=False):
        B, H, W, C = geom.B, geom.H, geom.W, geom.C
        ctx.master = master
        if master:                                      # fp32 weights: rounded here, and their gradient is fp32 too
            w32, wp = wp.contiguous(), _lib.empty(wp.shape, BF, wp.device)
            _lib.call("sb_cast", w32.data_ptr(), wp.data_ptr(), wp.numel(), 1, 1.0, _lib.stream())
            G.launch_count += 1
        OH, OW = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
        ctx.meta = (geom, k, stride, pad, OH, OW)
        ctx.implicit = implicit_ok(geom, wp.shape[0], k, stride, pad) and _tma_ok(x, wp, geom, k)
        if ctx.implicit:
            # a copy, as the patch matrix is one: the caller's tensor may be written before the backward pass, also by
            # kernels that its version counter does not see (128 x 32 x 32 x 64: 7 us, where the patch matrix took 86)
            keep = torch.empty_like(x) if want_dw else None
            ctx.save_for_backward(keep, wp)
            return _conv_gemm(_FPROP, x, wp, geom, wp.shape[0], k, stride, pad, OH, OW, keep)
        Kp = wp.shape[1]
        col = _lib.empty((B * OH * OW, Kp), BF, x.device)
        _lib.call("sb_im2col_nhwc", x.data_ptr(), col.data_ptr(), B, H, W, C, k, k, stride, pad, OH, OW, Kp,
                  _lib.stream())
        G.launch_count += 1
        y = G.matmul_nt(col, wp)
        ctx.save_for_backward(col, wp)
        return y

    @staticmethod
    def backward(ctx, dy):
        col, wp = ctx.saved_tensors                           # col: a copy of the input when no patch matrix was made
        geom, k, stride, pad, OH, OW = ctx.meta
        oc = wp.shape[0]
        dy = dy.contiguous()
        implicit = ctx.implicit and dy.dtype == BF and dy.data_ptr() % 16 == 0
        if ctx.implicit and not implicit:
            raise ValueError("conv2d: the output gradient must be bf16 and 16-byte aligned")
        dx = dw = None
        if ctx.needs_input_grad[1]:
            if implicit:
                dw = _conv_gemm(_WGRAD, dy, col, geom, oc, k, stride, pad, OH, OW, f32=ctx.master)
            else:
                dw = G.matmul_tn(dy, col)                     # [oc, Kp] = dy^T col
                if ctx.master:
                    dw = dw.float()
        if ctx.needs_input_grad[0]:
            if implicit and stride == 1 and _rows_tile(geom.H, geom.W, 128):
                return _conv_gemm(_DGRAD, dy, wp, geom, oc, k, stride, pad, OH, OW), dw, None, None, None, None, None, None
            dcol = G.matmul_nn(dy, wp)                        # [M, Kp]
            dx = _lib.empty((geom.rows, geom.C), BF, dy.device)
            _lib.call("sb_col2im_nhwc", dcol.data_ptr(), dx.data_ptr(), geom.B, geom.H, geom.W, geom.C, k, k, stride,
                      pad, OH, OW, wp.shape[1], _lib.stream())
            G.launch_count += 1
        return dx, dw, None, None, None, None, None, None


def _tma_ok(x, wp, geom, k) -> bool:
    """Types, shapes and 16-byte bases of the operands as the tensor maps need them; others take the patch matrix."""
    return (x.dtype == BF and wp.dtype == BF and wp.is_contiguous() and x.data_ptr() % 16 == 0
            and wp.data_ptr() % 16 == 0 and wp.shape[1] == k * k * geom.C and x.numel() == geom.rows * geom.C)


def conv2d(x, wp, geom: ConvGeom, k: int, stride: int = 1, pad: int = 0):
    """x [B*H*W, C], wp packed weight [oc, pad8(k*k*C)] -> (y [B*OH*OW, oc], geometry of y)."""
    OH, OW = (geom.H + 2 * pad - k) // stride + 1, (geom.W + 2 * pad - k) // stride + 1
    og = ConvGeom(geom.B, OH, OW, wp.shape[0])
    if not x.is_cuda:
        w4 = wp[:, : k * k * geom.C].reshape(wp.shape[0], k, k, geom.C).permute(0, 3, 1, 2)
        y4 = F.conv2d(rows_to_nchw(x.float(), geom), w4.float(), stride=stride, padding=pad)
        return nchw_to_rows(y4.to(x.dtype))[0], og
    want_dw = torch.is_grad_enabled() and wp.requires_grad
    return _Conv.apply(x.contiguous(), wp, geom, k, stride, pad, want_dw), og


def conv2d_master(x, w32, geom: ConvGeom, k: int, stride: int = 1, pad: int = 0):
    """``conv2d(x, w32.to(bfloat16), ...)`` for fp32 master weights, as one node of the graph: the same y and dx to the bit, and a
    weight gradient that is not rounded to bf16 where its sum is split."""
    if not x.is_cuda or w32.dtype != torch.float32 or w32.device != x.device:
        return conv2d(x, w32.to(BF), geom, k, stride, pad)
    og = ConvGeom(geom.B, (geom.H + 2 * pad - k) // stride + 1, (geom.W + 2 * pad - k) // stride + 1, w32.shape[0])
    want_dw = torch.is_grad_enabled() and w32.requires_grad
    return _Conv.apply(x.contiguous(), w32, geom, k, stride, pad, want_dw, True), og


class _MaxPool(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, geom, k, stride):
        B, H, W, C = geom.B, geom.H, geom.W, geom.C
        OH, OW = (H - k) // stride + 1, (W - k) // stride + 1
        y = _lib.empty((B * OH * OW, C), BF, x.device)
        arg = _lib.empty((B * OH * OW, C), torch.uint8, x.device)
        _lib.call("sb_maxpool_fwd", x.data_ptr(), y.data_ptr(), arg.data_ptr(), B, H, W, C, k, stride, OH, OW,
                  _lib.stream())
        G.launch_count += 1
        ctx.save_for_backward(arg)
        ctx.meta = (geom, k, stride, OH, OW)
        return y

    @staticmethod
    def backward(ctx, dy):
        (arg,) = ctx.saved_tensors
        geom, k, stride, OH, OW = ctx.meta
        dx = _lib.empty((geom.rows, geom.C), BF, dy.device)
        _lib.call("sb_maxpool_bwd", dy.contiguous().data_ptr(), arg.data_ptr(), dx.data_ptr(), geom.B, geom.H, geom.W,
                  geom.C, k, stride, OH, OW, _lib.stream())
        G.launch_count += 1
        return dx, None, None, None


def maxpool2d(x, geom: ConvGeom, k: int, stride: int):
    OH, OW = (geom.H - k) // stride + 1, (geom.W - k) // stride + 1
    og = ConvGeom(geom.B, OH, OW, geom.C)
    if not x.is_cuda:
        return nchw_to_rows(F.max_pool2d(rows_to_nchw(x, geom), k, stride))[0], og
    return _MaxPool.apply(x.contiguous(), geom, k, stride), og


class _BatchNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gamma, beta, run_mean, run_var, eps, momentum, relu, training, shortcut=None):
        rows, C = x.shape
        stat = _lib.empty((2, C), torch.float32, x.device)          # mean, 1 / standard deviation
        mean_p = stat.data_ptr()
        inv_p = mean_p + 4 * C
        part = None
        if training:
            part = torch.empty(2 * ((rows + 255) // 256) * C, dtype=torch.float32, device=x.device)
        else:
            stat[0].copy_(run_mean)
            stat[1].copy_(torch.rsqrt(run_var + eps))
        y = torch.empty_like(x)
        _lib.call("sb_bn_layer_fwd", x.data_ptr(), _lib.ptr(part), gamma.data_ptr(), beta.data_ptr(), mean_p, inv_p,
                  _lib.ptr(run_mean) if training else None, _lib.ptr(run_var) if training else None, _lib.ptr(shortcut),
                  y.data_ptr(), rows, C, float(eps), float(momentum), int(relu), _lib.stream())
        G.launch_count += 3 if training else 1
        ctx.save_for_backward(x, y, gamma, stat)
        ctx.relu, ctx.added = relu, shortcut is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        x, y, gamma, stat = ctx.saved_tensors
        rows, C = x.shape
        dy = dy.contiguous()
        mask = y if ctx.relu else None                  # the ReLU's mask is applied where dy is read
        ds = None
        if ctx.added and not ctx.relu:
            ds = dy
        elif ctx.added:                                 # the masked dy, written by the kernel that reads dy first
            ds = torch.empty_like(x)
            # which takes whole words only; the saved tensors may come from a hook
            dy, x, mask = (t if t.data_ptr() % 16 == 0 else t.clone() for t in (dy, x, mask))
        part = torch.empty(2 * ((rows + 255) // 256) * C, dtype=torch.float32, device=x.device)
        dgamma = _lib.empty(C, torch.float32, x.device)
        dbeta = _lib.empty(C, torch.float32, x.device)
        dx = torch.empty_like(x)
        mean_p = stat.data_ptr()
        _lib.call("sb_bn_layer_bwd", dy.data_ptr(), x.data_ptr(), _lib.ptr(mask), _lib.ptr(ds) if ctx.relu else None,
                  part.data_ptr(), mean_p, mean_p + 4 * C, gamma.data_ptr(), dgamma.data_ptr(), dbeta.data_ptr(), dx.data_ptr(),
                  rows, C, _lib.stream())
        G.launch_count += 3
        return dx, dgamma, dbeta, None, None, None, None, None, None, ds


def _adds_inside(x, gamma, beta, shortcut) -> bool:
    """Whether the BatchNorm kernels add ``shortcut`` themselves: whole 16-byte words of eight channels everywhere, within the range of
    their indexes (words) and grids (chunks of 256 rows). Else two torch operators do."""
    return (x.dtype == BF and shortcut.dtype == BF and shortcut.shape == x.shape and x.shape[1] % 8 == 0
            and x.numel() // 8 <= 0x7fffff00 and x.shape[0] <= 65535 * 256 and x.device == shortcut.device
            and all(t.is_contiguous() and t.data_ptr() % 16 == 0 for t in (x, shortcut, gamma, beta)))


def batchnorm(x, gamma, beta, run_mean, run_var, eps=1e-5, momentum=0.1, relu=False, training=True, shortcut=None):
    """Per-channel batch norm of [rows, C] (fp32 gamma/beta/running stats), optional fused ReLU. ``shortcut`` is added to the
    rounded result before the ReLU, with the results of ``relu(batchnorm(x) + shortcut)`` to the bit."""
    if not x.is_cuda:
        y = F.batch_norm(x.float().t().unsqueeze(0), run_mean, run_var, gamma, beta, training, momentum, eps)[0].t()
        if shortcut is not None:
            y = y.to(x.dtype) + shortcut
        return (torch.relu(y) if relu else y).to(x.dtype)
    x = x.contiguous()
    if shortcut is not None and not _adds_inside(x, gamma, beta, shortcut):
        y = _BatchNorm.apply(x, gamma, beta, run_mean, run_var, eps, momentum, False, training) + shortcut
        return torch.relu(y) if relu else y
    return _BatchNorm.apply(x, gamma, beta, run_mean, run_var, eps, momentum, relu, training, shortcut)


def bias_act(x, bias, relu=False):
    """y = act(x + bias[c]) with fp32 bias; differentiable through PyTorch for the bias."""
    if not x.is_cuda or torch.is_grad_enabled():
        y = x + bias.to(x.dtype) if bias is not None else x
        return torch.relu(y) if relu else y
    y = torch.empty_like(x)
    _lib.call("sb_bias_act", x.data_ptr(), _lib.ptr(bias), y.data_ptr(), x.numel(), x.shape[1], int(relu), _lib.stream())
    return y
