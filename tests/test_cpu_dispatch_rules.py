"""Rules that choose between two kernels by sizes, on the CPU, for a GPU of 148 SMs: each line is a shape at which both
sides were timed, with the side that the rule takes: the faster one (or, within 2 %, the one that was there first) when the line
was drawn. The attention forward's kernels have changed since its lines were; the rule's comment says where it is off."""
import subprocess
from pathlib import Path

import pytest
import torch

from scirust_b200.models.infer import _WidenAhead
from scirust_b200.ops import attention as A, conv as C, decode as D, gemm as G


@pytest.fixture(autouse=True)
def _sms(monkeypatch):
    monkeypatch.setattr(G, "num_sms", lambda device=None: 148)


@pytest.mark.parametrize("B,S,H,dh,causal,two", [
    # head dimension 128: one tile while the two-tile grid fits, or where it saves too few waves
    (1, 128, 32, 128, True, False), (1, 1000, 32, 128, True, False), (1, 4096, 8, 128, True, False),
    (9, 100, 32, 128, True, False), (5, 256, 32, 128, True, False), (6, 256, 32, 128, True, False),
    (3, 333, 32, 128, True, False), (5, 333, 32, 128, True, False),
    (9, 256, 32, 128, True, True), (9, 333, 32, 128, True, True), (3, 400, 32, 128, True, True),
    (1, 1300, 32, 128, True, True), (2, 1000, 32, 128, False, True), (1, 5000, 32, 128, True, True),
    # head dimension 64
    (1, 512, 16, 64, True, False), (2, 1000, 16, 64, True, False), (3, 333, 16, 64, True, False),
    (3, 600, 16, 64, True, True), (2, 800, 16, 64, True, True), (3, 1000, 16, 64, True, True),
    (3, 333, 16, 64, False, False), (2, 1000, 16, 64, False, True), (1, 4096, 16, 64, True, True),
])
def test_attention_forward_tiles(B, S, H, dh, causal, two):
    assert A._two_tiles_win(B, S, H, dh, causal, None) is two


@pytest.mark.parametrize("B,S,H,dh,causal,two", [
    # two tiles that save a wave, on both sides of the line; without the mask, and past seven tiles without it
    (1, 512, 32, 128, True, False), (2, 512, 32, 128, True, True), (1, 641, 32, 128, True, False), (2, 256, 32, 128, True, False),
    (4, 256, 32, 128, True, True), (2, 256, 32, 128, False, False), (3, 256, 32, 128, False, True), (1, 896, 8, 128, False, False),
    (1, 897, 8, 128, False, True),
    # head dimension 64: short heads keep one tile, five tiles two while their grid fits; without the mask by waves
    (16, 100, 16, 64, True, False), (24, 256, 16, 64, True, False), (12, 384, 16, 64, True, False), (3, 640, 16, 64, True, True),
    (4, 640, 16, 64, True, False), (4, 256, 16, 64, False, False), (5, 256, 16, 64, False, True), (5, 384, 16, 64, False, False),
    (8, 384, 16, 64, False, True), (1, 385, 16, 64, False, True),
])
def test_attention_forward_tiles_by_waves(B, S, H, dh, causal, two):
    assert A._two_tiles_win(B, S, H, dh, causal, None) is two


@pytest.mark.parametrize("B,L,H,Hkv,page,stream", [
    (1, 2048, 32, 8, 64, True), (4, 2048, 32, 8, 128, True), (16, 512, 32, 8, 64, True), (64, 256, 32, 8, 64, True),
    (64, 2048, 32, 8, 64, True), (16, 2304, 32, 2, 64, True), (1, 8192, 16, 2, 64, True),
    (1, 1024, 32, 8, 64, False), (4, 1024, 32, 8, 64, False), (16, 256, 32, 8, 64, False), (64, 128, 32, 8, 64, False),
    # small pages: one thread issues a copy per page
    (16, 2304, 32, 8, 32, True), (64, 2048, 32, 8, 32, False), (1, 8192, 32, 8, 16, True), (4, 2048, 32, 8, 16, True),
    (16, 512, 32, 8, 16, False), (64, 2048, 32, 8, 16, False), (1, 2048, 32, 8, 8, False), (64, 2048, 32, 8, 8, False),
    # few query heads per kv head
    (1, 2048, 8, 8, 64, False), (1, 4096, 8, 8, 64, False), (1, 8192, 8, 8, 64, True), (64, 512, 8, 8, 64, False),
    (64, 2048, 8, 8, 64, True), (32, 256, 32, 32, 64, False), (64, 1024, 32, 32, 64, False), (16, 2304, 32, 32, 64, True),
    (2, 2048, 16, 8, 64, False), (16, 512, 16, 8, 64, True), (32, 256, 16, 8, 64, False), (16, 1024, 24, 8, 32, False),
])
def test_streamed_decode_attention(B, L, H, Hkv, page, stream):
    assert D._stream_wins(L, B * Hkv, H // Hkv, page, None) is stream


@pytest.mark.parametrize("B,L,H,Hkv,page,stream", [
    # lines that lie lower since pieces are merged beside the stream, on both sides
    (64, 192, 32, 8, 64, True), (64, 191, 32, 8, 64, False), (64, 192, 32, 8, 32, False), (2, 1024, 32, 8, 64, True),
    (2, 1023, 32, 8, 64, False), (4, 1536, 32, 8, 64, True), (4, 1535, 32, 8, 64, False), (4, 1536, 32, 8, 32, False),
    (16, 1024, 32, 32, 64, True), (16, 1023, 32, 32, 64, False), (32, 1024, 32, 32, 64, False),
])
def test_streamed_decode_attention_of_shorter_sequences(B, L, H, Hkv, page, stream):
    assert D._stream_wins(L, B * Hkv, H // Hkv, page, None) is stream


def test_kernel_attributes_are_set_for_every_device(tmp_path):
    """The helper of the launchers, with a counting stand-in for the CUDA call: once per device, again after a failure, and
    every time for device numbers beyond its mask."""
    src = tmp_path / "once.cpp"
    src.write_text('''
        #include "per_device.h"
        #include <cstdio>
        #include <initializer_list>
        int main() {
          static sb::PerDeviceOnce once;
          int calls[128] = {}, rc = 0;
          auto set = [&](int d, int r) { return once(d, [&] { ++calls[d]; return r; }); };
          for (int i = 0; i < 3; ++i) for (int d : {0, 1, 63}) rc |= set(d, 0);
          int failed = set(2, -7) == -7 && set(2, -7) == -7;
          rc |= set(2, 0) | set(2, -7);                      // set by now: not called again
          rc |= set(64, 0) | set(64, 0);
          std::printf("%d %d %d %d %d %d %d", rc, failed, calls[0], calls[1], calls[63], calls[2], calls[64]);
        }''')
    csrc = Path(__file__).resolve().parent.parent / "scirust_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(csrc), str(src), "-o", str(tmp_path / "once")], check=True)
    out = subprocess.run([str(tmp_path / "once")], check=True, capture_output=True, text=True).stdout
    assert out == "0 1 1 1 1 3 2"


@pytest.mark.parametrize("B,H,W,Cin,oc,k,stride,pad,implicit", [
    (128, 32, 32, 64, 64, 3, 1, 1, True), (5, 4, 4, 128, 64, 3, 1, 1, True), (2, 32, 16, 128, 64, 3, 2, 1, True),
    (1, 224, 224, 64, 64, 3, 1, 1, False), (4, 28, 28, 64, 64, 3, 1, 1, False), (8, 32, 32, 3, 64, 3, 1, 1, False),
    # no output pixel, no image: the patch path, whose native call reports the error
    (1, 2, 2, 64, 64, 3, 1, 0, False), (1, 8, 2, 64, 64, 3, 1, 0, False), (1, 1, 8, 64, 64, 3, 2, 0, False),
    (0, 32, 32, 64, 64, 3, 1, 1, False),
])
def test_convolution_without_patch_matrix(B, H, W, Cin, oc, k, stride, pad, implicit):
    assert C.implicit_ok(C.ConvGeom(B, H, W, Cin), oc, k, stride, pad) is implicit


@pytest.mark.parametrize("K,N,M,quant,splits", [
    (4096, 4096, 1, True, 18), (14336, 4096, 1, True, 18), (28672, 2048, 1, True, 44), (28672, 3584, 1, True, 42),
    (28672, 2048, 8, True, 18), (512, 2048, 1, True, 8), (512, 2048, 8, True, 4), (1376, 1024, 1, True, 14),
    (2816, 1024, 1, False, 22), (1024, 1024, 1, False, 10), (4096, 6144, 1, False, 12), (64, 256, 1, False, 1),
    (4096, 128256, 1, False, 8), (73728, 256, 8, True, 18), (98304, 256, 8, True, 24),
])
def test_splits_of_the_weight_stream(K, N, M, quant, splits):
    assert D._auto_splits(N, K, 512 if quant else 256, M, quant) == splits


@pytest.mark.parametrize("K,N,M,quant,splits", [
    # up to eight finish in a cluster
    (4096, 4096, 1, False, 8), (14336, 4096, 1, False, 8), (11008, 1024, 1, False, 8), (14336, 8192, 1, False, 8),
    (14336, 3072, 1, True, 8), (14336, 3840, 1, True, 8), (4096, 8704, 1, True, 8), (8192, 4096, 1, True, 8), (14336, 2048, 2, False, 8),
    (14336, 4096, 2, True, 8), (1024, 1536, 1, False, 8), (4096, 128256, 1, True, 2), (28672, 2048, 1, True, 44),
    # one row, a long stream and about one CTA per SM with eight: as many as through memory
    (14336, 1024, 1, False, 74), (14336, 2048, 1, False, 37), (8192, 512, 1, False, 64), (9472, 4608, 1, False, 16),
    (14336, 5120, 1, False, 14), (14336, 4096, 1, True, 18), (9472, 4096, 1, True, 18), (9472, 8704, 1, True, 17),
    (6144, 8704, 1, True, 17), (9472, 12288, 1, True, 12), (14336, 4352, 1, True, 18),
])
def test_splits_that_finish_in_a_cluster(K, N, M, quant, splits):
    assert D._gemv_splits(N, K, 512 if quant else 256, M, quant) == splits


@pytest.mark.parametrize("M,K,ff,fused", [
    # four waves of 256 x 128 tiles on 74 pairs, k of 1024, one whole tile of rows, columns by the eight
    (16384, 1024, 2816, True), (4096, 1024, 2816, True), (4000, 1024, 2816, True), (1024, 4096, 11008, True), (2048, 4096, 14336, True),
    (2048, 1024, 2816, False), (600, 4096, 11008, False), (4096, 512, 1408, False), (16384, 1023, 2816, False), (16384, 1024, 2820, False),
    (512, 1024, 148 * 128, True), (512, 1024, 147 * 128, False),
    (256, 1024, 296 * 128, True), (256, 1024, 295 * 128, False), (255, 1024, 296 * 128, False), (8, 1024, 65536, False),
])
def test_swiglu_in_the_epilogue(M, K, ff, fused, monkeypatch):
    monkeypatch.setattr(G, "FUSE_SWIGLU", None)
    monkeypatch.setattr(G, "PAIR_MODE", "auto")
    assert G.swiglu_in_epilogue(M, K, ff) is fused
    monkeypatch.setattr(G, "FUSE_SWIGLU", True)                     # forced: wherever the kernel takes the call
    assert G.swiglu_in_epilogue(M, K, ff) is (M >= 256 and ff % 8 == 0)
    for name, value in (("PAIR_MODE", "0"), ("FUSE_SWIGLU", False)):
        monkeypatch.setattr(G, name, value)
        assert not G.swiglu_in_epilogue(M, K, ff)


@pytest.mark.parametrize("rows,d,ff,ahead", [
    # 1024 rows, and 2^35 products of rows and elements of gate/up
    (2048, 4096, 14336, True), (1024, 4096, 14336, True), (1023, 4096, 14336, False), (1024, 4096, 4096, True), (1023, 4096, 4096, False),
    (1024, 4096, 4095, False), (8192, 1024, 2816, True), (5958, 1024, 2816, True), (5957, 1024, 2816, False), (2000, 1024, 2816, False),
])
def test_prefill_plans_expansions_for_long_prompts(rows, d, ff, ahead):
    shapes = {"wqkv": (d, 3 * d // 2), "wo": (d, d), "wgu": (d, 2 * ff), "wd": (ff, d)}
    layer = {k: torch.empty(s, dtype=torch.int8, device="meta") for k, s in shapes.items()}
    assert bool(_WidenAhead([layer, layer], rows).order) is ahead
    assert not _WidenAhead([], rows).order
