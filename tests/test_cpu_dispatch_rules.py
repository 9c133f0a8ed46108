"""Rules that choose between two kernels by sizes, on the CPU, for a GPU of 148 SMs: each line is a shape at which both
sides were timed, with the side that was faster (or, within 2 %, the one that was there first)."""
import pytest

from scirust_b200.ops import attention as A, gemm as G


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
