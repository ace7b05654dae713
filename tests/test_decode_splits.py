"""KV-split heuristic of paged decode attention (pure arithmetic; runs without a GPU)."""

import math

import pytest

from axlearn_b200.ops import decode_ops


@pytest.mark.parametrize("batch,kv,group,tokens,want", [
    (32, 32, 1, 2048, 1),      # 1024 CTAs fit the 1184 resident ones: one wave, no split
    (64, 32, 1, 2048, 4),      # 2048 CTAs = 1.73 waves; 4 splits = 6.92 waves of 7
    (16, 4, 1, 2048, 10),      # small grid: split until about four CTAs per SM
    (64, 8, 4, 2048, 9),       # row kernel (two resident CTAs per SM): 9 splits = 3.89 waves of 4
    (16, 8, 4, 2048, 9),
    (64, 16, 2, 2048, 4),      # two query heads per KV head run one per CTA
    (1, 32, 1, 64, 1),         # never below 8 pages per split
])
def test_default_splits(batch, kv, group, tokens, want, monkeypatch):
    monkeypatch.delenv("AXB_DECODE_ATTN", raising=False)
    assert decode_ops.default_splits(batch, kv, group, tokens, 16) == want


def test_last_wave_is_nearly_full_once_past_one_wave(monkeypatch):
    monkeypatch.delenv("AXB_DECODE_ATTN", raising=False)
    for batch in (24, 40, 48, 64, 96, 128, 200):
        for kv, group in ((32, 1), (8, 4), (16, 2)):
            s = decode_ops.default_splits(batch, kv, group, 4096, 16)
            ctas, resident = decode_ops._kernel_shape(batch, kv, group)  # pylint: disable=protected-access
            x = ctas * s / (148 * resident)
            assert 1 <= s <= 32
            if x > 1:
                assert x / math.ceil(x) >= 0.85, (batch, kv, group, s, x)


def test_kernel_shape_follows_the_environment(monkeypatch):
    monkeypatch.delenv("AXB_DECODE_ATTN", raising=False)
    assert decode_ops._kernel_shape(64, 8, 4) == (128, 2)        # pylint: disable=protected-access
    assert decode_ops._kernel_shape(4, 8, 4) == (128, 8)         # few row CTAs: one query head per CTA
    assert decode_ops._kernel_shape(8, 2, 4) == (16, 2)          # KV heads not a multiple of 4: 4 heads per CTA
    monkeypatch.setenv("AXB_DECODE_ATTN", "head")
    assert decode_ops._kernel_shape(64, 8, 4) == (512, 2)        # pylint: disable=protected-access
    monkeypatch.setenv("AXB_DECODE_ATTN", "head1")
    assert decode_ops._kernel_shape(64, 8, 4) == (2048, 8)       # pylint: disable=protected-access


@pytest.mark.parametrize("batch,kv,group,tokens,want", [
    (1, 16, 1, 320, 8),        # few CTAs: as many as a cluster merges
    (1, 8, 4, 4000, 16),       # 8 would leave most SMs empty
    (16, 8, 4, 2048, 3),       # 128 CTAs: one wave of three per SM
    (64, 32, 1, 2000, 1),      # more than a wave of CTAs as it is
    (1, 8, 4, 40, 1),          # half a tile for each of four warps
    (1, 8, 4, 16, 1),
    (4, 2, 9, 2048, 8),        # nine query heads are two CTAs
])
def test_tile_splits(batch, kv, group, tokens, want):
    assert decode_ops.tile_splits(batch, kv, group, tokens) == want


def test_tile_splits_stay_within_a_wave_and_a_cluster():
    for batch in (1, 2, 7, 16, 64, 300):
        for kv, group in ((32, 1), (8, 4), (2, 16), (1, 1)):
            for tokens in (1, 31, 64, 1000, 100000):
                s = decode_ops.tile_splits(batch, kv, group, tokens)
                ctas = batch * kv * ((group + 7) // 8)
                assert 1 <= s <= 16 and s * 32 <= max(tokens, 32)
                assert s == 1 or s * ctas <= 3 * 148
                assert s <= 8 or 16 * ctas <= 148
