"""Scratch of prompt attention, which the host sizes (no GPU): only blocks whose keys are divided among CTAs leave anything."""
import pytest

from axono_b200 import _capi


def scratch(n, hq, hkv, d, skv, causal, dtype):
    return _capi.lib().axb200_sdpa_scratch_bytes(n, hq, hkv, d, skv, causal, dtype)


@pytest.mark.parametrize("tokens,heads,causal,most", [
    (8192, 16, 1, 0),              # no block divided
    (57344, 16, 1, 64 << 20), (57344, 16, 0, 64 << 20), (100000, 16, 0, 64 << 20), (100000, 64, 0, 64 << 20)])
def test_only_divided_blocks_take_scratch(tokens, heads, causal, most):
    assert scratch(tokens, heads, heads // 2, 128, tokens, causal, _capi.FLOAT16) <= most


@pytest.mark.parametrize("tokens,heads,d,causal,divided", [
    (1100, 1, 64, 1, True), (1100, 2, 64, 1, True), (1100, 4, 64, 0, True), (1100, 8, 64, 1, True), (1100, 2, 128, 1, True),
    (1100, 4, 128, 0, False), (1100, 8, 128, 1, False), (1100, 16, 64, 0, False), (2048, 16, 128, 1, False),
    (40000, 1, 128, 0, True), (57600, 1, 64, 0, True), (77000, 1, 128, 0, True)])  # more than 448 blocks or units
def test_prompts_are_divided_where_that_was_measured_faster(tokens, heads, d, causal, divided):
    assert (scratch(tokens, heads, heads, d, tokens, causal, _capi.FLOAT16) > 0) == divided


@pytest.mark.parametrize("dtype", [_capi.FLOAT16, _capi.FLOAT32])
def test_scratch_is_bounded(dtype):
    """2 GB at most; fp32 that would want more (its tiles of K and V) asks for none."""
    asked = set()
    for tokens in (16, 100, 257, 2000, 5000, 20000, 57344, 100000, 200000, 500000, 4000000):
        for hq, hkv in ((1, 1), (2, 2), (16, 8), (64, 8), (128, 128)):
            for d in (8, 64, 128):
                for causal in (0, 1):
                    need = scratch(tokens, hq, hkv, d, tokens, causal, dtype)
                    assert 0 <= need <= 2 << 30
                    asked.add(need > 0)
    assert asked == {True, False}
    assert scratch(2000000, 16, 8, 128, 2000000, 1, _capi.FLOAT32) == 0
    assert scratch(4096, 2, 2, 128, 4096, 1, dtype) > 0


def test_keys_that_no_row_sees_take_none():
    """Under a causal mask row t sees key t at most: a few rows over a long cache are the small problem they are alone."""
    assert scratch(16, 16, 8, 128, 8192, 1, _capi.FLOAT32) == 0 < scratch(16, 16, 8, 128, 8192, 0, _capi.FLOAT32)
    assert scratch(300, 16, 8, 128, 50000, 1, _capi.FLOAT32) == scratch(300, 16, 8, 128, 300, 1, _capi.FLOAT32)


@pytest.mark.parametrize("bad", [(0, 2, 2, 64, 64), (64, 0, 2, 64, 64), (64, 2, 0, 64, 64), (64, 3, 2, 64, 64), (64, 2, 2, 0, 64),
                                 (64, 2, 2, 64, 0), (64, 2, 2, 64, 2 ** 31)])
def test_calls_that_are_refused_want_none(bad):
    for dtype in (_capi.FLOAT16, _capi.FLOAT32):
        assert scratch(*bad, 1, dtype) == 0
