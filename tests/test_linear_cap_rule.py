"""Sizes for which the soft cap goes into the product (148 SMs)."""
import pytest

from nanochat_b200.mixer_ops import cap_in_product


@pytest.mark.parametrize("rows,words,channels,inside", [
    (16384, 32768, 1536, True), (6007, 32768, 2048, True), (1000, 32768, 1536, True), (256, 32768, 1536, True), (2048, 4096, 1024, True),
    (1, 32768, 1536, False), (64, 32768, 2048, False), (128, 32768, 1536, False), (257, 32768, 1536, False), (256, 16384, 2048, False),
    (1025, 16384, 1536, False), (16384, 32768, 1016, False), (16384, 64, 1536, False), (0, 32768, 1536, False), (300, 0, 1536, False)])
def test_sizes(rows, words, channels, inside):
    assert cap_in_product(rows, words, channels, 148) == inside
