"""Sizes for which the feed-forward's activation goes into its product (148 SMs)."""
import pytest

from nanochat_b200.mixer_ops import gate_up_in_one


@pytest.mark.parametrize("rows,values,channels,inside", [
    (16384, 4096, 1536, True), (4096, 4096, 1536, True), (1024, 4096, 1536, True), (2048, 5504, 2048, True), (5521, 512, 512, True), (1407, 2752, 8192, False),
    (1537, 1376, 4096, False), (2561, 1024, 4096, False), (1091, 2048, 2048, False), (1308, 2132, 1024, False), (1568, 5504, 8192, False),
    (1501, 3453, 4096, True), (1025, 2056, 72, True), (1023, 8192, 1536, False), (1024, 2047, 64, False), (0, 4096, 1536, False), (4096, 0, 1536, False)])
def test_sizes(rows, values, channels, inside):
    assert gate_up_in_one(rows, values, channels, 148) == inside
