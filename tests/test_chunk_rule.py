"""The rule for steps without a barrier between them (runtime.chunks_pay, the library's): networks measured faster in
chunks take them, networks measured slower do not, at its lines and between them."""

import re
from pathlib import Path

import pytest

from naer2_b200 import runtime

SMS2 = 296  # two blocks on each of 148 SMs


def _pays(sizes, row, k):
    return runtime.chunks_pay(sizes, row * sum(sizes), k, SMS2)


@pytest.mark.parametrize("sizes, row, k, want", [
    ([800, 200], 100, 15, True), ([10000, 2500], 1250, 15, True), ([10000, 2500], 1250, 2, False),
    ([16000, 4000], 390 * 3, 3, True), ([16000, 4000], 390 * 3 + 1, 3, False),
    ([37888], 780, 2, True), ([37889], 780, 2, False), ([37889], 256, 2, True), ([37889], 257, 2, False),
    ([75776], 1300, 15, True), ([75776], 1301, 15, False), ([75777], 640, 15, True), ([75777], 641, 32, False),
    ([75777], 100, 2, True), ([75777], 101, 2, False), ([4823] * 8, 1935, 15, False), ([8592] * 10, 1000, 15, False),
    ([100], 0, 2, True), ([0, 50], 5, 2, True)])
def test_lines(sizes, row, k, want):
    assert _pays(sizes, row, k) is want


def test_the_library_has_the_same_lines():
    text = (Path(__file__).resolve().parents[1] / "naer2_b200" / "csrc" / "naer2b.cu").read_text()
    body = text[text.index("bool chunks_pay("):]
    body = body[:body.index("\n}\n")]
    assert re.findall(r"\d+ \* k(?:, \d+)?", body) == ["390 * k", "128 * k, 1300", "50 * k, 640"]
