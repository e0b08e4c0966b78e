"""SVG numbers and colours at the edges of their readers' fast forms: 18 digits (more are left to
strtoll, which saturates), powers of ten a double holds exactly (up to 22), six and three hex digits,
rgb() with plain numbers of up to nine digits; against the same arithmetic written here."""
import numpy as np
import pytest

import pfcuda

LONG = "123456789012345678901234"
NUMBERS = ["7", "-0.5", "+.25", "1e2", "35.79", "5.41e+01", "3.57e-01", "2e22", "2e23", "1.5e-22", "4e-23", "1e",
           *(LONG[:n] for n in (17, 18, 19, 20, 24)), *("0." + LONG[:n] for n in (17, 18, 19, 21)),
           *("0." + "0" * n + "7" for n in (15, 17, 18, 21, 22))]
COLORS = {"#1a2B3c": (0x1a, 0x2b, 0x3c), "#aBc": (0xaa, 0xbb, 0xcc), "#abcd": (0xaa, 0xbb, 0xcc),
          "#abcde": (0xab, 0xcd, 0x0e), "#abcdef12": (0xab, 0xcd, 0xef), "#ab": (128, 128, 128), "#": (128, 128, 128),
          "#1 2 3": (1, 2, 3), "rgb(1,2,3)": (1, 2, 3), "rgb( 1, 22,  255)": (1, 22, 255), "rgb(300,2,3)": (255, 2, 3),
          "rgb(1, 2, 3": (1, 2, 3), "rgb(123456789,2,3)": (255, 2, 3), "rgb(0000000012,2,3)": (12, 2, 3),
          "rgb(1 ,2,3)": (128, 128, 128), "rgb(50%, 0%, 100%)": (128, 0, 255), "blue": (0, 0, 255)}


def expected(s):
    sign, s = (-1.0 if s[0] == "-" else 1.0), s.lstrip("+-")
    mant, _, exp = s.partition("e")
    i, _, f = mant.partition(".")
    v = float(min(int(i), 2**63 - 1)) if i else 0.0
    if f:
        v += float(min(int(f), 2**63 - 1)) / 10.0 ** len(f)
    return np.float32((v * 10.0 ** int(exp) if exp else v) * sign)


@pytest.mark.parametrize("s", NUMBERS)
def test_numbers(s):
    # a view box of the canvas size: no scaling
    doc = f'<svg width="100" height="100" viewBox="0 0 100 100"><path d="M{s} 0 L{s} 90 95 95z" fill="red"/></svg>'
    assert pfcuda.parse_svg(doc).points[0, 0] == expected(s)


@pytest.mark.parametrize("s", COLORS)
def test_colors(s):
    sc = pfcuda.parse_svg(f'<svg><path d="M0 0L9 0 9 9z" fill="{s}"/></svg>')
    r, g, b = COLORS[s]
    assert int(sc.color[0]) == r | g << 8 | b << 16 | 0xff000000
