"""CPU: the error bound of the SPR engine's eigen products in float pairs
(csrc/spr.cu, eigen_pair), which decides where FP64 forms them again: numpy's
float32 does the same operations, and exact fractions say how far off they are,
on random terms and on terms that a search found to be the worst."""
from __future__ import annotations

import re
from fractions import Fraction
from pathlib import Path

import numpy as np

f = np.float32
SRC = Path(__file__).resolve().parent.parent / "phylocaml_gb300" / "csrc" / "spr.cu"

# coefficients (double), values' high and low floats
WORST = [
    ([-1.4511340092263023, -1.3929032605367426, -0.27859713038002154, -0.5221876177958176],
     [0.7066000699996948, 0.730354368686676, 0.9227317571640015, 0.3345324695110321],
     [2.905603402325596e-08, 1.6302974970017203e-08, 2.1541360695209733e-08, 5.851715223492704e-10]),
    ([-2.0431550640886043, -1.9851134406660031, -0.543252494826906, -0.1825664151029516],
     [0.5008680820465088, 0.5511341094970703, 0.5798100233078003, 0.6501164436340332],
     [2.9263667045142938e-08, -3.020436167844309e-08, 2.149335642798178e-08, -3.768627365730026e-08]),
    ([1.7996574371418623, 1.8621730260340907, 0.4490508330983204, 0.21178140856186495],
     [0.5922005772590637, 0.5515062212944031, 0.5647966265678406, 0.4603835344314575],
     [3.001167314664599e-08, 3.156521088953923e-08, 3.097711598343267e-08, 1.8799825696191874e-08]),
]


def rounded(x: Fraction) -> np.float32:
    """x to the nearest float, ties to even."""
    y = f(float(x))
    near = sorted({y, np.nextafter(y, f(-np.inf)), np.nextafter(y, f(np.inf))},
                  key=lambda v: (abs(Fraction(float(v)) - x), int(v.view(np.uint32)) & 1))
    return near[0]


def fma(a, b, c):
    return rounded(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


def two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def relative_error(c, xh, xl) -> Fraction:
    exact = mag = Fraction(0)
    s = lo = f(0)
    for j in range(4):
        h, l = two_sum(f(xh[j]), f(xl[j]))
        ch = f(c[j])
        cl = f(c[j] - float(ch))
        p = ch * h
        e = fma(cl, h, fma(ch, l, fma(ch, h, -p)))
        if j == 0:
            s, lo = p, e
        else:
            s, te = two_sum(s, p)
            lo = lo + (te + e)
        exact += Fraction(c[j]) * (Fraction(float(h)) + Fraction(float(l)))
        mag += abs(Fraction(float(p)))
    return abs(Fraction(float(s)) + Fraction(float(lo)) - exact) / mag


def test_sums_stay_within_the_bound():
    const = re.search(r"constexpr float EIGEN_ERR = 0x1p-(\d+)f", SRC.read_text())
    bound = Fraction(1, 2 ** int(const.group(1)))
    # the product of two sums adds 3 u^2, the rounding test and FP64 2 u^2
    room = bound - 5 * Fraction(1, 2 ** 48)
    worst = max(relative_error(*w) for w in WORST)
    assert worst > Fraction(1, 2 ** 45)          # what a bound of 2^-45 would miss
    rng = np.random.default_rng(4)
    for _ in range(400):
        xh = rng.uniform(0.1, 1.0, 4).astype(f)
        c = rng.uniform(0.1, 2.0, 4) * rng.choice([-1.0, 1.0], 4)
        worst = max(worst, relative_error(list(map(float, c)), xh, xh * f(2.0 ** -25) * rng.uniform(-1, 1, 4).astype(f)))
    assert worst <= room
