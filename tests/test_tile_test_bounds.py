"""The division-free tile test against the four-candidate one, in numpy's
32-bit floats: where it answers, it answers the same. Conics from round to a
condition of 1e4, boxes from inside the ellipse to far outside, and many
whose nearest edge lies within a few ulps of the cutoff."""
from __future__ import annotations

import numpy as np
import pytest

F = np.float32
U = 2.0 ** -24


def fma(a, b, c):
    """Rounded once (up to the rare double rounding of the 64-bit sum)."""
    return (a.astype(np.float64) * b + c.astype(np.float64)).astype(F)


def four_candidates(a, b, c, lox, loy, hix, hiy, cutoff):
    inside = (lox <= 0) & (hix >= 0) & (loy <= 0) & (hiy >= 0)
    hit = inside & (cutoff >= 0)
    for x in (lox, hix):
        y = np.clip(-b * x / c, loy, hiy)
        hit |= ~inside & (a * x * x + F(2) * b * x * y + c * y * y <= cutoff)
    for y in (loy, hiy):
        x = np.clip(-b * y / a, lox, hix)
        hit |= ~inside & (a * x * x + F(2) * b * x * y + c * y * y <= cutoff)
    return hit


def division_free(a, b, c, lox, loy, hix, hiy, cutoff):
    """(certainly touched, certainly not)."""
    lmin = F(0.5) * (a + c) - np.sqrt(F(0.25) * (a - c) * (a - c) + b * b)
    with np.errstate(divide="ignore", invalid="ignore"):
        kappa = (a + np.abs(b) + c) / lmin
    usual = (lmin > 0) & (kappa <= 1e4)
    gate = np.where(usual, cutoff * (F(1) + F(64 * 5.9604645e-08) * np.where(usual, kappa, 0)), F(np.inf)).astype(F)
    sure = np.where(usual, cutoff - (gate - cutoff), F(-np.inf)).astype(F)
    inside = (lox <= 0) & (hix >= 0) & (loy <= 0) & (hiy >= 0)
    x = np.where(np.abs(hix) < np.abs(lox), hix, lox)
    y = np.where(np.abs(hiy) < np.abs(loy), hiy, loy)
    yx, xy = np.clip(x * (-b / c), loy, hiy), np.clip(y * (-b / a), lox, hix)
    q0 = fma(fma(F(2) * b, yx, a * x), x, c * yx * yx)
    q1 = fma(fma(F(2) * b, xy, c * y), y, a * xy * xy)
    yes = usual & (inside | (q0 <= sure) | (q1 <= sure))
    return yes, usual & ~yes & ~inside & (q0 > gate) & (q1 > gate)


@pytest.mark.parametrize("near", [False, True], ids=["anywhere", "at-the-cutoff"])
@pytest.mark.parametrize("most", [1.0, 2.0, 4.0], ids=["kappa-10", "kappa-100", "kappa-1e4"])
def test_the_division_free_test_agrees_where_it_answers(most, near):
    rng = np.random.default_rng(int(most) * 2 + near)
    n = 400_000
    angle, ratio = rng.uniform(0, np.pi, n), 10.0 ** rng.uniform(0, most, n) / 2.5
    small = 10.0 ** rng.uniform(-4, -0.5, n)
    large = small * np.maximum(ratio, 1.0)
    cs, sn = np.cos(angle), np.sin(angle)
    a, b, c = ((large * cs * cs + small * sn * sn).astype(F), ((large - small) * cs * sn).astype(F),
               (large * sn * sn + small * cs * cs).astype(F))
    cutoff = rng.uniform(0.01, 9.0, n).astype(F)
    reach = np.sqrt(cutoff * c / np.maximum(a.astype(np.float64) * c - b.astype(np.float64) ** 2, 1e-30))
    lox = (reach * rng.uniform(-1.5, 1.3, n)).astype(F)
    loy = (np.sqrt(cutoff / c) * rng.uniform(-3, 3, n)).astype(F)
    if near:   # the box's left edge at the ellipse's rightmost point, within a few ulps
        lox = (reach * (1.0 + rng.integers(-200, 200, n) * U)).astype(F)
        loy = (-b * lox / c - F(7.5)).astype(F)
    hix, hiy = lox + F(15), loy + F(15)
    want = four_candidates(a, b, c, lox, loy, hix, hiy, cutoff)
    yes, no = division_free(a, b, c, lox, loy, hix, hiy, cutoff)
    assert not (yes & ~want).any() and not (no & want).any()
    assert not (yes & no).any()
    if not near:
        assert yes.any() and no.any() and (yes | no).mean() > 0.9
