"""The division-free tile test against the four-candidate one: where it
answers, it answers the same. Once in numpy's 32-bit floats (the bound as
derived), once with the projection's own functions (the header that the
kernels include, compiled here for the host). Conics from round to a
condition of 1e4, boxes from inside the ellipse to far outside, and many
whose nearest edge lies within a few ulps of the cutoff."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from lucabrtrender_b200 import build

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


def draw_boxes(most, near):
    """Conics, cutoffs, and boxes of 15 x 15 pixels from the centre."""
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
    return a, b, c, cutoff, lox, loy


@pytest.mark.parametrize("near", [False, True], ids=["anywhere", "at-the-cutoff"])
@pytest.mark.parametrize("most", [1.0, 2.0, 4.0], ids=["kappa-10", "kappa-100", "kappa-1e4"])
def test_the_division_free_test_agrees_where_it_answers(most, near):
    a, b, c, cutoff, lox, loy = draw_boxes(most, near)
    hix, hiy = lox + F(15), loy + F(15)
    want = four_candidates(a, b, c, lox, loy, hix, hiy, cutoff)
    yes, no = division_free(a, b, c, lox, loy, hix, hiy, cutoff)
    assert not (yes & ~want).any() and not (no & want).any()
    assert not (yes & no).any()
    if not near:
        assert yes.any() and no.any() and (yes | no).mean() > 0.9


HOST_TEST = r"""
#include "raster_common.cuh"
extern "C" void tile_tests(unsigned n, const float* conic, const float* cutoff, const float* centre, unsigned char* touched,
                           unsigned char* touch) {
    for (unsigned i = 0; i < n; ++i) {
        const float a = conic[3 * i], b = conic[3 * i + 1], c = conic[3 * i + 2];
        const lrt::TileTest t = lrt::tile_test(a, b, c, cutoff[i]);
        touched[i] = lrt::tile_touched(64, 64, centre[2 * i], centre[2 * i + 1], a, b, c, cutoff[i], 1, 1);
        touch[i] = (unsigned char)lrt::tile_touch(64, 64, centre[2 * i], centre[2 * i + 1], a, b, c, t, 1, 1);
    }
}
"""


@pytest.fixture(scope="module")
def host_tests(tmp_path_factory):
    folder = tmp_path_factory.mktemp("tile_tests")
    source, library = folder / "tile_tests.cu", folder / "tile_tests.so"
    source.write_text(HOST_TEST)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-fmad=false", "-I", str(build.CSRC), "-shared",
                    "-o", str(library), str(source)], check=True)
    return C.CDLL(str(library)).tile_tests


@pytest.mark.parametrize("near", [False, True], ids=["anywhere", "at-the-cutoff"])
@pytest.mark.parametrize("most", [1.0, 2.0, 4.0], ids=["kappa-10", "kappa-100", "kappa-1e4"])
def test_the_projections_own_test_agrees_where_it_answers(host_tests, most, near):
    """Of a 64 x 64 frame, tile (1, 1): its pixel centres are 16.5 .. 31.5."""
    a, b, c, cutoff, lox, loy = draw_boxes(most, near)
    n = len(a)
    conic = np.ascontiguousarray(np.stack([a, b, c], 1))
    centre = np.ascontiguousarray(np.stack([F(16.5) - lox, F(16.5) - loy], 1))
    touched, touch = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
    host_tests(n, *(v.ctypes.data_as(C.c_void_p) for v in (conic, cutoff, centre, touched, touch)))
    no, yes = touch == 0, touch == 1
    assert not (yes & (touched == 0)).any() and not (no & (touched == 1)).any()
    if not near:
        assert yes.any() and no.any() and (yes | no).mean() > 0.9
