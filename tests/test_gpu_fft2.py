"""The two-pass transforms (lines of N = r1 r2 points, both radices at most 32)
through the pressure solve, against the oracle: in y and in z every radix in
either pass, tiles with lines beyond the box (odd row counts, ky counts that do not
fill a tile), and lengths that the tile kernels keep (a factor of 7, more than
1024 points)."""
import ctypes as C

import numpy as np
import pytest

from afid_b200 import _lib
from helpers import cfg_of, oracle_state, rel_l2
from oracle import afid_oracle as O

RADICES = [2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 27, 30, 32]
Y = [4, 6, 10, 12, 18, 20, 30, 32, 40, 48, 72, 80, 90, 120, 144, 150, 180, 240, 256, 270, 288, 324, 360, 400, 480,
     486, 600, 750, 864, 900, 960, 1024, 14, 56, 1152]
Z = [4, 9, 8, 15, 16, 25, 27, 12, 20, 36, 60, 64, 81, 100, 135, 144, 180, 225, 243, 256, 324, 375, 400, 432, 486,
     576, 625, 729, 768, 810, 900, 1024, 21, 1280]


@pytest.mark.parametrize("lines", [Y, Z])
def test_every_radix_in_either_pass(lines):
    """The plan takes n = r1 r2 with the smallest larger radix r2."""
    seen = set()
    for n in lines:
        plan = next(((n // r, r) for r in RADICES if n % r == 0 and n // r in RADICES and n // r <= r), None)
        assert (plan is None) == (_lib_tile(n) == 1), n
        seen |= {(q, r) for q, r in enumerate(plan or ())}
    assert seen == {(q, r) for q in (0, 1) for r in RADICES}


def _lib_tile(n):
    t = _lib.TileShape()
    _lib.check(_lib.lib().afid_fft_tile_shape(10, n, 0, 0, C.byref(t)))
    return t.z_tile


@pytest.mark.gpu
@pytest.mark.parametrize("nym,nzm", [(y, 9) for y in Y] + [(10, z) for z in Z] + [(150, 135), (64, 96), (32, 45)])
def test_pressure_solve_line_lengths(ctx, nym, nzm):
    # white noise on a uniform grid of 6 planes: the solve amplifies rounding
    # by the ratio of its largest to its smallest eigenvalue, (n/pi)^2 4 at
    # the longest line, of which the norm sees a part; 1e-12 as the other
    # short-grid solves of the tests
    cfg = cfg_of(6, nym, nzm, ylen=1.3, zlen=0.9, istr3=0)
    s = oracle_state(cfg, seed=None)
    s.dph[...] = np.random.default_rng(nym * 2000 + nzm).standard_normal(s.dph.shape)
    box = ctx.add_box(cfg, s.g.xc, validate=False)
    box.upload("dph", s.dph)
    box.solve_pressure_correction()
    O.solve_pressure_correction(s, vectorised=True)
    assert rel_l2(box.download("dph"), s.dph, remove_mean=True) <= 1e-12
    ctx.remove_box(box)
