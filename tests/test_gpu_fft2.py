"""The two-pass transforms (lines of N = r1 r2 points, both radices at most 32)
through the pressure solve, against the oracle: every radix in either pass, tiles
with lines beyond the box (odd row counts, ky counts that do not fill a tile),
and the sizes next to them that the tile kernels keep (a factor of 7, more
than 1024 points)."""
import numpy as np
import pytest

from helpers import cfg_of, oracle_state, rel_l2
from oracle import afid_oracle as O

pytestmark = pytest.mark.gpu

Y = [4, 6, 10, 18, 32, 40, 48, 80, 90, 144, 150, 256, 270, 324, 400, 480, 600, 750, 960, 1024, 14, 56, 1152]
Z = [4, 9, 8, 15, 25, 27, 12, 20, 60, 81, 135, 180, 225, 243, 375, 432, 486, 625, 729, 810, 1024, 21, 1280]


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
