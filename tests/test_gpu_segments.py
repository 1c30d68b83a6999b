"""The planewise marches (divergence, corrections, diagnostics) run whole
columns in launches that fill the device and segments of planes in small
ones.  Both forms against the oracle, bit for bit: segments with a last
segment of 1, 2, 3 and 4 planes, and one box whose column tiles are enough for
whole columns (288 x 270 columns)."""
import numpy as np
import pytest

from helpers import cfg_of, oracle_state
from oracle import afid_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxm,nym,nzm", [(5, 8, 12), (18, 30, 45), (19, 16, 12), (24, 16, 12), (10, 288, 270)])
def test_planewise_marches_match_oracle(ctx, nxm, nym, nzm):
    cfg = cfg_of(nxm, nym, nzm, dt=1e-3, ylen=1.2, zlen=0.9)
    s = oracle_state(cfg, seed=4)
    rng = np.random.default_rng(nxm)
    for f in ("vx", "vy", "vz", "pr"):
        getattr(s, f)[:nxm] = rng.standard_normal((nxm, nym, nzm))
    s.vx[0] = 0.0
    al = O.init_time_march_scheme(3)[2][1]
    box = ctx.add_box(cfg, s.g.xc)
    for f in ("vx", "vy", "vz", "temp", "pr"):
        box.upload(f, getattr(s, f))
    box.time_marcher_begin_substep(1)
    assert box.calc_max_cfl() == pytest.approx(O.calc_max_cfl(s), rel=1e-15)
    assert box.check_divergence() == pytest.approx(O.check_divergence(s), rel=1e-13)
    box.calc_local_divergence()
    O.calc_local_divergence(s, al, cfg.dt)
    assert np.array_equal(box.download("dph"), s.dph)
    box.correct_velocity()
    O.correct_velocity(s, al, cfg.dt)
    box.correct_pressure()
    O.correct_pressure(s, al, cfg.dt / s.p.ren * 0.5)
    for f in ("vx", "vy", "vz", "pr"):
        assert np.array_equal(box.download(f)[:nxm], getattr(s, f)[:nxm]), f
    ctx.remove_box(box)
