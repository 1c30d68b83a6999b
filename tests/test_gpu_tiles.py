"""The tile kernels of the transforms (lines with a factor of 7, of more than 1024
points or without two radices up to 32): z tiles whose copies need rows beyond
whole TMA boxes, and tiles whose size is no multiple of 128 bytes in blocks that
use both shared-memory slots."""
import numpy as np
import pytest

from helpers import cfg_of, oracle_state, rel_l2, FIELDS
from oracle import afid_oracle as O

pytestmark = pytest.mark.gpu


def _solve(ctx, cfg, fy=0, fz=0):
    s = oracle_state(cfg, seed=None)
    s.dph[...] = np.random.default_rng(cfg.nym * 2000 + cfg.nzm).standard_normal(s.dph.shape)
    box = ctx.add_box(cfg, s.g.xc, validate=False)
    box.set_tuning(fy, fz, 0)
    box.upload("dph", s.dph)
    box.solve_pressure_correction()
    got = box.download("dph")
    status = box.scalars()["status"]
    ctx.remove_box(box)
    assert status == 0
    return got, s


# copies of a z tile: TMA boxes of whole 128-byte multiples and 1 to 11 single rows (350
# at 4 ky, 441, 525, 735, 1125, 1215, 1458, 2187), or boxes of a height below the
# largest divisor (972, 1000, 2000)
@pytest.mark.parametrize("nym,nzm", [(6, 350), (10, 441), (10, 525), (18, 735), (10, 972), (10, 1000), (10, 1125),
                                     (10, 1215), (10, 1458), (10, 2000), (10, 2187), (972, 9), (1000, 9), (98, 98)])
def test_z_tile_copies(ctx, nym, nzm):
    # tolerance as test_gpu_fft2's short uniform grids
    got, s = _solve(ctx, cfg_of(6, nym, nzm, ylen=1.3, zlen=0.9, istr3=0))
    O.solve_pressure_correction(s, vectorised=True)
    assert rel_l2(got, s.dph, remove_mean=True) <= 1e-12


# more tiles than resident blocks (at most 296), so that blocks fill their second slot:
# one tile of 4 ky a plane (21 and 35 points: 84 and 140 values, 16 bytes x 4 off 128),
# one ky a tile (98 points)
@pytest.mark.parametrize("nxm,nym,nzm,fz", [(620, 4, 21, 0), (640, 6, 35, 0), (20, 64, 98, 1), (24, 64, 63, 2)])
def test_z_tiles_in_both_slots(ctx, nxm, nym, nzm, fz):
    # tolerance as the tall uniform grids of test_gpu_segments
    got, s = _solve(ctx, cfg_of(nxm, nym, nzm, ylen=1.3, zlen=0.9, istr3=0), 0, fz)
    O.solve_pressure_correction(s)
    assert rel_l2(got, s.dph, remove_mean=True) <= 1e-11


@pytest.mark.parametrize("fy,fz", [(0, 0), (1, 1), (4, 2)])
def test_tile_boxes_in_a_set(ctx, fy, fz):
    """Boxes of different tile lines in one launch of each transform come out
    as each does alone with the built-in lines per tile."""
    cfgs = [cfg_of(12, 56, 42, dt=2e-4, ylen=1.2), cfg_of(5, 14, 441, dt=1e-4), cfg_of(9, 98, 21, dt=2e-4),
            cfg_of(4, 1152, 28, dt=1e-5), cfg_of(7, 10, 972, dt=1e-5)]

    def boxes():
        out = []
        for q, cfg in enumerate(cfgs):
            s = oracle_state(cfg, seed=q)
            out.append(ctx.add_box(cfg, s.g.xc, validate=False))
            for f in FIELDS:
                out[-1].upload(f, getattr(s, f))
        return out

    alone, batch = boxes(), boxes()
    for b in alone:
        ctx.step([b], 2)
    for b in batch:
        b.set_tuning(fy if b.cfg.nym * fy <= 3584 else 0, fz, 0)
    ctx.step(batch, 2)
    for a, b in zip(alone, batch):
        assert b.scalars()["status"] == 0
        for f in FIELDS:
            assert np.array_equal(a.download(f), b.download(f)), f
    for b in alone + batch:
        ctx.remove_box(b)
