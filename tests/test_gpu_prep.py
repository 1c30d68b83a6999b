"""The preparation of the substeps (LU of the x-systems without pivoting).

A box whose systems need a row exchange gets status -2 before any substep.  Its
three substeps are prepared by blocks of one launch, which read and write
that status: each block decides once, so that none leaves threads behind, and a
failing box touches neither its own fields nor the other boxes of the set."""
import numpy as np
import pytest

from afid_b200.ic import initial_fields
from helpers import cfg_of, FIELDS

pytestmark = pytest.mark.gpu


def _jump_grid(nxm):
    """Node positions whose spacing grows twelvefold half way up."""
    h = np.where(np.arange(nxm) < nxm // 2, 1.0, 12.0)
    return np.concatenate([[0.0], np.cumsum(h)]) / h.sum()


def _needs_exchange(xc, beta_al):
    """dgttrf's test on the rows 1 + beta al (am + ap), -beta al am, -beta al ap of
    vx (SolveImpEqnUpdate_X.F90:25-44), scaled to a unit diagonal."""
    nx = len(xc)
    dl, du = np.zeros(nx), np.zeros(nx)
    for k in range(1, nx - 1):
        c = 2.0 / (xc[k + 1] - xc[k - 1])
        am, ap = c / (xc[k] - xc[k - 1]), c / (xc[k + 1] - xc[k])
        dl[k], du[k] = (-beta_al * a / (1.0 + beta_al * (am + ap)) for a in (am, ap))
    d, out = 1.0, False
    for k in range(nx - 1):
        out |= abs(d) < abs(dl[k + 1])
        d = 1.0 - dl[k + 1] / d * du[k]
    return out


def _box(ctx, cfg, seed, xc=None):
    box = ctx.add_box(cfg, xc)
    for f, v in initial_fields(cfg, box.xc, seed).items():
        box.upload(f, v)
    return box


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nsst,dt,fails", [(3, 50.0, (True, True, True)), (3, 1.0, (True, False, False)), (1, 1.0, (True,))])
def test_row_exchange_fails_the_box_before_its_substeps(ctx, nsst, dt, fails, graph):
    xc = _jump_grid(24)
    bad_cfg = cfg_of(24, 16, 12, ray=1e5, dt=dt, nsst=nsst)
    good_cfg = cfg_of(19, 16, 12, dt=5e-4)
    ren = np.sqrt(bad_cfg.ray / bad_cfg.pra)
    als = (8 / 15, 2 / 15, 1 / 3) if nsst == 3 else (1.0,)
    assert tuple(_needs_exchange(xc, 0.5 * dt / ren * al) for al in als) == fails
    assert not _needs_exchange(xc, 0.5 * 1e-3 / ren)
    alone = _box(ctx, good_cfg, 3)
    ctx.step([alone], 3)
    bad = [_box(ctx, bad_cfg, q, xc) for q in range(6)]
    good = _box(ctx, good_cfg, 3)
    before = [{f: b.download(f) for f in FIELDS} for b in bad]
    ctx.step(bad[:3] + [good] + bad[3:], 3, graph=graph)
    for b, was in zip(bad, before):
        sc = b.scalars()
        assert sc["status"] == -2 and sc["ntime"] == 0
        for f in FIELDS:
            assert np.array_equal(b.download(f), was[f]), f
    assert good.scalars()["status"] == 0
    for f in FIELDS:
        assert np.array_equal(good.download(f), alone.download(f)), f
    # a dt the grid can take: the box goes on
    bad[0].reset(1e-3)
    ctx.step([bad[0]], 2)
    sc = bad[0].scalars()
    assert sc["status"] == 0 and sc["ntime"] == 2
    for b in bad + [good, alone]:
        ctx.remove_box(b)
