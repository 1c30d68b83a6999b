"""The planewise marches (divergence, corrections, diagnostics) run whole
columns in launches that fill the device and segments of planes in small
ones.  Both forms against the oracle, bit for bit: segments with a last
segment of 1, 2, 3 and 4 planes, and one box whose column tiles are enough for
whole columns (288 x 270 columns).

The implicit solves of a small set run on chip from right-hand sides
(k_implicit_cols), those of a set that fills the device as column sweeps; a
box's result is the same bits either way."""
import numpy as np
import pytest

from helpers import cfg_of, compare_fields, oracle_state, FIELDS
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


def _boxes(ctx, cfgs):
    out = []
    for q, cfg in enumerate(cfgs):
        s = oracle_state(cfg, seed=20 + q)
        box = ctx.add_box(cfg, s.g.xc)
        for f in FIELDS:
            box.upload(f, getattr(s, f))
        out.append(box)
    return out


@pytest.mark.parametrize("k1", [0, 2, 3, 5, 6, 7, 8])
def test_on_chip_and_column_solves_agree(ctx, k1):
    cfgs = [cfg_of(19, 30, 45, dt=5e-4, ylen=1.2, zlen=1.8), cfg_of(18, 16, 12, dt=5e-4, inslws=0),
            cfg_of(41, 64, 36, dt=5e-4, nsst=1)]
    filler = cfg_of(6, 200, 200, dt=1e-4)      # 157 tiles of 256 columns: the set fills the device
    alone = _boxes(ctx, cfgs)
    for b in alone:
        ctx.step([b], 3)
    batch = _boxes(ctx, cfgs + [filler])
    for b in batch:
        b.set_tuning(0, 0, k1)
    ctx.step(batch, 3)
    for a, b in zip(alone, batch):
        for f in FIELDS + ("rux", "ruy", "ruz", "rutemp", "wall"):
            assert np.array_equal(a.download(f), b.download(f)), f
    for b in alone + batch:
        ctx.remove_box(b)


@pytest.mark.parametrize("nxm,n,on_chip", [(24, 16, 1), (64, 192, 1), (400, 96, 1), (400, 128, 1), (150, 160, 1),
                                           (256, 160, 0), (160, 192, 0), (256, 192, 0), (404, 16, 0), (16, 196, 0)])
def test_on_chip_solves_where_their_waves_are_few(ctx, nxm, n, on_chip):
    """256x192^2 needs 16 waves of on-chip blocks (1 per SM) and took 5% longer
    per step than with the column kernels."""
    box = ctx.add_box(cfg_of(nxm, n, n, dt=1e-5), validate=False)
    f = ctx.forms([box])
    assert f["implicit_on_chip"] == on_chip and (f["k1_variant"] == 0) == bool(on_chip)
    ctx.remove_box(box)


@pytest.mark.parametrize("n,column,diag", [(128, 2, 2), (160, 2, 1), (196, 2, 1), (240, 1, 1), (288, 1, 1)])
def test_segments_where_they_gain(ctx, n, column, diag):
    """Plane segments (>= 2) only in launches that leave SMs idle: on 256^3 they took
    0.20 ms per step for the diagnostics against 0.11 in whole columns."""
    box = ctx.add_box(cfg_of(32, n, n, dt=1e-5), validate=False)
    f = ctx.forms([box])
    assert (min(f["column_segments"], 2), min(f["diag_segments"], 2)) == (column, diag)
    ctx.remove_box(box)


def test_forms_of_mixed_sets(ctx):
    """Column kernels take as long as the tallest box's columns, so a set of mostly low
    boxes keeps the forms that spread its work: segments at 208 tiles, on-chip
    solves at 142; a set of equal heights does not."""
    low = [ctx.add_box(cfg_of(32, 128, 128, dt=1e-5)) for _ in range(3)]
    tall = [ctx.add_box(cfg_of(96, 64, 64, dt=1e-5))]
    assert ctx.forms(low + tall)["column_segments"] > 1
    same = [ctx.add_box(cfg_of(32, 128, 128, dt=1e-5))]
    assert ctx.forms(low + same)["column_segments"] == 1
    high = [ctx.add_box(cfg_of(96, 16, 16, dt=1e-5)) for _ in range(14)]
    flat = [ctx.add_box(cfg_of(96, 128, 128, dt=1e-5)) for _ in range(2)]
    assert ctx.forms(low[:2] + high)["implicit_on_chip"] == 1
    assert ctx.forms(flat + high)["implicit_on_chip"] == 0
    for b in low + tall + same + high + flat:
        ctx.remove_box(b)


@pytest.mark.parametrize("nxm", [4, 9, 33, 400, 404])
def test_on_chip_solves_match_oracle(ctx, nxm):
    """nxm = 400 is near the tallest on-chip column, 404 is beyond it."""
    cfg = cfg_of(nxm, 10, 12, dt=5e-4, ray=1e6, ylen=0.9, zlen=1.1, istr3=0 if nxm > 300 else 7)
    s = oracle_state(cfg, seed=6)
    box = ctx.add_box(cfg, s.g.xc)
    for f in FIELDS:
        box.upload(f, getattr(s, f))
    O.run(s, 2, cfg.dt)
    ctx.step([box], 2)
    err = compare_fields(box, s)
    assert all(v <= 1e-11 for v in err.values()), err
    ctx.remove_box(box)


@pytest.mark.parametrize("nxm,nym,nzm", [(4, 8, 12), (8, 10, 9), (9, 10, 9), (16, 12, 10), (17, 12, 10),
                                         (33, 60, 30), (436, 8, 12), (440, 8, 12)])
def test_on_chip_pressure_solve_matches_oracle(ctx, nxm, nym, nzm):
    """The x-solve with the modes' columns on chip (up to nxm = 438), over mode
    counts that do not fill the last warp, and one box beyond it."""
    cfg = cfg_of(nxm, nym, nzm, ylen=1.3, zlen=0.9, istr3=0 if nxm > 300 else 7)
    s = oracle_state(cfg, seed=None)
    s.dph[...] = np.random.default_rng(nxm).standard_normal(s.dph.shape)
    box = ctx.add_box(cfg, s.g.xc, validate=False)
    box.upload("dph", s.dph)
    box.solve_pressure_correction()
    O.solve_pressure_correction(s)
    d, o = box.download("dph"), s.dph
    assert np.linalg.norm((d - d.mean()) - (o - o.mean())) <= 1e-11 * np.linalg.norm(o - o.mean())
    ctx.remove_box(box)


def test_pressure_solve_forms_agree(ctx):
    """The same bits on chip (one small box) and marched (in a large set)."""
    cfg = cfg_of(40, 64, 30, dt=5e-4, ylen=1.3, zlen=0.9)
    filler = [cfg_of(200, 320, 256, dt=1e-4)]     # two warps per SM: beyond four rounds
    a, b = _boxes(ctx, [cfg])[0], _boxes(ctx, [cfg] + filler)
    assert ctx.forms([a])["poisson_on_chip"] == 1 and ctx.forms(b)["poisson_on_chip"] == 0
    ctx.step([a], 2)
    ctx.step(b, 2)
    for f in FIELDS:
        assert np.array_equal(a.download(f), b[0].download(f)), f
    for x in [a] + b:
        ctx.remove_box(x)


def test_pressure_solve_chunks(ctx):
    """k_poisson_x marches chunks of 8 planes: one chunk (3 to 8 planes), and every
    remainder of two and three, give the bits of the solve on chip."""
    cfgs = [cfg_of(nxm, 10, 9 + nxm % 2, dt=5e-4, ylen=1.3, zlen=0.9) for nxm in range(3, 18)]
    filler = cfg_of(440, 8, 12, dt=1e-4, istr3=0)     # too tall for the solve on chip
    alone, batch = _boxes(ctx, cfgs), _boxes(ctx, cfgs + [filler])
    assert ctx.forms(batch)["poisson_on_chip"] == 0
    for b in alone:
        assert ctx.forms([b])["poisson_on_chip"] == 1
        ctx.step([b], 2)
    ctx.step(batch, 2)
    for a, b in zip(alone, batch):
        for f in FIELDS:
            assert np.array_equal(a.download(f), b.download(f)), (a.cfg.nxm, f)
    for b in alone + batch:
        ctx.remove_box(b)


def _check_divergence(box, s, al, dt):
    """CalcLocalDivergence of s.vy alone uses the coefficient al."""
    box.upload("vy", s.vy)
    for f in ("vx", "vz"):
        box.upload(f, np.zeros_like(s.vy))
    box.calc_local_divergence()
    t = O.State(**{**s.__dict__, "vx": np.zeros_like(s.vx), "vz": np.zeros_like(s.vz), "dph": s.dph.copy()})
    O.calc_local_divergence(t, al, dt)
    assert np.array_equal(box.download("dph"), t.dph)


@pytest.mark.parametrize("nsst,ns", [(3, 0), (3, 2), (1, 0)])
def test_routines_use_the_substep_prepared_last(ctx, nsst, ns):
    """A step prepares its substeps together; a routine called on its own uses
    the substep begun last, whether that was by the routine-level call, by a
    fused substep or (the last one) by a step."""
    cfg = cfg_of(9, 10, 12, dt=1e-3, nsst=nsst)
    s = oracle_state(cfg, seed=2)
    s.vy[:9] = np.random.default_rng(1).standard_normal((9, 10, 12))
    al = O.init_time_march_scheme(nsst)[2]
    box = _boxes(ctx, [cfg])[0]

    div = lambda a: _check_divergence(box, s, a, cfg.dt)

    ctx.step([box], 1)
    div(al[nsst - 1])
    box.time_marcher_begin_substep(ns)
    div(al[ns])
    ctx.substep([box], nsst - 1)
    div(al[nsst - 1])
    ctx.step([box], 1, graph=True)
    div(al[nsst - 1])
    ctx.remove_box(box)


def test_a_skipped_preparation_leaves_the_substep(ctx):
    """Boxes that have failed or are on hold are skipped by steps and by
    begin_substep alike, so the substep prepared before stays the one that the
    routines use."""
    cfg = cfg_of(9, 10, 12, dt=1e-3)
    s = oracle_state(cfg, seed=2)
    s.vy[:9] = np.random.default_rng(1).standard_normal((9, 10, 12))
    al = O.init_time_march_scheme(3)[2]
    box = _boxes(ctx, [cfg])[0]

    div = lambda a: _check_divergence(box, s, a, cfg.dt)

    box.time_marcher_begin_substep(1)
    box.upload("vy", 1e6 * s.vy)
    ctx.step([box], 1)                      # CFL too large: no substep is prepared
    assert box.scalars()["status"] == 165
    box.reset()
    div(al[1])
    for f in FIELDS:
        box.upload(f, getattr(oracle_state(cfg, seed=2), f))
    box.set_stop(1, 0.0, 0.0)
    ctx.step([box], 1)
    assert box.scalars()["status"] == 1     # on hold after its step
    box.time_marcher_begin_substep(0)
    box.resume()
    div(al[2])
    ctx.remove_box(box)


@pytest.mark.parametrize("n,shape", [(8, (64, 96, 96)), (12, (32, 128, 128)), (24, (64, 64, 64))])
def test_halves_take_the_whole_sets_forms(ctx, n, shape):
    """The halves of a split set run side by side: each takes the forms that the
    whole set would, and the x-solve that leaves shared memory to the other
    half.  A half's boxes stepped by themselves choose for themselves."""
    boxes = [ctx.add_box(cfg_of(*shape, dt=1e-5)) for _ in range(n)]
    whole = ctx.forms(boxes)
    for part in (1, 2):
        f = ctx.forms(boxes, part)
        assert f == {**whole, "poisson_on_chip": 0}
    own = ctx.forms(boxes[::2])
    assert own["poisson_on_chip"] == 1
    if n // 2 * shape[1] * shape[2] < 197 * 256:       # column tiles for two thirds of the resident blocks
        assert own["column_segments"] > whole["column_segments"]
    for b in boxes:
        ctx.remove_box(b)
