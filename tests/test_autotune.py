"""Autotuner logic that needs no GPU: FFT plans and candidate ranges."""
import pytest

from afid_b200 import BouIn
from afid_b200.autotune import candidates, fft_plan, TuneCache


@pytest.mark.parametrize("n,plan", [(768, [16, 16, 3]), (1280, [16, 16, 5]), (384, [16, 8, 3]),
                                    (96, [16, 2, 3]), (48, [16, 3]), (32, [16, 2]), (64, [16, 4]),
                                    (128, [16, 8]), (16, [16]), (12, [4, 3]), (14, [2, 7])])
def test_fft_plan(n, plan):
    assert fft_plan(n) == plan
    prod = 1
    for r in plan:
        prod *= r
    assert prod == n


def test_fft_plan_rejects_large_primes():
    with pytest.raises(ValueError):
        fft_plan(22)


@pytest.mark.parametrize("nyz", [32, 48, 96, 128, 384, 768, 1280])
def test_candidates_fit_shared_memory(nyz):
    c = candidates(BouIn(nxm=64, nym=nyz, nzm=nyz))
    for v in c["fft_y_lines"]:
        assert (4 * v * (nyz // 2 + 1) + nyz) * 16 <= 200 * 1024 and v * nyz <= 14 * 256
        assert v & (v - 1) == 0
    for v in c["fft_z_lines"]:
        assert (2 * v * nyz + nyz) * 16 <= 200 * 1024 and v * nyz <= 14 * 256
        assert v & (v - 1) == 0
    assert c["fft_y_lines"] and c["fft_z_lines"]
    assert c["k1_minb"] == [2, 3, 4, 5, 6, 7, 8]


def test_cache_roundtrip(tmp_path):
    path = str(tmp_path / "t.json")
    c = TuneCache(path)
    cfg = BouIn(nxm=32, nym=48, nzm=48)
    assert c.get(cfg) is None
    c.put(cfg, {"fft_y_lines": 4, "fft_z_lines": 8, "k1_minb": 2})
    c.save()
    assert TuneCache(path).get(cfg)["fft_z_lines"] == 8


class FakeBox:
    def __init__(self, cfg):
        self.cfg, self.xc, self.shapes = cfg, [0.0] * cfg.nx, [(0, 0, 0)]

    def upload(self, name, a):
        pass

    def set_tuning(self, fy, fz, k1):
        self.shapes.append((fy, fz, k1))


class FakeCtx:
    """Kernel times that fall with every line count and variant, and the forms
    that a set's launches take."""

    def __init__(self, **acts):
        self.acts = {"y_tile": 0, "z_tile": 0, "k1_variant": 0, **acts}
        self.profiles = 0

    def add_box(self, cfg):
        self.box = FakeBox(cfg)
        return self.box

    def remove_box(self, box):
        pass

    def step(self, boxes, n):
        pass

    def forms(self, boxes):
        return self.acts

    def step_profiled(self, boxes, steps):
        self.profiles += 1
        fy, fz, k1 = boxes[0].shapes[-1]
        y, z, k = 100.0 - fy, 100.0 - fz, 100.0 - k1
        return {"fft_y_fwd": (y, 1), "fft_y_inv": (y, 1), "fft_z_fwd": (z, 1), "fft_z_inv": (z, 1),
                "explicit_fwd": (k, 1)}


@pytest.mark.parametrize("acts", [{}, {"y_tile": 1}, {"z_tile": 1}, {"k1_variant": 4},
                                  {"y_tile": 1, "z_tile": 1, "k1_variant": 4}])
def test_only_shapes_that_act_are_tuned(monkeypatch, acts):
    from afid_b200 import autotune
    monkeypatch.setattr(autotune, "initial_fields", lambda *a, **k: {})
    cfg = BouIn(nxm=8, nym=56, nzm=42)
    cand = candidates(cfg)
    want = {"fft_y_lines": max(cand["fft_y_lines"]) if acts.get("y_tile") else 0,
            "fft_z_lines": max(cand["fft_z_lines"]) if acts.get("z_tile") else 0,
            "k1_minb": 8 if acts.get("k1_variant") else 0}
    for choose in (lambda c: autotune.tune_class(c, cfg), lambda c: autotune.tune_batch(c, [FakeBox(cfg)])):
        ctx = FakeCtx(**acts)
        got = choose(ctx)
        assert {k: got[k] for k in want} == want
        assert bool(ctx.profiles) == bool(acts)
        assert len(got["ms_per_step"]) == ctx.profiles
