"""Performance cases: the work a program has this library do.

Kinds of pass, each through the entry points of ``afid_b200`` (the C-ABI of
``include/afid_gpu.h``):

* ``advance``: resident boxes advance ``steps`` time steps to their next
  output time; the five fields and every box's record are read back into
  pinned host memory, as a run writes its output;
* ``jobs``: solve jobs as a serving loop runs them: the initial fields come
  from pinned host memory, the boxes are reset, advance, and are read back;
* ``routines``: one time step through the routine-level entry points (the
  reference's subroutines one for one), then the fields;
* ``pressure``: SolvePressureCorrection on a device array the caller owns;
* ``output``: the output-time diagnostics of a resident box.

Sizes are those of the repository's configurations, benchmark and tests, or
lie between them.  ``exact`` restates the passes in plain torch, FP64.
"""
from __future__ import annotations

import ctypes as C
import math
import sys

import numpy as np
import torch

from afid_b200 import BouIn, Context, _lib, make_grid
from afid_b200.ensemble import ensemble_configs
from afid_b200.solver import slab_locations

FIELDS = ("vx", "vy", "vz", "temp", "pr")
REC_DOUBLES = 11          # afid_box_scalars: 10 doubles, then ntime and status
XSLAB = (0.03, 0.1, 0.25, 0.4, 0.5, 0.6, 0.75, 0.9)


# ----------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------
def _case(name, kind, nxm, nym, nzm, steps=1, ray=1e6, pra=1.0, graph=True, boxes=1, nsst=3, idtv=0,
          istr3=7, str3=0.0, inslws=1, inslwn=1):
    return {"name": name, "kind": kind, "nxm": nxm, "nym": nym, "nzm": nzm, "steps": steps, "ray": ray,
            "pra": pra, "graph": graph, "boxes": boxes, "nsst": nsst, "idtv": idtv, "istr3": istr3,
            "str3": str3, "inslws": inslws, "inslwn": inslwn}


def listed():
    return [
        # the smallest box of the tests, stepped launch by launch: latency and
        # launch count
        _case("box_24x16x12_direct", "advance", 24, 16, 12, steps=10, ray=1e5, pra=0.7, graph=False),
        # the smallest box of the ensemble, by graph: latency of one small job
        _case("box_32x32x32", "advance", 32, 32, 32, steps=40, ray=1e6),
        # the plain small configuration (65 x 64 x 64, Ra 1e6)
        _case("box_64x64x64", "advance", 64, 64, 64, steps=40, ray=1e6),
        # odd and ragged sizes, radices 3 and 5, tanh grid, CFL-adaptive dt
        _case("box_75x150x135_adaptive", "advance", 75, 150, 135, steps=20, ray=1e7, pra=4.38, idtv=1,
              istr3=4, str3=2.0),
        # Adams-Bashforth, one stress-free wall, clipped Chebyshev grid
        _case("box_96x128x80_ab2", "advance", 96, 128, 80, steps=40, ray=1e7, pra=0.7, nsst=1, istr3=6,
              str3=4.0, inslwn=0),
        # the benchmark's ensemble of 64 boxes in one batch
        _case("ensemble_64", "advance", 0, 0, 0, steps=20, boxes=64),
        # a small batch of served jobs: upload, reset, steps, download
        _case("jobs_12", "jobs", 0, 0, 0, steps=20, boxes=12),
        # the large box of the served mix
        _case("box_192x384x384", "advance", 192, 384, 384, steps=10, ray=1e9),
        # the plain large configuration (385 x 768 x 768, Ra 1e9)
        _case("box_384x768x768", "advance", 384, 768, 768, steps=10, ray=1e9),
        # the reference's subroutine boundaries, one time step
        _case("routines_64x96x96", "routines", 64, 96, 96, ray=1e7),
        # the pressure solve on the caller's device array
        _case("pressure_96x160x160", "pressure", 96, 160, 160),
        # output time of the served mix's large box
        _case("output_192x384x384", "output", 192, 384, 384, ray=1e9),
    ]


def _smooth(lo, hi, even):
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1 and not (even and n % 2):
            out.append(n)
    return out


def _pick(rng, choices):
    """One of sorted ``choices``, spread over their logarithm."""
    x = math.exp(rng.uniform(math.log(choices[0]), math.log(choices[-1] + 0.5)))
    return min(choices, key=lambda v: abs(math.log(v / x)))


def draw(rng):
    kind = rng.choice(["advance"] * 5 + ["set", "jobs", "routines", "pressure", "output"])
    if kind in ("set", "jobs"):
        n = int(round(math.exp(rng.uniform(math.log(2), math.log(64)))))
        c = _case("", "jobs" if kind == "jobs" else "advance", 0, 0, 0, steps=rng.randrange(10, 31), boxes=n,
                  graph=rng.random() < 0.8)
        c["set_seed"] = rng.randrange(1 << 20)
    else:
        most = {"advance": 40e6, "routines": 2e6, "pressure": 3.9e6, "output": 40e6}[kind]
        while True:
            nxm = int(round(math.exp(rng.uniform(math.log(16), math.log(400)))))
            nym = _pick(rng, _smooth(12, 800, True))
            nzm = min(_smooth(8, 800, False), key=lambda v: abs(math.log(v / (nym * math.exp(rng.uniform(-0.5, 0.5))))))
            if nxm * nym * nzm <= most and nxm / 8 <= nym <= 8 * nxm and (
                    kind != "pressure" or nxm * nzm * (nym // 2 + 1) <= 1 << 21):
                break
        cells = nxm * nym * nzm
        steps = 1 if kind in ("routines", "pressure", "output") else rng.randrange(20, 41) if cells < 2e6 else 10
        istr3 = rng.choice([7, 7, 7, 4, 6, 0])
        c = _case("", kind, nxm, nym, nzm, steps=steps, ray=10 ** rng.uniform(5, 8 if nxm < 128 else 9),
                  pra=rng.choice([0.7, 1.0, 4.38]), graph=rng.random() < 0.7,
                  nsst=rng.choice([3, 3, 3, 1]) if kind == "advance" else 3,
                  idtv=rng.choice([0, 0, 1]) if kind == "advance" else 0, istr3=istr3,
                  str3={4: 2.0, 6: 4.0}.get(istr3, 0.0), inslws=rng.choice([1, 1, 0]), inslwn=rng.choice([1, 1, 0]))
    del c["name"]
    return c


def _configs(case):
    if case["boxes"] > 1:
        return ensemble_configs(case["boxes"], seed=case.get("set_seed", 1000))
    nxm, nym, nzm, ray, pra = (case[k] for k in ("nxm", "nym", "nzm", "ray", "pra"))
    if _plain_large(case):
        ylen = zlen = 2.0
    else:
        ylen, zlen = (min(max(n / nxm, 0.5), 2.0) for n in (nym, nzm))
    h = min(ylen / nym, zlen / nzm)
    dt = min(5e-4, 0.1 * h, 0.1 * h * h * math.sqrt(ray / pra))
    return [BouIn(nxm=nxm, nym=nym, nzm=nzm, nsst=case["nsst"], ylen=ylen, zlen=zlen, ray=ray, pra=pra, dt=dt,
                  idtv=case["idtv"], dtmin=0.5 * dt, dtmax=2.0 * dt, istr3=case["istr3"], str3=case["str3"],
                  inslws=case["inslws"], inslwn=case["inslwn"], resid=0.0)]


def _plain_large(case):
    return case["nym"] == case["nzm"] and case["nym"] == 2 * case["nxm"]


def _cells(cfg):
    return cfg.nxm * cfg.nym * cfg.nzm


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid(cfg):
    return make_grid(cfg.nxm, cfg.istr3, cfg.str3, cfg.alx3)


def _inputs(cfg, xc, seed):
    """Fields in the boundary's order, (nzm, nym, rows) with x fastest:
    convection rolls of three seeded wavenumbers in a mean wind, with thermal
    noise of 1% (the benchmark's amplitude) between the plates; no pressure."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    f64 = dict(dtype=torch.float64, device=dev)
    nx, nym, nzm = cfg.nx, cfg.nym, cfg.nzm
    x = torch.tensor(xc, **f64)
    xm = torch.zeros(nx, **f64)
    xm[:-1] = 0.5 * (x[1:] + x[:-1])
    y = torch.arange(nym, **f64) / nym
    z = torch.arange(nzm, **f64) / nzm
    r = torch.rand(16, generator=gen, **f64).tolist()
    tau = 2.0 * math.pi
    out = {f: torch.zeros((nzm, nym, nx), **f64) for f in FIELDS}
    wall, slip = torch.sin(math.pi * x / xc[-1]), torch.cos(math.pi * xm / xc[-1])
    out["vx"] += 0.02 * wall
    out["vy"] += 0.05
    out["vz"] += 0.03
    for m in range(3):
        amp = 0.1 / (m + 1)
        py = torch.cos(tau * ((m + 1) * y + r[4 * m]))[None, :, None]
        qy = torch.sin(tau * ((m + 1) * y + r[4 * m]))[None, :, None]
        pz = torch.cos(tau * ((m + 1) * z + r[4 * m + 1]))[:, None, None]
        qz = torch.sin(tau * ((m + 1) * z + r[4 * m + 1]))[:, None, None]
        out["vx"] += amp * wall * (py * pz)
        out["vy"] += (0.5 * amp * (1.0 + 0.2 * r[4 * m + 2])) * slip * (qy * pz)
        out["vz"] += (0.5 * amp * (1.0 + 0.2 * r[4 * m + 3])) * slip * (py * qz)
        out["temp"] += amp * wall * (py * pz)
    noise = torch.rand((nzm, nym, nx - 2), generator=gen, **f64)
    out["temp"][:, :, 1:-1] += 0.02 * noise - 0.01
    out["temp"] += cfg.tempbp - (cfg.tempbp - cfg.temptp) * x / xc[-1]
    out["temp"][:, :, 0] = cfg.tempbp
    out["temp"][:, :, -1] = cfg.temptp
    for f in ("vy", "vz"):
        out[f][:, :, -1] = 0.0          # row nx of the staggered fields is unused
    out["vx"][:, :, 0] = 0.0
    out["vx"][:, :, -1] = 0.0
    return out


def _pressure_input(case, seed):
    """dph[k][i][j] as the divergence of a velocity field leaves it: noise
    over smooth modes, without a mean."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    d = torch.randn((case["nxm"], case["nzm"], case["nym"]), generator=gen, dtype=torch.float64, device=dev)
    return d - d.mean()


def _ptr(t, offset=0):
    return C.cast(t.data_ptr() + 8 * offset, C.POINTER(C.c_double))


_context = None


def _the_context():
    """The one context of the program: its boxes share a stream."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


class _State:
    """The boxes and the host buffers of one job; the boxes leave the context
    when the last reference goes."""

    def __init__(self, case):
        self.case = case
        self.boxes = []

    def __del__(self):
        for b in () if sys.is_finalizing() else self.boxes:
            self.ctx.remove_box(b)


def prepare(case, seed):
    s = _State(case)
    if case["kind"] == "pressure":
        s.rhs = _pressure_input(case, seed)
        s.dph = torch.empty_like(s.rhs)
        s.xc = make_grid(case["nxm"], case["istr3"], case["str3"], 1.0)
        s.stream = torch.cuda.current_stream()
        return s
    s.ctx = _the_context()
    cfgs = _configs(case)
    for c in cfgs:
        s.boxes.append(s.ctx.add_box(c))
    L, h = s.ctx._L, s.ctx.h
    s.sizes = [c.nx * c.nym * c.nzm for c in cfgs]
    s.at = [sum(s.sizes[:q]) for q in range(len(cfgs))]
    n = sum(s.sizes)
    s.inp = None
    if case["kind"] == "jobs":
        s.inp = {f: torch.empty(n, dtype=torch.float64, pin_memory=True) for f in FIELDS}
    stage = None if s.inp else torch.empty(max(s.sizes), dtype=torch.float64, pin_memory=True)
    for q, (box, cfg) in enumerate(zip(s.boxes, cfgs)):
        for f, v in _inputs(cfg, box.xc, seed + 1000 * q).items():
            host = s.inp[f][s.at[q]:s.at[q] + s.sizes[q]] if s.inp else stage[:s.sizes[q]]
            host.copy_(v.reshape(-1))
            _lib.check(L.afid_box_upload(h, box.id, _lib.FIELDS[f], _ptr(host)))
    s.ids = (C.c_int * len(cfgs))(*[b.id for b in s.boxes])
    if case["kind"] != "output":
        s.out = {f: torch.empty(n, dtype=torch.float64, pin_memory=True) for f in FIELDS}
    if case["kind"] in ("advance", "jobs"):
        s.rec = torch.zeros((len(cfgs), REC_DOUBLES), dtype=torch.float64, pin_memory=True)
        if case["graph"]:
            s.ctx.graph_kernels(s.boxes)         # the step graph a program keeps
    torch.cuda.synchronize()
    return s


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
def _upload(s):
    L, h = s.ctx._L, s.ctx.h
    for q, box in enumerate(s.boxes):
        for f in FIELDS:
            _lib.check(L.afid_box_upload_async(h, box.id, _lib.FIELDS[f], _ptr(s.inp[f], s.at[q])))
        box.reset(box.cfg.dt)


def _download(s):
    L, h = s.ctx._L, s.ctx.h
    for q, box in enumerate(s.boxes):
        for f in FIELDS:
            _lib.check(L.afid_box_download_async(h, box.id, _lib.FIELDS[f], _ptr(s.out[f], s.at[q])))
    return dict(s.out)


def run(s):
    kind = s.case["kind"]
    if kind == "pressure":
        c = s.case
        s.dph.copy_(s.rhs)
        _lib.check(_lib.lib().afid_solve_pressure_correction_noalloc(
            C.c_void_p(s.dph.data_ptr()), c["nxm"], c["nym"], c["nzm"], _lib.dptr(s.xc), 1.0, 1.0, 1.0,
            C.c_void_p(s.stream.cuda_stream), None))
        return s.dph
    if kind == "routines":
        s.boxes[0].time_marcher_routines()
        return _download(s)
    if kind == "output":
        b = s.boxes[0]
        nu_mu, nu_th = b.calc_dissipation_nu()
        b.calc_stats()
        g, st = b.global_quantities(), b.stats()
        out = {"cfl": b.calc_max_cfl(), "div": b.check_divergence(), "plate": list(b.calc_plate_nu()),
               "nu": [nu_mu, nu_th], "global": [g[k] for k in ("nu_vol", "tempm", "tempmax", "tempmin", "vx_rms")],
               "vmax": list(g["vmax"]), "slabs": b.slab_dump(slab_locations(b.xc, XSLAB))}
        n = st.pop("nstatsamples")
        out["stats"] = {k: v / n for k, v in st.items()}
        return out
    if kind == "jobs":
        _upload(s)
    s.ctx.step(s.boxes, s.case["steps"], graph=s.case["graph"])
    _lib.check(s.ctx._L.afid_boxes_get_scalars_async(
        s.ctx.h, s.ids, len(s.boxes), C.cast(s.rec.data_ptr(), C.POINTER(_lib.BoxScalars))))
    out = _download(s)
    out["time"] = s.rec[:, 0:2]                            # dt, time
    out["plate"] = s.rec[:, 8:10]                          # plate Nusselt numbers
    out["status"] = s.rec.view(torch.int32)[:, 20:22]      # step count and status
    return out


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def work(case):
    if case["kind"] == "pressure":
        n = case["nxm"] * case["nym"] * case["nzm"]
        lg = math.log2(case["nym"] * case["nzm"])
        return {"bytes": 16.0 * n, "flops": n * (5.0 * lg + 24.0)}
    byts = flops = 0.0
    for cfg in _configs(case):
        n = float(_cells(cfg))
        lg = math.log2(cfg.nym * cfg.nzm)
        sub = n * (400.0 + 5.0 * lg)                       # stencils, solves and transforms of a substep
        if case["kind"] == "output":
            byts += 32.0 * n
            flops += 120.0 * n
            continue
        # a substep reads and writes the five fields and the four histories
        # (its pressure solve couples the whole box, so substeps do not fuse)
        nsub = cfg.nsst * case["steps"]
        byts += nsub * 144.0 * n + 40.0 * n * (2 if case["kind"] == "jobs" else 1)
        flops += nsub * sub
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    # FP64 throughout.  Against ``exact`` the passes are off by up to 2e-12 in
    # the pressure (the x-solve is ill-conditioned in its lowest modes) and
    # 3e-12 in the plate Nusselt numbers (a rounding of the temperature over
    # the wall cell's height, 2e-5 at nxm = 384), the output sums by 1e-14;
    # taller and thinner grids raise the first two.
    return {"rel": 1e-12} if case["kind"] == "output" else {"rel": 1e-11}


# ----------------------------------------------------------------------------
# the same in plain torch, FP64 (fields indexed [k, j, i])
# ----------------------------------------------------------------------------
class _Plain:
    def __init__(self, cfg, xc, fields=None):
        dev = _device()
        self.c, self.dev = cfg, dev
        nxm, nym, nzm = cfg.nxm, cfg.nym, cfg.nzm
        nx = nxm + 1
        dx = nxm / cfg.alx3
        self.dy, self.dz = nym / cfg.ylen, nzm / cfg.zlen
        self.ren, self.pec = math.sqrt(cfg.ray / cfg.pra), math.sqrt(cfg.pra * cfg.ray)
        x = np.asarray(xc, dtype=np.float64)
        rm = (x[1:] - x[:-1]) * dx                          # g3rm(k), k < nxm
        rc = np.empty(nx)
        rc[1:-1] = (x[2:] - x[:-2]) * dx * 0.5
        rc[0], rc[-1] = rm[0], rm[-1]
        z = np.zeros(nx)
        self.udm, self.udc = dx / rm, dx / rc
        # nodes (vx, temp): rows 1..nxm-1
        cm, cp = z.copy(), z.copy()
        cp[1:-1] = dx * dx / rc[1:-1] / rm[1:]
        cm[1:-1] = dx * dx / rc[1:-1] / rm[:-1]
        self.node = (cm, -(cp + cm), cp)
        # centres (vy, vz) with the wall conditions
        sp, sm = dx * dx / rm / rc[1:], dx * dx / rm / rc[:-1]
        sc = -(sp + sm)
        sc[0] = -(sp[0] + cfg.inslws * 2.0 * sm[0])
        sc[-1] = -(sm[-1] + cfg.inslwn * 2.0 * sp[-1])
        sp2, sm2 = sp.copy(), sm.copy()
        sm2[0] = sp2[-1] = 0.0
        self.cent = (sm2, sc, sp2)
        # pressure rows
        pm, pp = dx * dx / rc[:-1] / rm, dx * dx / rc[1:] / rm
        pm[0] = pp[-1] = 0.0
        self.pois = (pm, -(pm + pp), pp)
        kz = np.minimum(np.arange(nzm), nzm - np.arange(nzm))
        self.ak1 = self._t(2.0 * (1.0 - np.cos(2.0 * np.pi * kz / nzm)) * self.dz ** 2)
        self.ak2 = self._t(2.0 * (1.0 - np.cos(2.0 * np.pi * np.arange(nym // 2 + 1) / nym)) * self.dy ** 2)
        self.xc, self.lu = x, None
        if fields is not None:
            self.q = {f: fields[f].permute(2, 1, 0).contiguous() for f in FIELDS}
            self.H = {f: torch.zeros_like(self.q["temp"]) for f in ("vx", "vy", "vz", "temp")}
            self.wall = torch.zeros((nym, nzm), dtype=torch.float64, device=dev)
            self.dt, self.time, self.ntime = cfg.dt, 0.0, 0
            self.rom, self.gam = ([0.0, -17 / 60, -5 / 12], [8 / 15, 5 / 12, 3 / 4]) if cfg.nsst > 1 else ([-0.5], [1.5])

    def _t(self, a):
        return torch.as_tensor(a, dtype=torch.float64, device=self.dev)

    def _k(self, a):
        return self._t(a)[:, None, None]

    @staticmethod
    def _p(a, d, s=-1):                                    # neighbour at +1 along d (1: y, 2: z)
        return torch.roll(a, s, d)

    def _m(self, a, d):
        return torch.roll(a, 1, d)

    def _implicit(self, row, n, bx, rhs):
        am, ac, ap = row
        A = np.eye(n)
        lo, hi = (0, n) if len(ac) == n and n == self.c.nxm else (1, n - 1)
        for k in range(lo, hi):
            A[k, k] = 1.0 - ac[k] * bx
            if k > 0:
                A[k, k - 1] = -am[k] * bx
            if k < n - 1:
                A[k, k + 1] = -ap[k] * bx
        inv = self._t(np.linalg.inv(A))
        return (inv @ rhs.reshape(n, -1)).reshape(rhs.shape)

    def _explicit(self):
        q, p, m = self.q, self._p, self._m
        vx, vy, vz, T = q["vx"], q["vy"], q["vz"], q["temp"]
        n = self.c.nxm
        udy, udz = self.dy * 0.25, self.dz * 0.25
        H = {f: torch.zeros_like(T) for f in ("vx", "vy", "vz", "temp")}

        def lap(a, nu):
            return (p(a, 1) - 2 * a + m(a, 1)) * (self.dy ** 2 / nu) + (p(a, 2) - 2 * a + m(a, 2)) * (self.dz ** 2 / nu)
        c, lo, hi = slice(1, n), slice(0, n - 1), slice(2, n + 1)
        wc = self._k(self.udc[1:n]) * 0.25
        ay, az = vy[c] + vy[lo], vz[c] + vz[lo]             # twice the velocities at the nodes
        vxc = vx[c]
        h = (vx[hi] + vxc) ** 2 - (vxc + vx[lo]) ** 2
        H["vx"][c] = (-(h * wc + (p(ay, 1) * (p(vxc, 1) + vxc) - ay * (vxc + m(vxc, 1))) * udy
                        + (p(az, 2) * (p(vxc, 2) + vxc) - az * (vxc + m(vxc, 2))) * udz)
                      + lap(vxc, self.ren) + T[c])
        t = T[c]
        h = (vx[hi] + vxc) * (T[hi] + t) - (vxc + vx[lo]) * (t + T[lo])
        H["temp"][c] = (-(h * wc + (p(ay, 1) * (p(t, 1) + t) - ay * (t + m(t, 1))) * udy
                          + (p(az, 2) * (p(t, 2) + t) - az * (t + m(t, 2))) * udz) + lap(t, self.pec))
        wm = self._k(self.udm) * 0.25
        for f, d in (("vy", 1), ("vz", 2)):
            a = q[f][:n]
            up = torch.cat([a[1:], a[-1:]])
            dn = torch.cat([a[:1], a[:-1]])
            fx = vx + m(vx, d)
            h = (fx[1:] * (up + a) - fx[:-1] * (a + dn)) * wm
            s = (p(a, d) + a) ** 2 - (a + m(a, d)) ** 2
            o, od, uo = (vz[:n], 2, udz) if f == "vy" else (vy[:n], 1, udy)
            fo = o + m(o, d)
            r = p(fo, od) * (p(a, od) + a) - fo * (a + m(a, od))
            H[f][:n] = -(h + s * (udy if d == 1 else udz) + r * uo) + lap(a, self.ren)
        return H

    def _second(self, row, a):
        am, ac, ap = (self._k(v) for v in row)
        up = torch.cat([a[1:], a[-1:]])
        dn = torch.cat([a[:1], a[:-1]])
        return up * ap + a * ac + dn * am

    def poisson(self, d):
        """dph from the right-hand side d[k, j, i]: Thomas along x per mode."""
        n = self.c.nxm
        if self.lu is None:
            lam = self.ak2[:, None] + self.ak1[None, :]
            pm, pc, pp = self.pois
            cp, rd = [], []
            for k in range(n):
                den = pc[k] - lam - (pm[k] * cp[-1] if k else 0.0)
                if k == n - 1:                             # the singular mode's last unknown is 0
                    den[0, 0] = math.inf
                rd.append(1.0 / den)
                cp.append(pp[k] * rd[-1])
            self.lu = cp, rd
        cp, rd = self.lu
        s = torch.fft.fft(torch.fft.rfft(d, dim=1), dim=2)
        s[0] *= rd[0]
        for k in range(1, n):
            s[k] = (s[k] - self.pois[0][k] * s[k - 1]) * rd[k]
        for k in range(n - 2, -1, -1):
            s[k] -= cp[k] * s[k + 1]
        return torch.fft.irfft(torch.fft.ifft(s, dim=2), n=self.c.nym, dim=1)

    def divergence(self):
        n, q = self.c.nxm, self.q
        vy, vz, vx = q["vy"][:n], q["vz"][:n], q["vx"]
        return ((self._p(vz, 2) - vz) * self.dz + (self._p(vy, 1) - vy) * self.dy
                + (vx[1:] - vx[:-1]) * self._k(self.udm))

    def max_cfl(self):
        n, q = self.c.nxm, self.q
        vy, vz, vx = q["vy"][:n], q["vz"][:n], q["vx"]
        return float((((vz + self._p(vz, 2)) * 0.5 * self.dz).abs() + ((vy + self._p(vy, 1)) * 0.5 * self.dy).abs()
                      + ((vx[1:] + vx[:-1]) * 0.5 * self._k(self.udm)).abs()).max())

    def plate(self):
        T, x = self.q["temp"], self.xc
        return [float((T[0] - T[1]).mean() / (x[1] - x[0])), float((T[-2] - T[-1]).mean() / (x[-1] - x[-2]))]

    def step(self):
        c, q, n = self.c, self.q, self.c.nxm
        if c.idtv:
            cfl = self.max_cfl()
            self.dt = min(c.cflmax / max(cfl, 1e-8), c.dtmax) if self.ntime > 1 else c.dtmin
        dt = self.dt
        for ga, ro in zip(self.gam, self.rom):
            al = ga + ro
            H = self._explicit()
            pr, bre, bpe = q["pr"], 0.5 * al * dt / self.ren, 0.5 * al * dt / self.pec
            grad = {"vx": torch.zeros_like(pr), "vy": (pr - self._m(pr, 1)) * self.dy,
                    "vz": (pr - self._m(pr, 2)) * self.dz, "temp": torch.zeros_like(pr)}
            grad["vx"][1:n] = (pr[1:n] - pr[:n - 1]) * self._k(self.udc[1:n])
            new = {}
            for f in ("vx", "vy", "vz", "temp"):
                rhs = (ga * H[f] + ro * self.H[f] - al * grad[f]) * dt
                if f in ("vy", "vz"):
                    rhs = rhs[:n] + 2.0 * bre * self._second(self.cent, q[f][:n])
                    d = self._implicit(self.cent, n, bre, rhs)
                    if f == "vz":
                        self.wall = d[0].clone()
                    new[f] = q[f].clone()
                    new[f][:n] += d
                else:
                    b = bre if f == "vx" else bpe
                    rhs = rhs + 2.0 * b * self._second(self.node, q[f])
                    # row 1 holds what the last vz solve left there, row nx zero
                    rhs[0] = self.wall
                    rhs[-1] = 0.0
                    new[f] = q[f] + self._implicit(self.node, n + 1, b, rhs)
            new["vx"][0] = 0.0
            new["vx"][-1] = 0.0
            new["temp"][0], new["temp"][-1] = c.tempbp, c.temptp
            self.H = H
            q.update(new)
            phi = self.poisson(self.divergence() / (al * dt))
            q["vx"][1:n] -= (phi[1:] - phi[:-1]) * (al * dt * self._k(self.udc[1:n]))
            q["vy"][:n] -= (phi - self._m(phi, 1)) * (al * dt * self.dy)
            q["vz"][:n] -= (phi - self._m(phi, 2)) * (al * dt * self.dz)
            lap = ((self._p(phi, 1) - 2 * phi + self._m(phi, 1)) * self.dy ** 2
                   + (self._p(phi, 2) - 2 * phi + self._m(phi, 2)) * self.dz ** 2 + self._second(self.pois, phi))
            q["pr"][:n] += phi - (al * 0.5 * dt / self.ren) * lap
        self.time += dt
        self.ntime += 1

    def out(self, f):
        return self.q[f].permute(2, 1, 0).reshape(-1)

    def diagnostics(self):
        c, q, n, x = self.c, self.q, self.c.nxm, self.xc
        vx, vy, vz, T = (q[f] for f in ("vx", "vy", "vz", "temp"))
        dx = n / c.alx3
        P = c.nym * c.nzm
        g = np.empty(n)
        g[0] = (x[1] - x[0]) * dx
        g[1:] = (x[2:] - x[:-2])[:n - 1] * dx * 0.5
        w = self._t(g)
        vol = 1.0 / (c.alx3 * dx * P)
        lo, hi = slice(0, n), slice(1, n + 1)

        def s(a):
            return a.sum(dim=(1, 2))
        tc = (T[lo] + T[hi]) * 0.5
        glob = [1.0 + self.pec * float((s(tc * (vx[lo] + vx[hi]) * 0.5) * w).sum()) * vol,
                float((s(tc) * w).sum()) * vol, float(T[lo].max()), float(T[lo].min()),
                math.sqrt(float((s(vx[lo] ** 2) * w).sum()) * vol) * self.ren]
        xm = 0.5 * (x[1:] + x[:-1])
        dm = np.append(xm[1:] - xm[:-1], xm[-1] - xm[-2])
        ic, im = self._k(1.0 / (x[1:] - x[:-1])), self._k(1.0 / dm)

        def grad2(a, ix):
            b = a[lo]
            return s(((a[hi] - b) * ix) ** 2 + ((self._p(b, 1) - b) * self.dy) ** 2 + ((self._p(b, 2) - b) * self.dz) ** 2)
        d1, d2, dt = grad2(vx, ic), grad2(vy, im) + grad2(vz, im), grad2(T, ic)
        lem, lec = self._t((x[1:] - x[:-1]) * dx), self._t(dm * dx)
        nu = [float((d1 * lem + d2 * lec).sum()) * c.pra / (n * P) + 1.0, float((dt * lem).sum()) / (n * P)]
        st = {"vx_me": s(vx[lo]), "vy_me": s(vy[lo]), "vz_me": s(vz[lo]), "temp_me": s(T[lo]), "vx_rms": s(vx[lo] ** 2),
              "vy_rms": s(vy[lo] ** 2), "vz_rms": s(vz[lo] ** 2), "temp_rms": s(T[lo] ** 2), "tempvx_me": s(T[lo] * vx[lo]),
              "disste": (d1 + d2) / self.ren, "dissth": dt / self.pec}
        ks = [2] * 9
        for k in range(2, n + 1):
            for m, p in enumerate(XSLAB):
                if xm[k - 2] < p < xm[k - 1]:
                    ks[m + 1] = k
        slabs = torch.stack([torch.stack([(vx[k - 1] + vx[k]) * 0.5, vy[k - 1], vz[k - 1], T[k - 1]]) for k in ks])
        return {"cfl": self.max_cfl(), "div": float(self.divergence().abs().max()), "plate": self.plate(), "nu": nu,
                "global": glob, "vmax": [float(a[lo].abs().max()) for a in (vz, vy, vx)], "slabs": slabs,
                "stats": {k: v / P for k, v in st.items()}}


def exact(case, seed):
    if case["kind"] == "pressure":
        cfg = BouIn(nxm=case["nxm"], nym=case["nym"], nzm=case["nzm"])
        p = _Plain(cfg, make_grid(case["nxm"], case["istr3"], case["str3"], 1.0))
        return p.poisson(_pressure_input(case, seed).permute(0, 2, 1)).permute(0, 2, 1)
    cfgs = _configs(case)
    # about 0.1 ms a plane, box and substep, and the time of the fields' traffic
    if sum(c.nxm for c in cfgs) * case["steps"] * cfgs[0].nsst * 1.5e-4 > 15.0:
        return None
    plain = []
    for q, cfg in enumerate(cfgs):
        xc = _grid(cfg)
        plain.append(_Plain(cfg, xc, _inputs(cfg, xc, seed + 1000 * q)))
    if case["kind"] == "output":
        return plain[0].diagnostics()
    for p in plain:
        for _ in range(case["steps"]):
            p.step()
    out = {f: torch.cat([p.out(f) for p in plain]) for f in FIELDS}
    if case["kind"] != "routines":
        out["time"] = np.array([[p.dt, p.time] for p in plain])
        out["plate"] = np.array([p.plate() for p in plain])
        out["status"] = None
    return out
