"""The work a user of this framework has it do, as cases that can be timed and
checked: single domains in FP64 (the reference's own arithmetic) and FP32,
with the reference's fixed time step and with the CFL rule, every kind of
forcing, ensembles in one batch, and a served stream of requests -- from grids
of a few thousand cells, where the latency of an iteration counts, to 8192 x
8192.  Every case goes through the package's public classes (Solver, Batch,
ServerHandle): set the state, advance, read the results back.

Terrain, roughness and water depths are seeded: a tilted plane with six
octaves of fractal noise, land-use patches for Manning's n, and a sheet of
water of varying depth -- with dry ground in it where a case starts an event or
a storm covers part of the domain, and a film of rain on all of it where a case
goes on in the middle of one.

Single-precision results are handed on as float32 rasters: the FP32 path holds
its planes in float32 and the reading calls only widen them.
"""
import os
import sys

import numpy as np
import torch
import torch.nn.functional as nnf

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sw2d-gpu_gb300"))
import sw2d  # noqa: E402

MANNING = (0.03, 0.05, 0.08, 0.12)  # land-use classes
G, TH = 9.80, 1.0e-4                # the library's defaults
HALF_STEP = 0.04                    # the reference's usual fixed half step [s]
CFL_HALF_STEP = 2.0                 # largest half step under the CFL rule [s]
TABLE_DT = 1.0e6                    # interval of the source and evaporation records [s]


def _solver(name, rows, cols, iters, **kw):
    case = {
        "name": name, "kind": "solver", "precision": "f32", "dt": "cfl", "rows": rows, "cols": cols, "dx": 5.0,
        "iters": iters, "bed": "terrain", "manning": "raster", "rain": "step", "sources": 0, "evaporation": False,
        "weights": False, "south_open": True, "fresh": False, "read": "depth",
    }
    case.update(kw)
    return case


def listed():
    return [
        # the plain method at its small size: a dam break along a frictionless channel, reflecting walls
        _solver("f64_dam_break", 256, 512, 100, precision="f64", dx=1.0, bed="channel", manning="none", rain="none",
                south_open=False, fresh=True, read="state"),
        # a run as the reference's own datasets ask for it: one small basin, the fixed time step up to the next
        # output time, the reference's rain formula, point sources, evaporation and runoff fractions, then the
        # depth and the cell velocities for the output file
        _solver("f64_basin_output", 117, 131, 150, precision="f64", dt="fixed", dx=10.0, manning="scalar",
                rain="compat", sources=3, evaporation=True, south_open=False, fresh=True, read="velocity"),
        # a catchment in double precision
        _solver("f64_catchment", 1013, 900, 30, precision="f64", read="state"),
        # the smallest domains: the time of one iteration is latency and launches
        _solver("f32_small", 96, 128, 250, fresh=True, read="state"),
        # a mid-size domain under the fixed time step
        _solver("f32_fixed_step", 512, 512, 300, dt="fixed", dx=10.0, manning="scalar", rain="compat", fresh=True,
                read="state"),
        # the synthetic catchment between two output times: per-cell roughness, rain, open south edge
        _solver("f32_catchment", 2048, 2048, 480),
        # the large domain under a moving storm cell, scalar roughness
        _solver("f32_large_storm", 8192, 8192, 96, dx=2.0, manning="scalar", rain="storm"),
        # inflows into an odd-sized domain with evaporation
        _solver("f32_sources", 701, 1237, 200, sources=6, evaporation=True, read="state"),
        # a rainfall raster on a mid-size domain
        _solver("f32_rain_raster", 1500, 900, 200, weights=True),
        # an ensemble of uneven grids in one batch
        {"name": "batch_ensemble", "kind": "batch", "count": 24, "side_min": 128, "side_max": 1024, "iters": 144},
        # a handful of small scenarios in one batch
        {"name": "batch_small", "kind": "batch", "count": 8, "side_min": 64, "side_max": 128, "iters": 240},
        # requests submitted together and served to their end times
        {"name": "served", "kind": "served", "count": 8, "side_min": 64, "side_max": 256, "horizon": 300.0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    what = rng.choice(("f64", "f64", "cfl", "cfl", "fixed", "forced", "batch", "served"))
    if what == "batch":
        hi = _log_int(rng, 96, 1024)
        return {"kind": "batch", "count": rng.randint(3, 24), "side_min": min(64, hi // 2), "side_max": hi,
                "iters": rng.randint(60, 200)}
    if what == "served":
        hi = _log_int(rng, 96, 300)
        return {"kind": "served", "count": rng.randint(2, 8), "side_min": 64, "side_max": hi,
                "horizon": float(rng.randint(150, 300))}
    south, raster = rng.random() < 0.7, rng.choice(("raster", "scalar"))
    if what == "f64":
        rows, cols = _log_int(rng, 48, 1100), _log_int(rng, 48, 1100)
        cells = rows * cols
        fixed = rng.random() < 0.5
        case = _solver("", rows, cols, rng.randint(20, 40) if cells > 200000 else rng.randint(60, 160),
                       precision="f64", dt="fixed" if fixed else "cfl", manning=raster, south_open=south,
                       dx=10.0 if fixed else 5.0, rain=rng.choice(("compat", "none")) if fixed else "step",
                       read=rng.choice(("state", "velocity")), fresh=cells < 300000)
    else:
        hi = 1300 if what == "fixed" else 3000
        rows, cols = _log_int(rng, 64, hi), _log_int(rng, 64, hi)
        case = _solver("", rows, cols, rng.randint(150, 300), manning=raster, south_open=south,
                       read="state" if rows * cols < 1000000 else "depth", fresh=rows * cols < 300000)
        if what == "fixed":
            case.update(dt="fixed", dx=10.0, rain="compat")
            case["fresh"] = True
        elif what == "forced":
            case.update(rng.choice(({"sources": rng.randint(1, 10), "evaporation": True}, {"weights": True},
                                    {"rain": "storm"})))
    del case["name"]
    return case


# ---- inputs ------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _noise(g, rows, cols, octaves=6, base=4):
    """Fractal value noise in [-1, 1]: bilinear lattices, frequency doubling and amplitude halving per octave."""
    out = torch.zeros((rows, cols), dtype=torch.float64, device=_device())
    amp, total = 1.0, 0.0
    for o in range(octaves):
        f = base * 2 ** o
        lat = torch.rand((1, 1, f + 1, f + 1), generator=g, dtype=torch.float64, device=_device()) * 2.0 - 1.0
        out += amp * nnf.interpolate(lat, size=(rows, cols), mode="bilinear", align_corners=True)[0, 0]
        total += amp
        amp *= 0.5
    return out / total


def _landuse(g, rows, cols):
    lat = torch.randint(0, len(MANNING), (1, 1, 16, 16), generator=g, device=_device()).to(torch.float64)
    idx = nnf.interpolate(lat, size=(rows, cols), mode="nearest")[0, 0].to(torch.int64)
    return torch.tensor(MANNING, dtype=torch.float64, device=_device())[idx]


def _water(g, rows, cols, start):
    """A sheet of up to a few centimetres of water: with dry ground in it at the start of an event, and a film of
    rain on all of it later on."""
    return torch.clamp(0.012 + 0.05 * _noise(g, rows, cols), min=0.0 if start else 0.002)


def _field(case, seed):
    """Bed, roughness (or None) and initial depth of a solver case, on the device, in float64."""
    rows, cols, dx = case["rows"], case["cols"], case["dx"]
    g = _generator(seed)
    if case["bed"] == "channel":
        r = torch.rand(2, generator=g, dtype=torch.float64, device=_device())
        z = torch.zeros((rows, cols), dtype=torch.float64, device=_device())
        x = (torch.arange(cols, dtype=torch.float64, device=_device()) + 0.5) * dx
        h = torch.where(x < cols * dx * (0.4 + 0.2 * r[0]), 8.0 + 4.0 * r[1], torch.zeros_like(x))
        return z, None, h.expand(rows, cols).clone()
    i = torch.arange(rows, dtype=torch.float64, device=_device())[:, None]
    z = 0.01 * dx * (rows - 1 - i) + 2.0 * _noise(g, rows, cols)
    if case["precision"] == "f64" and case["dt"] == "fixed":
        z = z.clone()
        z[:, :2] = -9999.0  # NODATA, as around a digitised basin
    n = _landuse(g, rows, cols) if case["manning"] == "raster" else None
    return z, n, _water(g, rows, cols, case["fresh"] or case["rain"] == "storm")


def _forcing(case, seed):
    """Rain, sources and evaporation of a solver case, as plain numbers and arrays."""
    r = np.random.default_rng([int(seed), 7])
    rows, cols, dx = case["rows"], case["cols"], case["dx"]
    f = {"manning": 0.05 if case["manning"] == "scalar" else 0.0, "rain": None, "storm": None, "sources": None,
         "ev": None, "weights": None}
    if case["rain"] == "step":      # mm/h, hour by hour
        f["rain"] = (r.uniform(20.0, 60.0, 2000), 3600.0)
    elif case["rain"] == "compat":  # mm per interval, the reference's formula
        f["rain"] = (r.uniform(2.0, 5.0, 64), 631.7)
    elif case["rain"] == "storm":
        f["storm"] = {"peak": float(r.uniform(60.0, 100.0)), "x0": 0.0, "y0": 0.0, "vx": 10.0 / 2 ** 0.5,
                      "vy": 10.0 / 2 ** 0.5, "sigma": 0.12 * dx * min(rows, cols)}
    if case["sources"]:
        k = case["sources"]
        f["sources"] = (r.choice(rows * cols, size=k, replace=False).astype(np.int32), r.uniform(0.2, 1.5, (4, k)))
    if case["evaporation"]:
        f["ev"] = r.uniform(0.1, 0.6, 8)  # mm per hour
    return f


def _weights(case, seed):
    return 1.0 + 0.8 * _noise(_generator(seed + 1000003), case["rows"], case["cols"], octaves=3)


def _fractions(case):
    """Runoff fractions of the reference's setup, where evaporation is on."""
    return {"INT": 0.1, "INF": 0.2, "LWL": 0.05, "EV_WL_min": 0.01} if case["evaporation"] else {}


def _half_step(case):
    return HALF_STEP if case["dt"] == "fixed" else CFL_HALF_STEP


def _t_end(case, t0=0.0):
    """The end time a fixed-step run of `iters` iterations is given (t0 + the steps, less a quarter step)."""
    return t0 + 2.0 * HALF_STEP * case["iters"] - 0.5 * HALF_STEP


def _members(case, seed):
    """The scenarios of a batch or of a request stream: windows of one terrain, each with its own rain and scaling
    of the roughness."""
    r = np.random.default_rng([int(seed), 11])
    lo, hi = case["side_min"], case["side_max"]
    size = hi + 256
    g = _generator(seed)
    i = torch.arange(size, dtype=torch.float64, device=_device())[:, None]
    z = 0.01 * 5.0 * (size - 1 - i) + 2.0 * _noise(g, size, size, octaves=6, base=max(4, size // 512 * 4))
    n, h = _landuse(g, size, size), _water(g, size, size, case["kind"] == "served")
    out = []
    for k in range(case["count"]):
        # the sides are the case's: the inputs are the seed's
        t = (k * 0.6180339887498949 + 0.11) % 1.0
        rows = int(round(lo * (hi / lo) ** t))
        cols = max(lo, min(hi, rows + (k * 37) % 23 - 11))
        a, b = int(r.integers(0, size - rows + 1)), int(r.integers(0, size - cols + 1))
        out.append({
            "rows": rows, "cols": cols, "z": z[a:a + rows, b:b + cols].contiguous(),
            "n": (n[a:a + rows, b:b + cols] * float(r.uniform(0.8, 1.2))).contiguous(),
            "h": h[a:a + rows, b:b + cols].contiguous(),
            # a triangular hyetograph, mm/h, over a long event
            "rain": np.array([20.0, float(r.uniform(40.0, 120.0)), 20.0]), "rain_dt": 40000.0,
        })
    return out


def _host(t):
    return None if t is None else t.cpu().numpy()


def _member_config(m):
    return sw2d.default_config(rows=m["rows"], cols=m["cols"], dx=5.0, dy=5.0, precision=sw2d.PREC_F32,
                               dt_mode=sw2d.DT_CFL, dt=CFL_HALF_STEP, cfl=0.5, south_open=1)


# ---- one pass ------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] in ("batch", "served"):
        members = _members(case, seed)
        if case["kind"] == "batch":
            b = sw2d.Batch(device=0, max_scenarios=case["count"])
            ids = [b.add(_member_config(m), _host(m["z"]), _host(m["h"]), manning=_host(m["n"]),
                         rain_kind=sw2d.RAIN_LINEAR, rain=m["rain"], rain_dt=m["rain_dt"]) for m in members]
            return {"case": case, "batch": b, "ids": ids}
        s = sw2d.ServerHandle(max_scenarios=max(16, case["count"]))
        return {"case": case, "server": s, "members": [
            dict(m, cfg=_member_config(m), z=_host(m["z"]), n=_host(m["n"]), h=_host(m["h"])) for m in members]}
    z, n, h = (_host(t) for t in _field(case, seed))
    f = _forcing(case, seed)
    s = sw2d.Solver(rows=case["rows"], cols=case["cols"], dx=case["dx"], dy=case["dx"], manning=f["manning"],
                    precision=sw2d.PREC_F64 if case["precision"] == "f64" else sw2d.PREC_F32,
                    dt_mode=sw2d.DT_FIXED if case["dt"] == "fixed" else sw2d.DT_CFL, dt=_half_step(case), cfl=0.5,
                    south_open=1 if case["south_open"] else 0, **_fractions(case))
    s.set_static(z, n)
    if f["rain"] is not None:
        s.set_rain(sw2d.RAIN_COMPAT if case["rain"] == "compat" else sw2d.RAIN_STEP, *f["rain"])
    if f["storm"] is not None:
        s.set_storm(**f["storm"])
    if f["sources"] is not None:
        s.set_point_sources(f["sources"][0], f["sources"][1], TABLE_DT)
    if f["ev"] is not None:
        s.set_evaporation(f["ev"], 3600.0)
    if case["weights"]:
        s.set_rain_weights(_host(_weights(case, seed)))
    s.set_state(h)
    return {"case": case, "solver": s, "h": h}


def _as_read(case, a):
    return torch.from_numpy(a) if case.get("precision") == "f64" else torch.from_numpy(a).to(torch.float32)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.advance(case["iters"])
        return {"depth": [_as_read(case, b.field(i)) for i in state["ids"]]}
    if case["kind"] == "served":
        s = state["server"]
        rids = [s.submit(m["cfg"], m["z"], m["h"], manning=m["n"], rain_kind=sw2d.RAIN_LINEAR, rain=m["rain"],
                         rain_dt=m["rain_dt"], t_end=case["horizon"]) for m in state["members"]]
        while any(s.step()):
            pass
        out = {"depth": [], "rain_in": []}
        for rid in rids:
            out["depth"].append(_as_read(case, s.depth(rid)))
            out["rain_in"].append(s.budget(rid)["rain_in"])
            s.release(rid)
        return out
    s = state["solver"]
    if case["fresh"]:  # the event from its start; otherwise on from the last output time
        s.set_state(state["h"])
    if case["dt"] == "fixed" and case["fresh"]:
        s.advance(10 ** 9, _t_end(case))
    else:
        s.advance(case["iters"])
    out = {"depth": _as_read(case, s.depth())}
    if case["read"] == "state":
        out["um"] = _as_read(case, s.field(sw2d.FIELD_UM))
        out["vn"] = _as_read(case, s.field(sw2d.FIELD_VN))
    elif case["read"] == "velocity":
        out["uu"] = _as_read(case, s.field(sw2d.FIELD_UU))
        out["vv"] = _as_read(case, s.field(sw2d.FIELD_VV))
    b = s.budget()
    out.update({k: b[k] for k in ("t", "volume", "rain_in", "outflow")})
    return out


def work(case):
    """Each iteration reads depth, the two discharges, bed and roughness of every cell and writes the first three;
    about 170 operations (a power, root or division counted as one) per cell and iteration."""
    if case["kind"] == "solver":
        per, cells = 8 if case["precision"] == "f64" else 4, case["rows"] * case["cols"]
        fields = 8 if case["manning"] == "raster" else 7
        return {"bytes": float(cells * case["iters"] * fields * per), "flops": 170.0 * cells * case["iters"]}
    lo, hi = case["side_min"], case["side_max"]
    cells = sum(int(round(lo * (hi / lo) ** ((k * 0.6180339887498949 + 0.11) % 1.0))) ** 2 for k in range(case["count"]))
    iters = case["iters"] if case["kind"] == "batch" else int(case["horizon"] / 1.0)  # about a second per CFL step
    return {"bytes": float(cells * iters * 32), "flops": 170.0 * cells * iters}


# ---- the same in 64 bits, in plain torch ----------------------------------------

def _pad(a, left, right, dim):
    p = [0, 0, 0, 0]
    p[2 * (1 - dim)], p[2 * (1 - dim) + 1] = left, right
    return nnf.pad(a, p)


class _Plain:
    """The scheme on whole arrays: x-faces (rows + 1, cols) and y-faces (rows, cols + 1) with zero walls."""

    def __init__(self, z, n, h, dx, manning=0.0, half=1.0, fixed=False, south=False, INT=0.0, INF=0.0, LWL=0.0,
                 EV_WL_min=0.0):
        self.z, self.dx, self.half, self.fixed, self.south = z, dx, half, fixed, south
        self.hi, self.lo, self.evmin = 1.0 - LWL, 1.0 - (INT + INF), EV_WL_min
        self.act = z != -9999.0
        self.ax = self.act[1:] & self.act[:-1]
        self.ay = self.act[:, 1:] & self.act[:, :-1]
        self.nx = 0.5 * (n[1:] + n[:-1]) if n is not None else manning
        self.ny = 0.5 * (n[:, 1:] + n[:, :-1]) if n is not None else manning
        self.h = torch.where(self.act, h, torch.zeros_like(h))
        rows, cols = h.shape
        self.um = torch.zeros((rows + 1, cols), dtype=torch.float64, device=h.device)
        self.vn = torch.zeros((rows, cols + 1), dtype=torch.float64, device=h.device)
        self.t = self.rain_in = self.outflow = 0.0
        self.derive()

    def derive(self):
        h = self.h
        hm = torch.cat([h[:1], 0.5 * (h[1:] + h[:-1]), h[-1:]], 0)
        hn = torch.cat([h[:, :1], 0.5 * (h[:, 1:] + h[:, :-1]), h[:, -1:]], 1)
        self.hm, self.hn = hm, hn
        self.uu = torch.where(hm >= TH, self.um / hm.clamp(min=TH), torch.zeros_like(hm))
        self.vv = torch.where(hn >= TH, self.vn / hn.clamp(min=TH), torch.zeros_like(hn))

    def cmax(self):
        c = 0.0
        for ok, h, v in ((self.ax, self.hm[1:-1], self.uu[1:-1]), (self.ay, self.hn[:, 1:-1], self.vv[:, 1:-1]),
                         (self.act[-1:] & self.south, self.hm[-1:], self.uu[-1:])):
            if h.numel():
                s = torch.where(ok & (h >= TH), v.abs() + torch.sqrt(G * h), torch.zeros_like(h))
                c = max(c, float(s.max()))
        return c

    @staticmethod
    def flux(vel, other, own, side):
        """The reference's upwinded flux through one side of a control volume."""
        d = own - other if side > 0 else other - own
        return vel * (other + own) * 0.5 + vel.abs() * d * 0.5

    @staticmethod
    def face(ha, hb, za, zb, hf, q, adv, slope_dt, speed, n, dt2, act):
        zero = torch.zeros_like(q)
        ram = G * n * n * speed / hf.clamp(min=TH) ** 1.3333330
        ram = torch.where(hf > TH, ram, zero)
        grav = G * hf * slope_dt * (hb + zb - ha - za)
        out = ((1.0 - dt2 * ram * 0.5) * q + (-adv - grav)) / (1.0 + dt2 * ram * 0.5)
        hh = (torch.maximum(hb + zb, ha + za) - torch.maximum(zb, za)).clamp(min=0.0)
        weir = -0.35 * torch.sign(hb - ha) * hh * torch.sqrt(2.0 * G * hh)
        out = torch.where((hb - TH) * (ha - TH) < 0, weir, out)
        out = torch.where(ha + za < zb, torch.where(hb > TH, -0.544 * hb * torch.sqrt(G * hb), zero), out)
        out = torch.where(hb + zb < za, torch.where(ha > TH, 0.544 * ha * torch.sqrt(G * ha), zero), out)
        return torch.where(act & ((ha > TH) | (hb > TH)), out, zero)

    def momentum(self, dt2):
        h, z, um, vn, uu, vv, dx = self.h, self.z, self.um, self.vn, self.uu, self.vv, self.dx
        k, F = dt2 / dx, self.flux
        umE, umW = _pad(um, 0, 1, 1)[:, 1:], _pad(um, 1, 0, 1)[:, :-1]
        adv = k * (F(0.5 * (uu[2:] + uu[1:-1]), um[2:], um[1:-1], 1) -
                   F(0.5 * (uu[1:-1] + uu[:-2]), um[:-2], um[1:-1], -1))
        side = k * (F(0.5 * (vv[1:, 1:] + vv[:-1, 1:]), umE[1:-1], um[1:-1], 1) -
                    F(0.5 * (vv[1:, :-1] + vv[:-1, :-1]), umW[1:-1], um[1:-1], -1))
        side[:, :1] = 0.0
        va = 0.25 * (vv[1:, :-1] + vv[1:, 1:] + vv[:-1, :-1] + vv[:-1, 1:])
        nu = torch.zeros_like(um)
        nu[1:-1] = self.face(h[:-1], h[1:], z[:-1], z[1:], self.hm[1:-1], um[1:-1], adv + side, k,
                             torch.sqrt(uu[1:-1] ** 2 + va ** 2), self.nx, dt2, self.ax)
        if self.south:
            hs = h[-1]
            nu[-1] = torch.where(self.act[-1] & (hs > TH), 0.544 * hs * torch.sqrt(G * hs), torch.zeros_like(hs))
        vnS, vnN = _pad(vn, 0, 1, 0)[1:], _pad(vn, 1, 0, 0)[:-1]
        adv = k * (F(0.5 * (uu[1:, 1:] + uu[1:, :-1]), vnS[:, 1:-1], vn[:, 1:-1], 1) -
                   F(0.5 * (uu[:-1, 1:] + uu[:-1, :-1]), vnN[:, 1:-1], vn[:, 1:-1], -1))
        adv[:1] = 0.0
        side = k * (F(0.5 * (vv[:, 2:] + vv[:, 1:-1]), vn[:, 2:], vn[:, 1:-1], 1) -
                    F(0.5 * (vv[:, 1:-1] + vv[:, :-2]), vn[:, :-2], vn[:, 1:-1], -1))
        ua = 0.25 * (uu[:-1, 1:] + uu[1:, 1:] + uu[:-1, :-1] + uu[1:, :-1])
        nv = torch.zeros_like(vn)
        nv[:, 1:-1] = self.face(h[:, :-1], h[:, 1:], z[:, :-1], z[:, 1:], self.hn[:, 1:-1], vn[:, 1:-1], adv + side,
                                k, torch.sqrt(ua ** 2 + vv[:, 1:-1] ** 2), self.ny, dt2, self.ay)
        return nu, nv

    def depth(self, nu, nv, dt2, rain, ev, ql):
        wet = self.h > self.evmin
        pct = torch.where(wet, torch.full_like(self.h, self.hi), self.lo)
        gain = rain * pct
        h = self.h - dt2 * ((nu[1:] - nu[:-1]) / self.dx + (nv[:, 1:] - nv[:, :-1]) / self.dx - ql - gain +
                            ev * wet)
        return torch.where(self.act, h.clamp(min=0.0), torch.zeros_like(h)), gain

    def step(self, dt2, forcing):
        dt = 0.5 * dt2
        nu, nv = self.momentum(dt2)
        hs, _ = self.depth(nu, nv, dt2, *forcing(self.t))
        dry = self.act & (hs < TH)
        below, above = _pad(dry, 0, 1, 0), _pad(dry, 1, 0, 0)
        nu = torch.where(((nu > 0) & above) | ((nu < 0) & below), torch.zeros_like(nu), nu)
        right, left = _pad(dry, 0, 1, 1), _pad(dry, 1, 0, 1)
        nv = torch.where(((nv > 0) & left) | ((nv < 0) & right), torch.zeros_like(nv), nv)
        h, gain = self.depth(nu, nv, dt2, *forcing(self.t + dt))
        self.rain_in += dt2 * self.dx ** 2 * float(torch.where(self.act, gain, torch.zeros_like(h)).sum())
        self.outflow += dt2 * self.dx * float(nu[-1].sum())
        self.h, self.um, self.vn = h, nu, nv
        self.t = (self.t + dt) + dt
        self.derive()

    def advance(self, iters, forcing, t_end=1e300):
        for _ in range(iters):
            if self.fixed:
                if not self.t + self.half <= t_end:
                    return
                dt2 = 2.0 * self.half
            else:
                if not t_end - self.t > 1e-9:
                    return
                c = self.cmax()
                dt2 = min(2.0 * self.half, 0.5 * self.dx / c) if c > 0 else 2.0 * self.half
                dt2 = min(dt2, t_end - self.t)
            self.step(dt2, forcing)

    def cell_velocity(self):
        wet, zero = self.h >= TH, torch.zeros_like(self.h)
        return (torch.where(wet, 0.5 * (self.uu[1:] + self.uu[:-1]), zero),
                torch.where(wet, 0.5 * (self.vv[:, 1:] + self.vv[:, :-1]), zero))


def _compat(v, dt, t):
    """The reference's interpolation of a record (it divides by the time inside the interval)."""
    if t <= 1.0:
        return v[0] * t
    k = int(t / dt)
    a, b = v[min(k, len(v) - 1)], v[min(k + 1, len(v) - 1)]
    return a + (b - a) / (dt * (t - dt * k))


def _linear(v, dt, t):
    k = int(t // dt)
    return 0.0 if k >= len(v) - 1 else (v[k] + (t / dt - k) * (v[k + 1] - v[k])) / 3.6e6


def exact(case, seed):
    if case["kind"] in ("batch", "served"):
        if case["kind"] == "served" and case["horizon"] * case["count"] > 2600.0:
            return None
        out = {"depth": [], "rain_in": []}
        for m in _members(case, seed):
            p = _Plain(m["z"], m["n"], m["h"], 5.0, half=CFL_HALF_STEP, south=True)
            forcing = lambda t, m=m: (_linear(m["rain"], m["rain_dt"], t), 0.0, 0.0)  # noqa: E731
            if case["kind"] == "batch":
                p.advance(case["iters"], forcing)
            else:
                p.advance(10 ** 6, forcing, case["horizon"])
            out["depth"].append(p.h.cpu())
            out["rain_in"].append(p.rain_in)
        return out if case["kind"] == "served" else {"depth": out["depth"]}
    z, n, h = _field(case, seed)
    f = _forcing(case, seed)
    dx, dev = case["dx"], z.device
    p = _Plain(z, n, h, dx, manning=f["manning"], half=_half_step(case), fixed=case["dt"] == "fixed",
               south=case["south_open"], **_fractions(case))
    w = _weights(case, seed) if case["weights"] else None
    if f["storm"] is not None:
        x = (torch.arange(case["cols"], dtype=torch.float64, device=dev) + 0.5) * dx
        y = ((torch.arange(case["rows"], dtype=torch.float64, device=dev) + 0.5) * dx)[:, None]

    def forcing(t):
        rain, ev, ql = 0.0, 0.0, 0.0
        if f["storm"] is not None:
            s = f["storm"]
            d2 = (x - (s["x0"] + s["vx"] * t)) ** 2 + (y - (s["y0"] + s["vy"] * t)) ** 2
            rain = s["peak"] / 3.6e6 * torch.exp(-d2 / (2.0 * s["sigma"] ** 2))
        elif f["rain"] is not None:
            v, every = f["rain"]
            if case["rain"] == "compat":
                rain = _compat(v, every, t) / (every * 1000.0)
            else:
                rain = v[int(t // every)] / 3.6e6 if t < every * len(v) else 0.0
            rain = float(rain)
        if w is not None:
            rain = rain * w
        if f["ev"] is not None:
            ev = float(_compat(f["ev"], 3600.0, t) / (3600.0 * 1000.0))
        if f["sources"] is not None:
            cells, q = f["sources"]
            ql = torch.zeros_like(z)
            rate = np.array([_compat(q[:, k], TABLE_DT, t) for k in range(cells.size)]) / dx ** 2
            ql.view(-1)[torch.from_numpy(cells.astype(np.int64)).to(dev)] = torch.from_numpy(rate).to(dev)
        return rain, ev, ql

    if case["dt"] == "fixed" and case["fresh"]:
        p.advance(10 ** 9, forcing, _t_end(case))
    else:
        p.advance(case["iters"], forcing)
    out = {"depth": p.h.cpu()}
    if case["read"] == "state":
        out.update(um=p.um.cpu(), vn=p.vn.cpu())
    elif case["read"] == "velocity":
        uu, vv = p.cell_velocity()
        out.update(uu=uu.cpu(), vv=vv.cpu())
    out.update(t=p.t, volume=float(p.h.sum()) * dx * dx, rain_in=p.rain_in, outflow=p.outflow)
    return out
