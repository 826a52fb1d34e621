"""The work users of the engine have it do, as measurable cases.

A case is one program: it holds its simulation on the device as a job (or the
specs of a batch, or the requests of a served mix), and a pass is one whole
call of it -- the job back to step 0 (``Job.reset``), every time step, the
result read back.  Results keep the dtype the reference saves them in:
complex64 port DFTs and S-parameters for float32 runs, complex128 for float64.

Families (``kind``):

* ``slab2d``   2D TMz symmetric slab with rough faces (``workloads.slab2d``):
               the 400 x 200 benchmark slab in the float64 exact arithmetic the
               drop-in uses for float64 runs, the sizes of the served mix, a
               wide slab of a million cells.
* ``te2``      2D TE guide set up from a reference user dictionary
               (``refsetup.build_spec``), float32.
* ``strip3d``  3D silicon strip with rough sidewalls (``workloads.strip3d``):
               the 128 x 128 x 256 benchmark run, a small guide where a launch
               is most of a step, the float64 exact run, ragged sizes, the
               out-of-plane ('TM') source.
* ``rib3d``    the etched rib of the large single run (384 x 384 section, 15 nm,
               16-cell CPML) on a guide of 256 cells.
* ``scatter``  scattering loss: one frequency, whole-plane DFTs at two cuts, a
               20-cell CPML, permittivity grids without a material index.
* ``zwave``    wave impedance: the same solver with the per-step line probe.
* ``batch``    stochastic roughness realizations of uneven size with shared
               incident runs, submitted, advanced together and reduced to S21.
* ``served``   requests of the served mix (2D and 3D, each a rough and a smooth
               incident run) through the serving loop.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from oidt_b200 import batch, large, refsetup, scatter, serve, zwave
from oidt_b200 import workloads as W
from oidt_b200.engine import Engine
from oidt_b200.spec import DFT_COMPS, FIELDS, PSI

_ENGINE = None


def _engine() -> Engine:
    """One context per process, as in a user's program."""
    global _ENGINE
    if _ENGINE is None:
        _ENGINE = Engine(0)
    return _ENGINE


def listed():
    return [
        # the smallest calls: a 2D run is 80 000 cells and a few ms for 2000 steps
        dict(name="slab2d_f64_exact", kind="slab2d", nx=400, ny=200, steps=2000, nf=21, prec="f64", arith="exact"),
        # a 2D request of the served mix, on its own, odd sizes
        dict(name="slab2d_f32", kind="slab2d", nx=613, ny=227, steps=2500, nf=21, prec="f32", arith="fast"),
        # a wide 2D slab, a million cells: more tiles than the GPU holds at once
        dict(name="slab2d_wide_f32", kind="slab2d", nx=603, ny=1601, steps=2500, nf=21, prec="f32", arith="fast"),
        # a 2D TE run of a user dictionary
        dict(name="te2_f32", kind="te2", length_um=14.0, clad_wl=1.1, ppw=20, nf=31, prec="f32", arith="fast"),
        # the smallest 3D call: launches count as much as cells
        dict(name="strip3d_small_f32", kind="strip3d", nx=48, ny=40, nz=96, P=6, gap=3, port_gap=6, steps=600, nf=5,
             source="TE", prec="f32", arith="fast"),
        # the benchmark run: 4.2 M cells, 4000 steps
        dict(name="strip3d_f32", kind="strip3d", nx=128, ny=128, nz=256, P=10, gap=10, port_gap=20, steps=4000, nf=41,
             source="TE", prec="f32", arith="fast"),
        # the drop-in's float64 default, 'TM' source, odd sizes
        dict(name="strip3d_f64_exact", kind="strip3d", nx=97, ny=114, nz=187, P=10, gap=10, port_gap=20, steps=1200,
             nf=21, source="TM", prec="f64", arith="exact"),
        # the largest: the large run's cross-section, 38 M cells
        dict(name="rib3d_f32", kind="rib3d", nx=384, ny=384, nz=256, steps=1000, nf=5, prec="f32", arith="fast"),
        # a scattering-loss realization
        dict(name="scatter_f32", kind="scatter", length_um=5.0, ppw=20, flights=1.2, source="TM", prec="f32",
             arith="fast"),
        # a wave-impedance run (line probe after every step)
        dict(name="zwave_f32", kind="zwave", length_um=4.0, ppw=17, flights=1.0, source="TE", prec="f32",
             arith="fast"),
        # a set of roughness realizations, creation included
        dict(name="batch_f32", kind="batch", count=4, steps=2000, nf=41, draw=0),
        # requests of the served mix, creation included
        dict(name="served_f32", kind="served", n2d=6, n3d=2, steps=2000, nf=21, draw=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the families, sizes spread over their ranges."""
    kind = rng.choice(["slab2d", "slab2d", "te2", "strip3d", "strip3d", "strip3d", "scatter", "zwave", "rib3d",
                       "batch", "served"])
    arith = lambda p: "exact" if p == "f64" else "fast"  # noqa: E731
    if kind == "slab2d":
        prec = rng.choice(["f32", "f32", "f64"])
        nx = _log(rng, 200, 900)  # enough steps for the pulse to pass the second port
        return dict(kind=kind, nx=nx, ny=_log(rng, 120, 1601), steps=rng.randint(800, 1000) + 4 * nx,
                    nf=rng.choice([5, 21, 41]), prec=prec, arith=arith(prec))
    if kind == "te2":
        prec = rng.choice(["f32", "f32", "f64"])
        return dict(kind=kind, length_um=round(rng.uniform(8.0, 16.0), 2), clad_wl=round(rng.uniform(0.8, 1.6), 2),
                    ppw=rng.randint(14, 24), nf=rng.choice([11, 31]), prec=prec, arith=arith(prec))
    if kind == "strip3d":
        prec = rng.choice(["f32", "f32", "f32", "f64"])
        nx, ny = rng.randint(64, 160), rng.randint(64, 160)
        nz = _log(rng, 120, 384)
        # at most the benchmark run's cell updates (half of it in float64)
        most = 4.0e9 if prec == "f64" else 1.6e10
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, P=rng.choice([6, 8, 10, 12]), gap=rng.randint(4, 10),
                    port_gap=rng.randint(8, 20), steps=int(min(3000, max(600, most / (nx * ny * nz)))),
                    nf=rng.choice([5, 21, 41]), source=rng.choice(["TE", "TM"]), prec=prec, arith=arith(prec))
    if kind in ("scatter", "zwave"):
        return dict(kind=kind, length_um=round(rng.uniform(3.5, 6.0), 2), ppw=rng.randint(14, 21),
                    flights=round(rng.uniform(1.0, 1.3), 2), source=rng.choice(["TE", "TM"]), prec="f32", arith="fast")
    if kind == "rib3d":
        return dict(kind=kind, nx=rng.randint(200, 380), ny=rng.randint(200, 380), nz=rng.randint(180, 256),
                    steps=rng.randint(800, 1000), nf=5, prec="f32", arith="fast")
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 4), steps=rng.randint(1000, 1500), nf=rng.choice([21, 41]),
                    draw=rng.randint(1, 10 ** 6))
    return dict(kind=kind, n2d=rng.randint(2, 6), n3d=rng.randint(1, 2), steps=rng.randint(1000, 1500), nf=21,
                draw=rng.randint(1, 10 ** 6))


# ---------------------------------------------------------------------------
# Inputs: the specs a program builds before its calls
# ---------------------------------------------------------------------------
def _np(prec):
    return np.float64 if prec == "f64" else np.float32


_TE2 = dict(eps_rel_bg=1.444 ** 2, eps_rel_fg=3.477 ** 2, sgl_wg_height=0.3e-6, port1_length=2.0e-6,
            port2_length=2.0e-6, rough_std=15.0e-9, rough_acl=200.0e-9, rough_toggle=True, profile_number=0,
            source_type=2, source_amp=5.0, wave_packet_bw=0.5, gauss_pulse_deg=-6, f0=193.5e12, harmonics=1.0,
            num_flights=1.5, num_cpml=12, buffer_xhat=12, sim_type="s-param", auto_condition=False, num_lines=1,
            pitch=0.0, sparam_fmin=182.0e12, sparam_fmax=207.0e12, prof_dir="rough_profiles", output_dir="Results")


def _loss_cfg(case):
    return dict(sgl_wg_length=case["length_um"] * 1e-6, port1_length=1.0e-6, points_per_wl=case["ppw"],
                num_flights=case["flights"], source_condition=case["source"], rough_toggle=True)


def _spec(case, seed):
    kind = case["kind"]
    if kind == "slab2d":
        nx = case["nx"]
        return W.slab2d(nx=nx, ny=case["ny"], steps=case["steps"], nf=case["nf"], ports=(60, nx - 60), rough=True,
                        seed=seed, precision=_np(case["prec"]))
    if kind == "strip3d":
        return W.strip3d(nx=case["nx"], ny=case["ny"], nz=case["nz"], P=case["P"], src_gap=case["gap"],
                         port_gap=case["port_gap"], steps=case["steps"], nf=case["nf"], source=case["source"],
                         seed=seed, precision=_np(case["prec"]))
    if kind == "rib3d":
        return W.strip3d(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=15e-9, P=16, steps=case["steps"],
                         nf=case["nf"], core_x_nm=1000, core_y_nm=220, slab_y_nm=90, sigma_nm=10.0, lc_nm=50.0,
                         seed=seed, precision=_np(case["prec"]))
    if kind == "te2":
        u = dict(_TE2, sgl_wg_length=case["length_um"] * 1e-6, ny_clad_wl=case["clad_wl"], points_per_wl=case["ppw"],
                 sparam_num_freqs=case["nf"], precision=_np(case["prec"]))
        dv = refsetup.derive(u, "te2", "r")
        rng = np.random.default_rng(seed)
        prof = tuple(W.sidewall_profile(dv.p2 - dv.p1, float(dv.rstd), float(dv.racl), rng) for _ in range(2))
        return refsetup.build_spec(u, "te2", 0, "f", "r", profiles=prof)
    if kind == "scatter":
        cfg = scatter.config(**_loss_cfg(case))
        return scatter.build_spec(cfg, scatter.realization_profiles(cfg, 1, seed)[0])
    cfg = zwave.config(**_loss_cfg(case))
    return zwave.build_spec(cfg, scatter.realization_profiles(cfg, 1, seed)[0])


def _batch_set(case, seed):
    """Realizations of the batched stochastic set, cross-sections in {96, 112,
    128}, roughness by the seed."""
    cfgs = W.batch_configs(n=case["count"], master_seed=case["draw"], steps=case["steps"])
    for r, c in enumerate(cfgs):
        c["seed"] = seed * 64 + r
    return batch.realization_set(cfgs, nf=case["nf"])


def _served_mix(case, seed):
    """The first 2D and 3D requests of a served mix, roughness by the seed."""
    mix = W.serving_mix(rate_hz=20.0, duration_s=5.0, seed=case["draw"])
    left = {"2d": case["n2d"], "3d": case["n3d"]}
    out = []
    for t, kw in mix:
        if left[kw["kind"]] > 0:
            left[kw["kind"]] -= 1
            out.append((t, dict(kw, seed=kw["seed"] ^ seed, steps=case["steps"])))
    return out


def _served(case, seed):
    return serve.requests_from_mix(_served_mix(case, seed), nf=case["nf"], short_incident=True)


class _State:
    """A job a program keeps, with page-locked buffers for what it reads."""

    def __init__(self, case, seed):
        self.kind = case["kind"]
        self.case = case
        if self.kind == "batch":
            self.set = _batch_set(case, seed)
        elif self.kind == "served":
            self.seed = seed
            self.requests = _served(case, seed)
        else:
            spec = _spec(case, seed)
            self.job = _engine().submit(spec, arith=case["arith"])
            self.pinned = self.out = None
            if self.kind != "zwave":
                plane = spec.shape[:2] if spec.mode == "yee3d" else spec.shape[1:]
                shape = (spec.nf,) + tuple(plane)
                self.pinned = torch.empty(shape, dtype=torch.complex128, pin_memory=True)
                self.names = [(p, c) for p in (0, 1) for c in DFT_COMPS[spec.mode]]
                dt = np.complex64 if spec.precision == np.float32 else np.complex128
                self.out = {"%s%d" % (c, p + 1): np.zeros(shape, dtype=dt) for p, c in self.names}

    def __del__(self):
        job = getattr(self, "job", None)
        if job is not None:
            job.release()


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    if state.kind == "batch":
        _, res = batch.run_batched(_engine(), state.set)
        # the reference's S dtype for float32 runs; S11 is left out: its power is a difference of
        # nearly equal planes whose square root sits on the branch cut
        return {"%02d" % r: {k: s[k].astype(np.complex64) for k in ("S21", "P_inc")} for r, s in enumerate(res)}
    if state.kind == "served":
        res = serve.Server(_engine()).run(state.requests, realtime=False)
        return {"%02d" % r.rid: r.S["S21"].astype(np.complex64) for r in res}
    job = state.job
    job.reset()
    job.run().sync()
    if state.kind == "zwave":
        return zwave.records_from_job(job, zwave.config(**_loss_cfg(state.case)))
    buf = state.pinned.numpy()
    for p, c in state.names:
        out = state.out["%s%d" % (c, p + 1)]
        if out.dtype == np.complex128:
            job.dft(p, c, out=out)
        else:
            np.copyto(out, job.dft(p, c, out=buf), casting="same_kind")
    return state.out


# ---------------------------------------------------------------------------
# Work of one pass
# ---------------------------------------------------------------------------
def _run_work(shape, mode, P, steps, nf, esz, window):
    """Per step, every field read and written once and the dt/eps values read
    once, every CPML psi element read and written once; the port planes'
    samples folded in float64 into nf accumulators, written once at the end.
    FLOPs: 6 differences, 6 divisions, 6 subtractions/sums and 3 products per
    half-step in 3D (half of it in 2D) and 5 per psi element."""
    cells = float(np.prod(shape))
    psi = 0.0
    for _, axis in PSI[mode]:
        s = list(shape)
        s[axis] = P
        psi += 2.0 * float(np.prod(s))
    nfield, ncb = len(FIELDS[mode]), {"tm2": 1, "te2": 2, "yee3d": 3}[mode]
    per_cell = 36.0 if mode == "yee3d" else 12.0
    ncomp = len(DFT_COMPS[mode])
    dft = 2.0 * ncomp * window
    return (steps * (cells * (2 * nfield + ncb) + 2 * psi) * esz + dft * nf * 16.0,
            steps * (cells * per_cell + 5 * psi + 4.0 * dft * nf))


def _spec_sizes(case):
    """(shape, mode, P, steps, nf, bytes per value) of each run of a case."""
    kind = case["kind"]
    esz = 8 if case.get("prec") == "f64" else 4
    if kind == "slab2d":
        return [((case["nx"], case["ny"]), "tm2", 10, case["steps"], case["nf"], esz)]
    if kind == "strip3d":
        return [((case["nx"], case["ny"], case["nz"]), "yee3d", case["P"], case["steps"], case["nf"], esz)]
    if kind == "rib3d":
        return [((case["nx"], case["ny"], case["nz"]), "yee3d", 16, case["steps"], case["nf"], esz)]
    if kind == "te2":
        u = dict(_TE2, sgl_wg_length=case["length_um"] * 1e-6, ny_clad_wl=case["clad_wl"], points_per_wl=case["ppw"],
                 sparam_num_freqs=case["nf"], precision=_np(case["prec"]))
        dv = refsetup.derive(u, "te2", "r")
        return [((dv.nx, dv.ny), "te2", u["num_cpml"], dv.nt, case["nf"], esz)]
    if kind in ("scatter", "zwave"):
        cfg = scatter.config(**_loss_cfg(case)) if kind == "scatter" else zwave.config(**_loss_cfg(case))
        dv = scatter.derive(cfg)
        return [((dv.nx, dv.ny, dv.nz), "yee3d", cfg["num_cpml"], dv.nt, 1, esz)]
    if kind == "batch":
        cfgs = W.batch_configs(n=case["count"], master_seed=case["draw"], steps=case["steps"])
        runs = [((c["nx"], c["ny"], c["nz"]), "yee3d", 10, c["steps"], case["nf"], 4) for c in cfgs]
        sections = sorted({(c["nx"], c["ny"]) for c in cfgs})
        return runs + [(s + (batch.incident_length({}),), "yee3d", 10, case["steps"], case["nf"], 4)
                       for s in sections]
    runs = []
    for _, kw in _served_mix(case, 0):
        if kw["kind"] == "2d":
            shapes, mode = ((kw["nx"], kw["ny"]), (122, kw["ny"])), "tm2"
        else:
            shapes, mode = ((kw["nx"], kw["ny"], kw["nz"]), (kw["nx"], kw["ny"], batch.incident_length({}))), "yee3d"
        runs += [(s, mode, 10, kw["steps"], case["nf"], 4) for s in shapes]
    return runs


def work(case):
    total = [0.0, 0.0]
    for shape, mode, P, steps, nf, esz in _spec_sizes(case):
        window = (shape[0] - 2 * P) * (shape[1] - 2 * P) if mode == "yee3d" else shape[1] - 2 * P
        b, f = _run_work(shape, mode, P, steps, nf, esz, window)
        if case["kind"] == "zwave":
            b += 2.0 * steps * shape[0] * esz
        total[0] += b
        total[1] += f
    return {"bytes": total[0], "flops": total[1]}


# ---------------------------------------------------------------------------
# The same results in plain float64 torch
# ---------------------------------------------------------------------------
class _Plain:
    """Yee leapfrog with CPML, soft source, port DFTs and line probe over a
    spec's arrays, in float64 torch tensors.

    E_c gains dt/eps (D_a H_b - D_b H_a), H_c gains dt/mu (D_b E_a - D_a E_b)
    with (a, b) the axes after c: forward differences over kappa dx for E,
    backward for H, each difference convolved in the CPML slabs by
    psi = b psi + c diff / dx."""

    def __init__(self, spec, device):
        self.s, self.mode = spec, spec.mode
        self.nd = len(spec.shape)
        t64 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=device)  # noqa: E731
        self.t64 = t64
        self.F = {f: torch.zeros(spec.shape, dtype=torch.float64, device=device) for f in FIELDS[spec.mode]}
        self.cb = {k: t64(v) for k, v in spec.cb.items()}
        self.kd = {}
        for key, v in spec.kdx.items():
            sh = [1] * self.nd
            sh["xyz".index(key[0])] = -1
            self.kd[key] = t64(v).reshape(sh)
        self.lo, self.hi, self.P = spec.lim_lo, spec.lim_hi, spec.num_cpml
        coef = {n: t64(getattr(spec, n)) for n in ("be", "ce", "bh", "ch")}
        P = self.P
        flip = lambda v: torch.flip(v, (0,))  # noqa: E731
        # slab cells of an axis: (first, last, b, c) on the low and the high side
        self.slabs = {}
        for a in range(self.nd):
            b, e = self.lo[a], self.hi[a]
            sh = [1] * self.nd
            sh[a] = -1
            r = lambda v, sh=sh: v.reshape(sh)  # noqa: E731
            self.slabs[("e", a)] = [(b, b + P, r(flip(coef["be"])), r(flip(coef["ce"]))),
                                    (e - P, e, r(coef["be"]), r(coef["ce"]))]
            self.slabs[("h", a)] = [(b + 1, b + P, r(flip(coef["bh"][1:])), r(flip(coef["ch"][1:]))),
                                    (e - P + 1, e, r(coef["bh"][1:]), r(coef["ch"][1:]))] if P > 1 else []
        self.dx = float(spec.dx)
        self.plan = {"e": [self._plan("e", c) for c in range(3)], "h": [self._plan("h", c) for c in range(3)]}

    def _plan(self, half, c):
        """How component c is updated: its range, its two differences and
        their slabs; None where the solver has no such component."""
        name, other = ("E", "H") if half == "e" else ("H", "E")
        f = name + "XYZ"[c]
        if f not in self.F:
            return None
        rng = []
        for a in range(self.nd):
            inner = (a == c) if half == "e" else (a != c)
            if self.mode == "te2" and f == "EX":
                inner = False
            rng.append((self.lo[a] + (1 if inner else 0), self.hi[a]))
        sl = tuple(slice(*r) for r in rng)
        terms = []
        a, b = (c + 1) % 3, (c + 2) % 3
        for axis, src, sign in (((a, other + "XYZ"[b], 1.0), (b, other + "XYZ"[a], -1.0)) if half == "e" else
                                ((b, other + "XYZ"[a], 1.0), (a, other + "XYZ"[b], -1.0))):
            if axis >= self.nd or src not in self.F:
                continue
            up, down = list(sl), list(sl)
            lo, hi = rng[axis]
            (up if half == "e" else down)[axis] = slice(lo + 1, hi + 1) if half == "e" else slice(lo - 1, hi - 1)
            kd = self.kd["xyz"[axis] + half]
            ks = [slice(None)] * self.nd
            ks[axis] = slice(lo, hi)
            slabs = []
            for first, last, cb, cc in self.slabs[(half, axis)]:
                f0, f1 = max(first, lo), min(last, hi)
                cut, pos = [slice(None)] * self.nd, [slice(None)] * self.nd
                cut[axis], pos[axis] = slice(f0 - first, f1 - first), slice(f0 - lo, f1 - lo)
                shape = [r[1] - r[0] for r in rng]
                shape[axis] = f1 - f0
                psi = torch.zeros(shape, dtype=torch.float64, device=self.F[f].device)
                slabs.append((tuple(pos), cb[tuple(cut)], cc[tuple(cut)] / self.dx, psi))
            terms.append((src, tuple(up), tuple(down), 1.0 / kd[tuple(ks)], sign, slabs))
        coef = self.cb["xyz"[c]][sl] if half == "e" else float(self.s.db)
        return f, sl, terms, coef

    def _half(self, half, n):
        for plan in self.plan[half]:
            if plan is None:
                continue
            f, sl, terms, coef = plan
            total = None
            for src, up, down, rk, sign, slabs in terms:
                d = self.F[src][up] - self.F[src][down]
                g = d * rk
                for pos, b, c, psi in slabs:
                    psi.mul_(b).add_(c * d[pos])
                    g[pos] += psi
                total = g if total is None and sign > 0 else (-g if total is None else total.add_(g, alpha=sign))
            self.F[f][sl] += coef * total

    def _source(self, n):
        f = "%s%s" % ("EH"[self.s.src_field // 3], "XYZ"[self.s.src_field % 3])
        box = tuple(slice(self.s.src_lo[a], self.s.src_hi[a]) for a in range(self.nd))
        self.F[f][box] -= float(self.s.j_src[n])

    @staticmethod
    def _next(v, axis):
        """v at the next cell along ``axis`` (zeros past the end)."""
        z = torch.zeros_like(v.narrow(axis, 0, 1))
        return torch.cat([v.narrow(axis, 1, v.shape[axis] - 1), z], axis)

    def _ports(self):
        """Colocated port samples [2 ports][components] of the present state."""
        out = []
        for q in self.s.port_pos:
            F = self.F
            if self.mode == "tm2":
                out.append([F["EZ"][q], 0.5 * (F["HY"][q] + F["HY"][q + 1])])
            elif self.mode == "te2":
                h = F["HZ"][q] + F["HZ"][q + 1]
                out.append([0.5 * (F["EY"][q] + self._next(F["EY"][q], 0)), 0.25 * (h + self._next(h, 0))])
            else:
                hx, hy = F["HX"][:, :, q] + F["HX"][:, :, q + 1], F["HY"][:, :, q] + F["HY"][:, :, q + 1]
                ex, ey = F["EX"][:, :, q], F["EY"][:, :, q]
                out.append([0.5 * (ex + self._next(ex, 0)), 0.5 * (ey + self._next(ey, 1)),
                            0.25 * (hx + self._next(hx, 1)), 0.25 * (hy + self._next(hy, 0))])
        return out

    def run(self, probe=None, chunk=64):
        """(DFTs {name + port: [nf, plane]}, probe records or None)."""
        s = self.s
        comps = DFT_COMPS[self.mode]
        (i0, j0), (i1, j1) = s.win_lo, s.win_hi
        win = (slice(i0, i1), slice(j0, j1)) if self.nd == 3 else (slice(j0, j1),)
        shape = s.shape[:2] if self.nd == 3 else s.shape[1:]
        tw = [self.t64(a) for a in s.twiddles]
        rot = [torch.complex(tw[0], -tw[1]), torch.complex(tw[2], -tw[3])]
        dft = {"%s%d" % (c, p + 1): torch.zeros((s.nf,) + tuple(shape), dtype=torch.complex128, device=tw[0].device)
               for p in (0, 1) for c in comps}
        rec = {k: [] for k in dft}
        lines = {c: torch.zeros((s.nt, s.shape[0]), dtype=torch.float64, device=tw[0].device)
                 for c in ("ey", "ez", "hy", "hz")} if probe else None

        def fold(n0, n1):
            for k, v in rec.items():
                x = torch.stack(v).to(torch.complex128)
                r = rot[0 if k[0] == "e" else 1][:, n0:n1]
                y = (r @ x.reshape(len(v), -1)).reshape((s.nf,) + tuple(x.shape[1:]))
                dft[k][(slice(None),) + win] += y
                v.clear()

        first = 0
        for n in range(s.nt):
            self._half("e", n)
            if s.src_field < 3 or self.mode == "yee3d":
                self._source(n)  # 3D: E and H sources both land before the H update
            self._half("h", n)
            if self.mode == "te2":
                self._source(n)
            for p, planes in enumerate(self._ports()):
                for c, v in zip(comps, planes):
                    rec["%s%d" % (c, p + 1)].append(v[win].clone())
            if probe:
                y, z = probe
                F, m = self.F, self.hi[0]
                x0, x1 = slice(0, m), slice(1, m + 1)
                lines["ey"][n, :m] = 0.5 * (F["EY"][x0, y, z] + F["EY"][x0, y + 1, z])
                lines["ez"][n, :m] = 0.5 * (F["EZ"][x0, y, z] + F["EZ"][x0, y, z + 1])
                lines["hy"][n, :m] = 0.25 * (F["HY"][x0, y, z] + F["HY"][x1, y, z] + F["HY"][x0, y, z + 1] +
                                             F["HY"][x1, y, z + 1])
                lines["hz"][n, :m] = 0.25 * (F["HZ"][x0, y, z] + F["HZ"][x1, y, z] + F["HZ"][x0, y + 1, z] +
                                             F["HZ"][x1, y + 1, z])
            if n + 1 - first == chunk or n + 1 == s.nt:
                fold(first, n + 1)
                first = n + 1
        return dft, lines


def _power(spec, d, port):
    """Complex Poynting flux through a port over the spec's power window."""
    w = spec.meta["power_window"]
    c = [d["%s%d" % (n, port + 1)] for n in DFT_COMPS[spec.mode]]
    if spec.mode == "yee3d":
        (i0, i1), (j0, j1) = w
        s = 0.5 * (c[0] * c[3].conj() - c[1] * c[2].conj())
        return s[:, i0:i1, j0:j1].sum(dim=(1, 2))
    return (-0.5 * (c[0] * c[1].conj()))[:, w[0]:w[1]].sum(dim=1)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "served":
        return None  # sixteen whole runs
    if kind == "batch":
        roughs, keys, incidents = _batch_set(case, seed)
        p_inc = {k: _power(s, _Plain(s, dev).run()[0], 0) for k, s in incidents.items()}
        out = {}
        for r, (s, k) in enumerate(zip(roughs, keys)):
            p_tr = _power(s, _Plain(s, dev).run()[0], 1)
            out["%02d" % r] = {"S21": torch.sqrt(p_tr / p_inc[k]), "P_inc": p_inc[k]}
        return out
    spec = _spec(case, seed)
    dft, lines = _Plain(spec, dev).run(probe=spec.meta.get("probe"))
    if kind == "zwave":
        return {name: lines[c] for c, name in zwave.RECORDS[case["source"]]}
    return dft
