"""The work that users of this framework have it do, as timed cases.

Each case is one pass of a user's program between two looks at the result: a
driver advances a lattice by the steps between two outputs and takes the fields
out (the reference's drivers write density and velocity every few hundred
steps).  Sizes and physics are those of the repository's own configurations,
tests and benchmark (sc_lbm_b200/workloads.py): the 200 x 50 channel, the 256 x
256 droplet, the 400 x 306 contact-angle shelf, the 2048 x 1024 porous medium,
the mixed ensemble, the 4096 x 4096 spinodal lattice, and ragged lattices in
between.

Fields come back in host memory through the calls that a program uses: the
Python classes' download methods on small lattices, the C entry points into a
pinned buffer kept by the program on large ones.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import sc_lbm_b200 as sc
from sc_lbm_b200 import capi
from sc_lbm_b200 import workloads as W

PREC = {"fp64": sc.FP64, "fp32": sc.FP32_SHIFTED, "fp16": sc.FP16_SHIFTED}
SIZE = {"fp64": 8, "fp32": 4, "fp16": 2}


def listed():
    return [
        # the smallest lattice in the repository: a channel under a body force,
        # one component, ten thousand steps of it in a run; launches count
        dict(name="channel_200x50_fp64", kind="channel", nx=200, ny=50, prec="fp64", steps=1000),
        # a droplet in its own vapour (Laplace law), reference-exact storage
        dict(name="droplet_256_fp64", kind="droplet", nx=256, ny=256, prec="fp64", steps=1000),
        # the same physics as a C++ driver of the reference runs it: one call
        # per operator, every step
        dict(name="operators_256_fp64", kind="operators", nx=256, ny=256, prec="fp64", steps=200),
        # the drop-in classes' fused step, walls and a body force
        # (droplet in a channel), arrays owned by the fluid objects
        dict(name="fluids_520x260_fp64", kind="fluids", nx=520, ny=260, prec="fp64", steps=400),
        # eight contact angles at once: a batch of equal, mid-sized lattices
        dict(name="contact_8x400x306_fp32", kind="contact", nx=400, ny=306, prec="fp32", steps=200,
             members=8),
        # a mixed ensemble: uneven sizes, geometries and parameters in one batch
        dict(name="ensemble_64_fp32", kind="ensemble", nx=512, ny=256, prec="fp32", steps=100,
             members=64),
        # a ragged lattice (rows off every 16-byte boundary) whose program looks
        # at mass and momentum every ten steps
        dict(name="monitored_1021x763_fp32", kind="monitored", nx=1021, ny=763, prec="fp32", steps=100),
        # flow through a porous medium under a body force
        dict(name="drainage_2048x1024_fp32", kind="drainage", nx=2048, ny=1024, prec="fp32", steps=100),
        # a whole job on host data: populations in, steps, densities out
        dict(name="run_1024_fp32", kind="run", nx=1024, ny=1024, prec="fp32", steps=100),
        # the headline lattice in each storage form
        dict(name="spinodal_4096x2048_fp64", kind="spinodal", nx=4096, ny=2048, prec="fp64", steps=60),
        dict(name="spinodal_4096_fp32", kind="spinodal", nx=4096, ny=4096, prec="fp32", steps=100),
        dict(name="spinodal_4096_fp16", kind="spinodal", nx=4096, ny=4096, prec="fp16", steps=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel", "droplet", "operators", "fluids", "contact", "ensemble",
                       "monitored", "drainage", "run", "spinodal", "spinodal"])
    # reference-exact runs use FP64, production runs FP32; FP16 for throughput
    prec = rng.choice(["fp64", "fp32", "fp32"])
    if kind == "channel":
        return dict(kind=kind, nx=_log(rng, 64, 1500), ny=_log(rng, 32, 600), prec=prec,
                    steps=_log(rng, 100, 800))
    if kind == "droplet":
        return dict(kind=kind, nx=_log(rng, 64, 700), ny=_log(rng, 64, 700), prec=prec,
                    steps=_log(rng, 100, 1000))
    if kind in ("operators", "fluids"):
        return dict(kind=kind, nx=_log(rng, 64, 800), ny=_log(rng, 64, 500), prec="fp64",
                    steps=_log(rng, 40, 200))
    if kind == "contact":
        return dict(kind=kind, nx=_log(rng, 380, 520), ny=_log(rng, 280, 400), prec=prec,
                    steps=_log(rng, 50, 200), members=rng.randint(2, 9))
    if kind == "ensemble":
        return dict(kind=kind, nx=512, ny=256, prec=prec, steps=_log(rng, 20, 100),
                    members=_log(rng, 4, 64))
    if kind == "run":
        return dict(kind=kind, nx=_log(rng, 128, 1600), ny=_log(rng, 128, 1200), prec=prec,
                    steps=_log(rng, 20, 200))
    if kind == "drainage":
        # periodic rows of any width: also ones off a 16-byte boundary
        return dict(kind=kind, nx=_log(rng, 300, 2600), ny=_log(rng, 200, 1600), prec=prec,
                    steps=_log(rng, 10, 100))
    if kind == "monitored":
        return dict(kind=kind, nx=_log(rng, 200, 2400), ny=_log(rng, 150, 1500), prec=prec,
                    steps=10 * rng.randint(1, 10))
    prec = rng.choice(["fp64", "fp32", "fp32", "fp16"])
    wide = 16 * _log(rng, 24, 256) if rng.random() < 0.7 else _log(rng, 300, 4000)
    return dict(kind=kind, nx=wide, ny=_log(rng, 256, 2048 if prec == "fp64" else 4096), prec=prec,
                steps=_log(rng, 10, 60))


# ---------------------------------------------------------------------- physics
# one dict of plain data per lattice: what prepare() hands to the framework and
# exact() to the 64-bit evaluation
def _rows_columns(nx, ny):
    y, x = np.divmod(np.arange(nx * ny), nx)
    return x, y


def _phases(inside, rho_in, rho_out, seed, noise=1e-3):
    n = inside.size
    r1 = np.where(inside, rho_in, rho_out) * (1 + noise * (2 * W.uniform(seed, n) - 1))
    r2 = np.where(inside, rho_out, rho_in) * (1 + noise * (2 * W.uniform(seed + 1, n) - 1))
    return r1, r2


def _lattices(case, seed):
    """The lattices of a case: sizes, mask, parameters, initial densities."""
    kind, nx, ny = case["kind"], case["nx"], case["ny"]
    base = dict(nx=nx, ny=ny, tau=(1.0, 1.0), G=0.9, Gs=(0.0, 0.0), force=(None, None))
    ones = np.ones(nx * ny, np.int32)
    if kind == "channel":
        m = ones.reshape(ny, nx).copy()
        m[0] = m[-1] = 0
        rho = 1.0 + 1e-3 * (2 * W.uniform(seed, nx * ny) - 1)
        return [dict(base, mask=m.ravel(), force=(W.force_vec(1e-6, "x"), None), rho=(rho,))]
    if kind in ("droplet", "operators", "fluids", "run"):
        x, y = _rows_columns(nx, ny)
        r = (0.15 + 0.1 * W.uniform(seed + 5, 1)[0]) * min(nx, ny)
        inside = (x - nx / 2) ** 2 + (y - ny / 2) ** 2 <= r * r
        m, force, gs = ones, (None, None), (0.0, 0.0)
        if kind == "fluids":
            m = ones.reshape(ny, nx).copy()
            m[0] = m[-1] = 0
            m = m.ravel()
            force, gs = (W.force_vec(1e-6, "x"), W.force_vec(1e-6, "x")), (-0.1, 0.1)
        return [dict(base, mask=m, Gs=gs, force=force, rho=_phases(inside, 2.0, 0.06, seed))]
    if kind == "contact":
        out = []
        for k in range(case["members"]):
            gs = (-0.4, -0.3, -0.2, -0.1, 0.1, 0.2, 0.3, 0.4)[k % 8]
            g = sc.Geometry(nx, ny)
            g.add_rectangle(nx * 17 // 20, 20, nx // 2 - 1, ny // 2 - 1)
            x, y = _rows_columns(nx, ny)
            drop = (abs(x - nx // 2) < 30) & (abs(y - ny // 2 - 39) < 30)
            out.append(dict(base, mask=g.get_geom(), Gs=(-gs, gs),
                            rho=_phases(~drop, 2.0, 0.06, seed + 10 * k)))
        return out
    if kind == "ensemble":
        out = []
        for k in range(case["members"]):
            # sizes and fluid fractions of the repository's seeded ensemble;
            # its parameters from the part of their box that stays stable
            e = W.ensemble_draws(k)
            u = W.uniform(seed + 77 * k, 3)
            n = e["nx"] * e["ny"]
            disks = dict(e["disks"], porosity=max(0.6, e["phi"]), seed=seed + 7919 * k)
            out.append(dict(nx=e["nx"], ny=e["ny"], disks=disks, tau=(0.9 + 0.3 * u[0],) * 2, G=0.8 + 0.2 * u[1],
                            Gs=(0.1 * u[2], -0.1 * u[2]), force=(None, None),
                            rho=tuple(1.0 + 0.01 * (2 * W.uniform(seed + 3 * k + c, n) - 1)
                                      for c in range(2))))
        return out
    if kind in ("drainage", "monitored"):
        x, _ = _rows_columns(nx, ny)
        phi = 0.6 if kind == "drainage" else 0.75
        return [dict(base, disks=dict(porosity=phi, rmin=4, rmax=min(20, min(nx, ny) // 12),
                                      seed=seed, wall_rows=0, max_tries=20000, max_misses=300),
                     Gs=(-0.1, 0.1), force=(W.force_vec(1e-6, "x"), None),
                     rho=_phases(x < 0.3 * nx, 1.8, 0.1, seed))]
    # spinodal decomposition: seeded noise, written on the device
    return [dict(base, G=1.2, mask=ones, noise=((1.0, 0.01, seed), (1.0, 0.01, seed + 1)))]


def _params(L, ncomp=2):
    if "noise" in L:
        ref = tuple(c[0] for c in L["noise"])
    else:
        ref = tuple(float(r.mean()) for r in L["rho"])
    return sc.make_params(ncomp=ncomp, tau=L["tau"], g_fluid=(L["G"],) * 2, g_solid=L["Gs"],
                          rho_ref=(ref * 2)[:2], force=L["force"])


def _domain(L, prec, ncomp=2):
    mask = L.get("mask")
    if mask is None:
        mask = np.ones(L["nx"] * L["ny"], np.int32)
    d = sc.Domain(L["nx"], L["ny"], mask, _params(L, ncomp), PREC[prec])
    if "disks" in L:
        d.add_random_disks(**L["disks"])
        mask = d.download_mask()
    for k in range(ncomp):
        if "noise" in L:
            d.init_noise(k, *L["noise"][k])
        else:
            d.upload_f(k, W.populations(L["rho"][k], mask))
    return d


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def _dptr(t, at=0):
    return C.cast(C.c_void_p(t.data_ptr() + 8 * at), C.POINTER(C.c_double))


def prepare(case, seed):
    kind, prec = case["kind"], case["prec"]
    Ls = _lattices(case, seed)
    s = dict(kind=kind, steps=case["steps"])
    if kind in ("operators", "fluids"):
        L = Ls[0]
        g = sc.Geometry.from_mask(L["nx"], L["ny"], L["mask"])
        fluids = []
        for k in range(2):
            f = sc.Fluid(g, L["tau"][k])
            f.initialize_interactions(L["Gs"][k], L["G"])
            f.set("f", W.populations(L["rho"][k], L["mask"]))
            fluids.append(f)
        lbm = sc.LBM(g)
        lbm.compute_solid_surface_force(g, fluids[0], fluids[1], L["Gs"][0], L["Gs"][1])
        return dict(s, g=g, fluids=fluids, lbm=lbm, force=L["force"])
    if kind == "run":
        L = Ls[0]
        f = [torch.from_numpy(W.populations(r)).pin_memory() for r in L["rho"]]
        d = _domain(L, prec)
        n = L["nx"] * L["ny"]
        return dict(s, d=d, f=f, rho=[_pinned(n) for _ in range(2)])
    ncomp = 1 if kind == "channel" else 2
    doms = [_domain(L, prec, ncomp) for L in Ls]
    total = sum(d.N for d in doms)
    if kind in ("contact", "ensemble"):
        return dict(s, doms=doms, batch=sc.Batch(doms), rho=[_pinned(total) for _ in range(2)])
    return dict(s, d=doms[0], rho=[_pinned(total) for _ in range(ncomp)])


def _densities(s, doms):
    for k, out in enumerate(s["rho"]):
        at = 0
        for d in doms:
            capi.call("sclbm_domain_download_rho", d.handle, k, _dptr(out, at), d.N)
            at += d.N
    return list(s["rho"])


def run(s):
    kind, steps = s["kind"], s["steps"]
    if kind == "channel":
        # a validation run keeps the whole state
        s["d"].step(steps)
        return [s["d"].download_f(0)]
    if kind == "droplet":
        s["d"].step(steps)
        return [s["d"].download_f(0), s["d"].download_f(1)]
    if kind == "operators":
        g, lbm, (a, b) = s["g"], s["lbm"], s["fluids"]
        for _ in range(steps):
            a.compute_density()
            b.compute_density()
            lbm.compute_fluid_repulsive_interactions(g, a, b)
            lbm.compute_equilibrium_velocities(g, a, b)
            lbm.collide(a, b)
            lbm.stream(g, a, b)
        return [a.get("f"), b.get("f"), a.get("rho"), b.get("rho"), a.get("uex"), a.get("uey")]
    if kind == "fluids":
        g, lbm, (a, b) = s["g"], s["lbm"], s["fluids"]
        lbm.step(g, a, b, steps, s["force"][0], s["force"][1])
        return [a.get("f"), b.get("f")]
    if kind in ("contact", "ensemble"):
        s["batch"].step(steps)
        return _densities(s, s["doms"])
    if kind == "run":
        d, f, r = s["d"], s["f"], s["rho"]
        capi.call("sclbm_domain_run", d.handle, _dptr(f[0]), _dptr(f[1]), steps, _dptr(r[0]), _dptr(r[1]))
        return list(r)
    if kind == "monitored":
        seen = []
        for _ in range(steps // 10):
            s["d"].step(10)
            seen.append(s["d"].mass_momentum())
        return _densities(s, [s["d"]]) + [np.stack(seen)]
    s["d"].step(steps)
    return _densities(s, [s["d"]])


def work(case):
    """Bytes: the populations read once and written once in their storage form,
    the mask, the host input of a job, and the fields handed out.  Operations:
    one component's step takes about 170, the coupled two-component step about
    400 per node."""
    kind, steps, size = case["kind"], case["steps"], SIZE[case["prec"]]
    n = case["nx"] * case["ny"]
    if kind == "contact":
        n *= case["members"]
    if kind == "ensemble":
        n = sum(e["nx"] * e["ny"] for e in map(W.ensemble_draws, range(case["members"])))
    ncomp = 1 if kind == "channel" else 2
    out = 8 * ncomp * (9 if kind in ("channel", "droplet", "operators", "fluids") else 1)
    if kind == "run":
        out += 8 * 18
    return {"bytes": n * (18 * ncomp * size + 1 + out),
            "flops": float(n) * steps * (170 if ncomp == 1 else 400)}


# --------------------------------------------------------------- 64-bit evaluation
CX, CY = (0, 1, 0, -1, 0, 1, -1, -1, 1), (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
WEQ = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4


def _shift(a, i, sign):
    """a at the node sign * c_i away (periodic)"""
    out = a
    if CY[i]:
        out = torch.roll(out, -sign * CY[i], 0)
    if CX[i]:
        out = torch.roll(out, -sign * CX[i], 1)
    return out


class _Exact:
    """The step sequence of the reference's drivers on whole arrays."""

    def __init__(self, L, mask, rho, ncomp, dev):
        nx, ny = L["nx"], L["ny"]
        self.L, self.ncomp = L, ncomp
        self.fl = torch.from_numpy(np.asarray(mask).reshape(ny, nx)).to(dev) != 0
        self.flf = self.fl.double()
        self.solid = not bool(self.fl.all())
        self.f = []
        for k in range(ncomp):
            r = torch.from_numpy(np.asarray(rho[k]).reshape(ny, nx)).to(dev) / 9.0 * self.flf
            self.f.append([r.clone() for _ in range(9)])
        self.S = [torch.zeros_like(self.flf), torch.zeros_like(self.flf)]
        if self.solid:
            for i in range(1, 9):
                s = 1.0 - _shift(self.flf, i, 1)
                w = WEQ[i]
                self.S[0] += w * CX[i] * s
                self.S[1] += w * CY[i] * s
            self.from_fluid = [None] + [_shift(self.fl, i, -1) for i in range(1, 9)]
        self.ue = None

    @staticmethod
    def _feq(r, ux, uy):
        usq = 1.5 * (ux * ux + uy * uy)
        out = []
        for i in range(9):
            cu = CX[i] * ux + CY[i] * uy
            out.append(WEQ[i] * r * (1.0 + 3.0 * cu + 4.5 * cu * cu - usq))
        return out

    def step(self):
        L, f = self.L, self.f
        rho = [sum(c) for c in f]
        one = torch.ones_like(rho[0])
        safe = [torch.where(self.fl, r, one) for r in rho]
        j = [(sum(CX[i] * c[i] for i in range(1, 9) if CX[i]), sum(CY[i] * c[i] for i in range(1, 9) if CY[i]))
             for c in f]
        om = [1.0 / t for t in L["tau"]]
        if self.ncomp == 1:
            ue = [(j[0][0] / safe[0], j[0][1] / safe[0])]
        else:
            den = om[0] * safe[0] + om[1] * safe[1]
            uc = [(om[0] * j[0][a] + om[1] * j[1][a]) / den for a in range(2)]
            psi = [r * self.flf for r in rho]
            sums = [[torch.zeros_like(one), torch.zeros_like(one)] for _ in range(2)]
            for i in range(1, 9):
                for k in range(2):
                    p = _shift(psi[k], i, 1)
                    sums[k][0] += WEQ[i] * CX[i] * p
                    sums[k][1] += WEQ[i] * CY[i] * p
            ue = []
            for k in range(2):
                ue.append(tuple(uc[a] + (-L["G"] * psi[k] * sums[1 - k][a]) / om[k] / safe[k]
                                + (-L["Gs"][k] * self.S[a]) / om[k] for a in range(2)))
        self.rho, self.ue = rho, ue
        for k in range(self.ncomp):
            fe = self._feq(rho[k], *ue[k])
            F = L["force"][k]
            post = [((1.0 - om[k]) * f[k][i] + om[k] * fe[i] + (0.0 if F is None else float(F[i])))
                    for i in range(9)]
            out = []
            for i in range(9):
                v = _shift(post[i], i, -1)
                if self.solid:
                    if i:
                        v = torch.where(self.from_fluid[i], v, post[OPP[i]])
                    v = v * self.flf
                out.append(v)
            f[k] = out
        self.f = f

    def densities(self):
        return [sum(c).ravel() for c in self.f]

    def populations(self, k):
        return torch.stack(self.f[k]).ravel()

    def monitor(self):
        out = []
        for c in self.f:
            out += [float(sum(v.sum() for v in c)), float(sum(CX[i] * c[i].sum() for i in range(9))),
                    float(sum(CY[i] * c[i].sum() for i in range(9)))]
        return out + [0.0] * (7 - len(out))


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    n = case["nx"] * case["ny"]
    if n * steps > 2.2e9:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ncomp = 1 if kind == "channel" else 2
    runs = []
    for L in _lattices(case, seed):
        mask = L.get("mask")
        if "disks" in L:
            # the host packer of the reference's circles, on the host geometry
            g = sc.Geometry(L["nx"], L["ny"])
            g.add_random_disks(**L["disks"])
            mask = g.get_geom()
        if "noise" in L:
            rho = [c[0] * (1.0 + c[1] * (2.0 * W.uniform(c[2], L["nx"] * L["ny"]) - 1.0)) for c in L["noise"]]
        else:
            rho = L["rho"]
        runs.append(_Exact(L, mask, rho, ncomp, dev))
    seen = []
    for e in runs:
        for k in range(steps):
            e.step()
            if kind == "monitored" and k % 10 == 9:
                seen.append(e.monitor())
    e = runs[0]
    host = lambda t: t.cpu()  # noqa: E731
    if kind in ("channel", "droplet", "fluids"):
        return [host(e.populations(k)) for k in range(ncomp)]
    if kind == "operators":
        # rho and u_eq are those of the last step's collision (before streaming)
        return [host(e.populations(0)), host(e.populations(1))] + [host(r.ravel()) for r in e.rho] + \
            [host(u.ravel()) for u in e.ue[0]]
    out = [host(torch.cat([r.densities()[k] for r in runs])) for k in range(ncomp)]
    if kind == "monitored":
        # momentum starts at zero and stays near it beside the mass: no relative error
        out.append(None)
    return out
