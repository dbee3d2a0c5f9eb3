"""The work whose time is measured: time steps of the implicit Monte Carlo engine as its users
run them, through the drop-in modules, the batched engine, the device loop and the adjoint.

A case of a time-stepping kind is a run from its initial state: `prepare` holds the problem (the
mesh, the material callables, the source definition) as a driver has it in hand, and `run` makes
the initial census and takes `steps` steps, so that every pass is the same work however often it
is made.  Launch shapes are the package's defaults: a driver that swaps its import tunes nothing.

`exact` replays the differentiable step's histories in 64 bits (plain torch, the same counter-based
random numbers); for the other kinds it gives the boundary energy in closed form, the remaining
outputs being sums over random histories that have no closed value.
"""
import math

import numpy as np
import torch

from radtranbook_b200 import (adjoint, batch, driver, imc1d, imc2d, imc2d_cf, mg_imc1d, mg_imc2d, problems)

C_LIGHT, A_RAD = 29.98, 0.01372

# Track segments per tracked history on each problem, measured over the runs below (for work()).
SEGMENTS = {"slab": 70.0, "pipe": 8.0, "pipe_cf": 7.5, "mg_pipe": 1.2, "mg_slab": 20.0, "mg_sphere": 4.0,
            "loop": 16.0, "batch": 12.0, "adjoint": 24.0}
# Operations of one segment: ten Philox rounds (60), the distances to the cell's faces, the move
# and the attenuation (about 60).
SEGMENT_OPS = 120


def listed():
    return [
        # the slab Marshak wave at the reference's statistics size: a few thousand particles, the
        # latency of a step's launches
        {"name": "slab 4k", "kind": "slab", "cells": 100, "particles": 4_000, "steps": 20, "host": True},
        # the slab Marshak wave at its full size (20k emission + 20k boundary particles a step)
        {"name": "slab 40k", "kind": "slab", "cells": 100, "particles": 40_000, "steps": 20, "host": False},
        # crooked pipe on the coarse mesh with the reference driver's NumPy callables: the
        # launch-bound size
        {"name": "pipe 20k", "kind": "pipe", "nr": 30, "nz": 105, "particles": 20_000, "steps": 20, "host": True},
        # a desktop-sized crooked pipe on the full mesh, NumPy callables
        {"name": "pipe 200k", "kind": "pipe", "nr": 60, "nz": 210, "particles": 200_000, "steps": 10, "host": True},
        # the headline workload: 2e6 source particles a step, census of 6.67e6, device materials
        {"name": "pipe 2M", "kind": "pipe", "nr": 60, "nz": 210, "particles": 2_000_000, "steps": 10, "host": False},
        # the same pipe with Carter-Forest transport
        {"name": "pipe_cf 500k", "kind": "pipe_cf", "nr": 60, "nz": 210, "particles": 500_000, "steps": 8, "host": False},
        # the multigroup crooked pipe, 'standard' preset (200k + 200k a step, census 1e6 growing)
        {"name": "mg_pipe 400k", "kind": "mg_pipe", "nr": 60, "nz": 210, "groups": 10, "particles": 400_000, "steps": 16,
         "host": False},
        # the multigroup Marshak wave, 200 cells x 10 groups, 1e6 particles a step
        {"name": "mg_slab 1M", "kind": "mg_slab", "particles": 1_000_000, "steps": 8, "host": False},
        # a multigroup sphere of the MG_IMC1D module
        {"name": "mg_sphere 30k", "kind": "mg_sphere", "cells": 50, "groups": 4, "particles": 30_000, "steps": 10,
         "host": True},
        # the crooked-pipe driver's time loop replayed on the device (one captured graph)
        {"name": "loop 20k", "kind": "loop", "nr": 30, "nz": 105, "particles": 20_000, "steps": 20},
        # a batch of 256 uneven slab instances, 5.8e6 source particles a step, three steps
        {"name": "batch 256", "kind": "batch", "instances": 256, "scale": 0.1, "steps": 3},
        # the differentiable step: deposition and its vector-Jacobian product, 128 x 128 random
        # opacity, 4e6 histories
        {"name": "adjoint 4M", "kind": "adjoint", "n": 128, "particles": 4_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["slab", "slab", "pipe", "pipe", "pipe", "pipe_cf", "mg_pipe", "mg_slab", "mg_sphere", "loop",
                       "batch", "adjoint"])
    if kind == "slab":
        return {"kind": kind, "cells": _log(rng, 20, 800), "particles": _log(rng, 1_000, 100_000),
                "steps": rng.randint(8, 20), "host": rng.random() < 0.5}
    if kind in ("pipe", "pipe_cf"):
        nr = rng.randint(16, 64)
        return {"kind": kind, "nr": nr, "nz": rng.randint(3 * nr, 4 * nr), "particles": _log(rng, 5_000, 1_800_000),
                "steps": rng.randint(4, 8), "host": rng.random() < 0.5}
    if kind == "mg_pipe":
        nr = rng.randint(16, 60)
        return {"kind": kind, "nr": nr, "nz": rng.randint(3 * nr, int(3.5 * nr)), "groups": rng.randint(2, 16),
                "particles": _log(rng, 10_000, 800_000), "steps": rng.randint(4, 12), "host": rng.random() < 0.25}
    if kind == "mg_slab":
        return {"kind": kind, "particles": _log(rng, 20_000, 1_000_000), "steps": rng.randint(3, 8),
                "host": rng.random() < 0.5}
    if kind == "mg_sphere":
        return {"kind": kind, "cells": rng.randint(20, 200), "groups": rng.randint(2, 16),
                "particles": _log(rng, 8_000, 200_000), "steps": rng.randint(4, 10), "host": rng.random() < 0.5}
    if kind == "loop":
        nr = rng.randint(16, 60)
        return {"kind": kind, "nr": nr, "nz": rng.randint(3 * nr, 4 * nr), "particles": _log(rng, 5_000, 100_000),
                "steps": 2 * rng.randint(4, 12)}
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(16, 300), "scale": math.exp(rng.uniform(math.log(0.01), math.log(0.08))),
                "steps": rng.randint(2, 4)}
    return {"kind": "adjoint", "n": rng.randint(33, 160), "particles": _log(rng, 50_000, 3_500_000)}


# ------------------------------------------------------------------ problems
def _marshak_slab(case):
    p = problems.marshak_slab(scale=case["particles"] / 40_000)
    n, L = case["cells"], 0.20
    e = np.linspace(0.0, L, n + 1)
    p.update(mesh=np.stack([e[:-1], e[1:]], 1), Tinit=np.full(n, 0.001), Tr_init=np.full(n, 0.001), source=np.zeros(n))
    return p


def _sphere(case):
    """A heated multigroup sphere: power-law opacity per group, a 1 keV surface source."""
    n, G = case["cells"], case["groups"]
    edges = np.logspace(-2, np.log10(20.0), G + 1)
    nu = 0.5 * (edges[:-1] + edges[1:])
    e = np.linspace(0.0, 1.0, n + 1)
    ops = [lambda T, k=3.0 * v ** -3: np.clip(k * np.power(T, -0.5), 0.05, 1e4) for v in nu]
    dev = [_group_opacity(3.0 * v ** -3) for v in nu]
    N = case["particles"] // 2
    return dict(mesh=np.stack([e[:-1], e[1:]], 1), energy_edges=edges, Tinit=np.full(n, 0.3), Tr_init=np.full(n, 0.3),
                sigma_host=ops, sigma_dev=dev, cv_host=lambda T: np.full_like(T, 0.3),
                cv_dev=problems.Constant(0.3), eos_host=lambda T: 0.3 * T, inv_eos_host=lambda e_: e_ / 0.3,
                eos_dev=problems.LinearEOS(0.3).eos, inv_eos_dev=problems.LinearEOS(0.3).inv_eos,
                Ntarget=N, Nboundary=case["particles"] - N, Nmax=2 * case["particles"], T_boundary=(0.0, 1.0), dt=0.005,
                source=np.zeros(n))


def _group_opacity(k):
    """A power-law group opacity on the device: clamp(k T^-1/2, 0.05, 1e4)."""
    return problems.device_callable(lambda T: torch.clamp(k * torch.pow(T, -0.5), min=0.05, max=1e4))


def _counts(p, particles, census_factor):
    """`particles` new particles a step, split 2:1 between emission and the boundary."""
    nb = particles // 3
    p.update(Ntarget=particles - nb, Nboundary=nb, Nmax=int(census_factor * particles))
    return p


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": dict(case), "kind": kind, "seed": 0x5EED0000 + 7919 * int(seed)}
    if kind == "slab":
        s["p"] = _marshak_slab(case)
    elif kind in ("pipe", "pipe_cf", "loop"):
        s["p"] = _counts(problems.crooked_pipe(nr=case["nr"], nz=case["nz"]), case["particles"], 3.335)
    elif kind == "mg_pipe":
        p = problems.mg_crooked_pipe(n_groups=case["groups"], nr=case["nr"], nz=case["nz"])
        n = case["particles"]
        p.update(Ntarget=n // 2, Nboundary=n - n // 2, Nmax=int(2.5 * n), Nmax_growth=n // 8, Nmax_final=int(12.5 * n))
        s["p"] = p
    elif kind == "mg_slab":
        s["p"] = problems.marshak_mg(scale=case["particles"] / 1_000_000)
    elif kind == "mg_sphere":
        s["p"] = _sphere(case)
    elif kind == "batch":
        spec = batch.uneven_slab_batch(n_inst=case["instances"], particle_scale=case["scale"])
        spec.seed = spec.seed ^ np.uint64(s["seed"])  # the same instances, other histories
        s["engine"] = batch.BatchEngine(spec)
        s["engine"].init()
        s["engine"].capture()
    if kind not in ("loop", "batch", "adjoint"):
        p = s["p"]
        two_d = kind not in ("slab", "mg_sphere")
        nbins = (case["nr"] * case["nz"] if "nr" in case else len(p["source"])) * case.get("groups", 10)
        room = int(1.15 * max(p["Nmax"] + case["steps"] * p.get("Nmax_growth", 0), 0)) + 2 * nbins + 4096
        dev = torch.device("cuda")
        s["census"] = {k: torch.zeros(room, dtype=torch.int32 if k == "cell" else torch.float32, device=dev)
                       for k in ("weight", "pos1", "dir1", "cell") + (("pos2", "dir2") if two_d else ())}
    if kind == "loop":
        # the loop's captured graph outlives its runs, as a driver that continues a run keeps it; the
        # state goes on from run to run, from where the work per step has nearly stopped growing
        p = s["p"]
        st = imc2d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"], p["eos_dev"],
                                   p["inv_eos_dev"], geometry="rz", seed=s["seed"])
        s["loop"] = driver.DeviceLoop(st, Ntarget=p["Ntarget"], Nboundary=p["Nboundary"], Nsource=0, Nmax=p["Nmax"],
                                      T_boundary=p["T_boundary"], sigma_a_func=p["sigma_dev"],
                                      inv_eos=p["inv_eos_dev"], cv=p["cv_dev"], source=p["source"],
                                      reflect=p["reflect"], geometry="rz", max_events=1_000_000,
                                      boundary_source_func=p["boundary_source_func"])
        s["loop"].run([p["dt"]] * 2000)
    if kind == "adjoint":
        n = case["n"]
        edges = np.linspace(0.0, 1.0, n + 1)
        setup = adjoint.AdjointSetup("xy", edges, edges, T=0.01, cv=0.1, face_T=(1.0, 0.0, 0.0, 0.0),
                                     reflect=(False, False, False, False), dt=0.02, n_boundary=case["particles"],
                                     seed=s["seed"])
        field = adjoint.gaussian_random_field(n, seed=0xAD50 + int(seed))
        s["problem"] = adjoint.AdjointProblem(setup)
        dev = s["problem"].device
        s["sigma"] = torch.as_tensor(np.exp(field).T.reshape(-1).copy(), device=dev).requires_grad_(True)
        s["cot"] = torch.as_tensor(adjoint.unit_cotangent(n * n, seed=0xC07A + int(seed)), device=dev)
    return s


# ------------------------------------------------------------------ one pass
def _out(s, st, info):
    """What a driver reads after a step: the material state, the ledger, the event counts, and the
    census, copied into the driver's own arrays (their unused end zeroed)."""
    te = info["profiling"]["transport_events"]
    bank = st._engine.bank
    for k, keep in s["census"].items():
        keep[:bank.size].copy_(bank.view(k))
        keep[bank.size:].zero_()
    return {"T": st.temperature, "Tr": st.radiation_temperature, "e": st.internal_energy,
            "N_particles": int(info["N_particles"]), "events": int(te["total"]),
            "crossings": int(te["boundary_crossings"]), "transported": int(te["n_particles_transported"]),
            "total_energy": float(info["total_energy"]), "boundary_emission": float(info["boundary_emission"]),
            "boundary_loss": float(info["boundary_loss"]),
            "census": s["census"]}


def run(s):
    kind = s["kind"]
    if kind == "adjoint":
        s["sigma"].grad = None
        dep = adjoint.deposition(s["sigma"], s["problem"])
        dep.backward(s["cot"])
        return {"dep": dep.detach(), "grad": s["sigma"].grad}
    if kind == "batch":
        eng = s["engine"]
        eng.init()
        eng.step(s["case"]["steps"])
        return {"T": eng.s["T"], "Tr": eng.s["tr"], "e": eng.s["e"], "ledger": eng.s["ledger"],
                "n_census": eng.s["n_census"], "stats": eng.s["stats"]}
    p, case = s["p"], s["case"]
    n = case["steps"]
    if kind == "loop":
        res = s["loop"].run([p["dt"]] * n)
        st = s["loop"].state
        te = [q["transport_events"] for q in res["steps"]]
        return {"T": st.temperature, "Tr": st.radiation_temperature, "e": st.internal_energy,
                "events": [int(q["total"]) for q in te][-1], "N_particles": int(res["steps"][-1]["N_particles"])}
    h = "host" if case["host"] else "dev"
    sig, cv, eos, inv = p["sigma_" + h], p["cv_" + h], p["eos_" + h], p["inv_eos_" + h]
    if kind == "slab":
        st = imc1d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["mesh"], eos, inv, seed=s["seed"])
        for _ in range(n):
            st, info = imc1d.step(st, p["Ntarget"], p["Nboundary"], 0, p["Nmax"], p["T_boundary"], p["dt"], p["mesh"],
                                  sig, inv, cv, p["source"])
    elif kind in ("pipe", "pipe_cf"):
        mod = imc2d if kind == "pipe" else imc2d_cf
        st = mod.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"], eos, inv,
                                 geometry="rz", seed=s["seed"])
        for _ in range(n):
            st, info = mod.step(st, p["Ntarget"], p["Nboundary"], 0, p["Nmax"], p["T_boundary"], p["dt"], p["edges1"],
                                p["edges2"], sig, inv, cv, p["source"], reflect=p["reflect"], geometry="rz",
                                boundary_source_func=p["boundary_source_func"])
    elif kind == "mg_pipe":
        st = mg_imc2d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"],
                                      p["energy_edges"], eos, inv, T_emit_floor=p["T_emit_floor"], geometry="rz",
                                      seed=s["seed"])
        dt, nmax = p["dt_initial"], p["Nmax"]
        for _ in range(n):
            st, info = mg_imc2d.step(st, p["Ntarget"], p["Nboundary"], 0, nmax, p["T_boundary"], dt, p["edges1"],
                                     p["edges2"], p["energy_edges"], sig, inv, cv, p["source"], reflect=p["reflect"],
                                     geometry="rz", boundary_source_func=p["boundary_source_func"],
                                     T_emit_floor=p["T_emit_floor"])
            dt, nmax = min(dt * p["dt_growth"], p["dt_max"]), min(nmax + p["Nmax_growth"], p["Nmax_final"])
    elif kind == "mg_slab":
        st = mg_imc2d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"],
                                      p["energy_edges"], eos, inv, geometry="xy", seed=s["seed"])
        for _ in range(n):
            st, info = mg_imc2d.step(st, p["Ntarget"], p["Nboundary"], 0, p["Nmax"], p["T_boundary"], p["dt"],
                                     p["edges1"], p["edges2"], p["energy_edges"], sig, inv, cv, p["source"],
                                     reflect=p["reflect"], geometry="xy")
    else:
        st = mg_imc1d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["mesh"], p["energy_edges"], eos, inv,
                                      seed=s["seed"])
        for _ in range(n):
            st, info = mg_imc1d.step(st, p["Ntarget"], p["Nboundary"], 0, p["Nmax"], p["T_boundary"], p["dt"],
                                     p["mesh"], p["energy_edges"], sig, inv, cv, p["source"],
                                     conserve_comb_energy=False)
    return _out(s, st, info)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Each history's record (28 bytes in 2-D, 20 in 1-D, 4 more with groups) read once and written
    once per step by the tracking and once by the comb, and the operations of its segments."""
    kind = case["kind"]
    if kind == "adjoint":
        seg = case["particles"] * SEGMENTS[kind]
        return {"bytes": 8.0 * 3 * case["n"] ** 2, "flops": 3.0 * seg * SEGMENT_OPS}
    if kind == "batch":
        src = case["instances"] * case["scale"] * 2.15e5  # the mean of 10^U[4, 6]
        hist = 2.5 * src * case["steps"]  # the census grows over these first steps
        return {"bytes": 3 * 20.0 * hist, "flops": hist * SEGMENTS[kind] * SEGMENT_OPS}
    n = case["particles"]
    census = {"slab": 2.0, "mg_slab": 1.33, "mg_sphere": 2.0, "mg_pipe": 2.5}.get(kind, 3.335) * n
    hist = sum(min(census, (k + 0.67) * n) + n for k in range(case["steps"]))
    rec = (20 if kind in ("slab", "mg_sphere") else 28) + (4 if kind.startswith("mg") else 0)
    return {"bytes": 3.0 * rec * hist, "flops": hist * SEGMENTS[kind] * SEGMENT_OPS}


# ------------------------------------------------------------------ values in 64 bits
M32 = 0xFFFFFFFF


def _philox(i, block, step, tag, key):
    """Philox-4x32-10 (Salmon et al., SC'11) of the counters (i, block, step, tag), as int64 words."""
    c = [i, block, torch.full_like(i, step), torch.full_like(i, tag)]
    k0, k1 = key & M32, (key >> 32) & M32
    for r in range(10):
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # 64-bit products (wrapped: the low words are exact)
        c = [((b >> 32) & M32) ^ c[1] ^ k0, b & M32, ((a >> 32) & M32) ^ c[3] ^ k1, a & M32]
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return [((x >> 9) * 2 + 1).double() * 2.0 ** -24 for x in c]


class _Step64:
    """The differentiable XY step in 64 bits: boundary histories from x = 0, effective scatter,
    implicit capture, and the derivative of cot . dep by the path-length and likelihood-ratio terms."""

    def __init__(self, case, seed, dev):
        n = self.n = case["n"]
        self.N, self.key, self.dev = case["particles"], 0x5EED0000 + 7919 * int(seed), dev
        T, cv, dt = 0.01, 0.1, 0.02
        g = adjoint_field(n, 0xAD50 + int(seed))
        self.sigma = torch.as_tensor(np.exp(g).T.reshape(-1).copy(), device=dev)
        f = 1.0 / (1.0 + 4.0 * A_RAD * T ** 3 / cv * self.sigma * C_LIGHT * dt)
        self.f, self.sa, self.ss = f, self.sigma * f, self.sigma * (1.0 - f)
        self.vol = 1.0 / n ** 2
        self.edges = torch.linspace(0.0, 1.0, n + 1, dtype=torch.float64, device=dev)
        self.dt = dt
        self.w0 = A_RAD * C_LIGHT / 4.0 * dt / self.N

    def births(self, lo, hi):
        i = torch.arange(lo, hi, device=self.dev)
        z = torch.zeros_like(i)
        a = _philox(i, z, 0, 0x20000000, self.key)
        b = _philox(i, z + 1, 0, 0x20000000, self.key)
        j = torch.clamp((a[0] * self.n).ceil().long() - 1, 0, self.n - 1)
        y = self.edges[j] + a[1] * (self.edges[j + 1] - self.edges[j])
        u = a[2].sqrt()
        v = (1.0 - u * u).clamp(min=0.0).sqrt() * torch.cos(2.0 * math.pi * a[3])
        return dict(id=i, ev=z, x=torch.zeros_like(y), y=y, u=u, v=v, w=torch.full_like(y, self.w0),
                    left=(self.dt - b[0] * self.dt) * C_LIGHT, i=z.clone(), j=j, k=i - lo)

    def track(self, lo, hi, segment):
        """Follows histories lo..hi; calls segment(h, c, d, wn, scatter) for every segment."""
        h = self.births(lo, hi)
        n, E, floor = self.n, self.edges, 1e-10 * self.w0
        while h["id"].numel():
            c = h["i"] + n * h["j"]
            r = _philox(h["id"], h["ev"], 0, 0x10000000, self.key)
            x, y, u, v = h["x"], h["y"], h["u"], h["v"]
            big = torch.full_like(x, 1e30)
            sx = torch.where(u > 0, (E[h["i"] + 1] - x) / u, torch.where(u < 0, (E[h["i"]] - x) / u, big)).clamp(min=0)
            sy = torch.where(v > 0, (E[h["j"] + 1] - y) / v, torch.where(v < 0, (E[h["j"]] - y) / v, big)).clamp(min=0)
            sb = torch.minimum(sx, sy)
            ss = self.ss[c]
            ds = torch.where(ss > 1e-12, -r[0].log() / ss, big)
            census = h["left"] < torch.minimum(sb, ds)
            scatter = ~census & (ds < sb)
            cross = ~census & ~scatter
            d = torch.where(census, h["left"], torch.minimum(sb, ds))
            wn = h["w"] * torch.exp(-self.sa[c] * d)
            segment(h, c, d, wn, scatter)
            inx = cross & (sx <= sy)
            iny = cross & ~inx
            uz = 2.0 * r[1] - 1.0
            rxy = (1.0 - uz * uz).clamp(min=0.0).sqrt()
            i2 = h["i"] + torch.where(inx, torch.where(u > 0, 1, -1), 0)
            j2 = h["j"] + torch.where(iny, torch.where(v > 0, 1, -1), 0)
            x2 = torch.where(inx, E[torch.where(u > 0, h["i"] + 1, h["i"])], x + u * d)
            y2 = torch.where(iny, E[torch.where(v > 0, h["j"] + 1, h["j"])], y + v * d)
            u2 = torch.where(scatter, rxy * torch.cos(2.0 * math.pi * r[2]), u)
            v2 = torch.where(scatter, rxy * torch.sin(2.0 * math.pi * r[2]), v)
            keep = ~census & (wn > floor) & (i2 >= 0) & (i2 < n) & (j2 >= 0) & (j2 < n)
            h = {k: t[keep] for k, t in dict(id=h["id"], ev=h["ev"] + 1, x=x2, y=y2, u=u2, v=v2, w=wn,
                                             left=h["left"] - d, i=i2, j=j2, k=h["k"]).items()}

    def values(self, cot):
        dep = torch.zeros(self.n * self.n, dtype=torch.float64, device=self.dev)
        grad = torch.zeros_like(dep)
        a = cot / self.vol
        part = 1_000_000
        for lo in range(0, self.N, part):
            hi = min(lo + part, self.N)
            score = torch.zeros(hi - lo, dtype=torch.float64, device=self.dev)
            run_ = torch.zeros_like(score)

            def first(h, c, d, wn, scatter):
                dep.index_add_(0, c, h["w"] - wn)
                score[h["k"]] += a[c] * (h["w"] - wn)

            def second(h, c, d, wn, scatter):
                k = h["k"]
                before = run_[k]
                after = before + a[c] * (h["w"] - wn)
                run_[k] = after
                total = score[k]
                path = d * (a[c] * wn + after - total)
                f2 = self.f[c] ** 2
                rest = total - before
                ratio = torch.where(scatter, rest / self.ss[c], torch.zeros_like(rest)) - rest * d
                grad.index_add_(0, c, f2 * path + (1.0 - f2) * torch.where(self.ss[c] > 1e-12, ratio, 0.0))

            self.track(lo, hi, first)
            self.track(lo, hi, second)
        return dep / self.vol, grad


def _normals(n, key, tag):
    """Standard normals by Box-Muller on Philox uniforms, counter (i, 0, 0, tag)."""
    i = torch.arange((n + 1) // 2)
    u = _philox(i, torch.zeros_like(i), 0, tag, key)
    r, t = (-2.0 * u[0].log()).sqrt().numpy(), (2.0 * math.pi * u[1]).numpy()
    return np.stack([r * np.cos(t), r * np.sin(t)], 1).reshape(-1)[:n]


def adjoint_field(n, key):
    """The log-opacity field: stationary Gaussian of mean ln 50, unit variance and squared-exponential
    covariance of length 0.1 on the unit square, by circulant embedding (Dietrich & Newsam 1997)."""
    m = 2 * n
    k = np.arange(m)
    r = np.minimum(k, m - k) * (1.0 / n)
    lam = np.maximum(np.real(np.fft.fft2(np.exp(-(r[:, None] ** 2 + r[None, :] ** 2) / (2.0 * 0.1 ** 2)))), 0.0)
    z = _normals(2 * m * m, key, 0x71000000).reshape(2, m, m)
    return math.log(50.0) + np.real(np.fft.fft2((z[0] + 1j * z[1]) * np.sqrt(lam / (m * m))))[:n, :n]


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        n = case["n"]
        cot = _normals(n * n, 0xC07A + int(seed), 0x72000000)
        cot = torch.as_tensor(cot / np.linalg.norm(cot), device=dev)
        dep, grad = _Step64(case, seed, dev).values(cot)
        return {"dep": dep, "grad": grad}
    if kind in ("batch", "loop"):
        return None
    # a c T^4 / 4 times the face's area and the last step's length
    if kind == "slab":
        e = A_RAD * C_LIGHT / 4.0 * 0.01
    elif kind == "mg_slab":
        e = A_RAD * C_LIGHT / 4.0 * 0.005
    elif kind == "mg_sphere":
        e = A_RAD * C_LIGHT / 4.0 * 4.0 * math.pi * 0.005
    else:
        dt = 0.01 if kind != "mg_pipe" else 1e-4
        for _ in range(case["steps"] - 1 if kind == "mg_pipe" else 0):
            dt = min(dt * 1.1, 0.01)
        r = np.linspace(0.0, 2.0, case["nr"] + 1)
        lit = 0.5 * (r[:-1] + r[1:]) < 0.5
        e = A_RAD * C_LIGHT * 0.5 ** 4 / 4.0 * math.pi * float(np.sum((r[1:] ** 2 - r[:-1] ** 2)[lit])) * dt
    return {"boundary_emission": e}
