"""Cases that time the model time step through the package's public entry points.

A case is a dict of plain values; `prepare` builds the handle a program keeps (a PlanktonModel with
its PlanktonSimulation, a PlanktonBatch, or the device fields of one advection call) and `run` is one
pass of that program: an update! of `steps` time steps followed by the read-back of what the program
records, into page-locked buffers it keeps. update! indexes its forcing by the step of the call
(time_offset), so a pass can be repeated and the model goes on from where the last pass left it.

A Float32 model's results cross the boundary as Float64 arrays; the program records them as Float32.
`exact` restates the time step in Float64 torch, independent of this package's kernels.
"""
import ctypes as ct
import math
import os
import sys
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "planktonindividuals.jl_b200"))

from PlanktonIndividuals import _abi, _lib  # noqa: E402
from PlanktonIndividuals import (GPU, Bounded, CarbonMode, Member, Periodic, PlanktonBatch, PlanktonModel,  # noqa: E402
                                 PlanktonSimulation, QuotaMode, RectilinearGrid, phyto_setup, set_bc_b, tracer_names,
                                 update_b, update_bgc_params, update_phyt_params)
from PlanktonIndividuals._native import make_grid_struct  # noqa: E402
from PlanktonIndividuals.grids import fill_halo_tracer  # noqa: E402
from PlanktonIndividuals.init import empty_individuals  # noqa: E402

NTR = _abi.NTRACERS
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # one 0D water parcel with the default population (2^10 of 8192 slots): the smallest model
        # a user runs, four hours at one-minute steps; launches and latency
        dict(name="parcel_f32", kind="steps", ft="f32", nx=1, ny=1, nz=1, nsp=1, n=1024, cap=8, steps=240),
        # the 2D double-gyre model (128 x 128, 16,384 individuals) in either precision
        dict(name="gyre_f64", kind="steps", ft="f64", nx=128, ny=128, nz=1, nsp=1, n=16384, cap=4, steps=120),
        dict(name="gyre_f32", kind="steps", ft="f32", nx=128, ny=128, nz=1, nsp=1, n=16384, cap=4, steps=240),
        # the flagship: 256 x 256 x 64 cells, 2 x 2,097,152 individuals, two hours at 30 s with an
        # hourly velocity refresh, tracers and light recorded at the end
        dict(name="ocean_f32", kind="steps", ft="f32", nx=256, ny=256, nz=64, nsp=2, n=2097152, cap=2, steps=240,
             inds=False),
        # the same density in Float64 on a 128 x 128 x 64 domain
        dict(name="ocean_f64", kind="steps", ft="f64", nx=128, ny=128, nz=64, nsp=2, n=524288, cap=2, steps=30,
             inds=False),
        # a ragged coastal domain: Bounded x and y, land, tracer and individual diffusion, flux
        # boundary conditions
        dict(name="shelf_f32", kind="steps", ft="f32", nx=117, ny=93, nz=31, nsp=2, n=60000, cap=2, steps=120,
             inds=False, shelf=True),
        # CarbonMode, 64 x 64 x 32 with 2 x 50,000 individuals
        dict(name="carbon_f64", kind="steps", ft="f64", nx=64, ny=64, nz=32, nsp=2, n=50000, cap=2, steps=60,
             mode="carbon"),
        # an ensemble of uneven 3D members and an ensemble of 0D parcels, each advanced as one batch
        dict(name="ensemble_f32", kind="batch", ft="f32", nx=0, ny=0, nz=0, nsp=1, n=0, cap=2, steps=60, members=8,
             inds=False),
        dict(name="parcels_f32", kind="batch", ft="f32", nx=1, ny=1, nz=1, nsp=1, n=0, cap=8, steps=480, members=64),
        # coupled to a host ocean model: every step uploads its velocity, light and temperature from
        # page-locked Float32 arrays and reads the population back
        dict(name="coupled_f32", kind="coupled", ft="f32", nx=128, ny=128, nz=32, nsp=2, n=262144, cap=2, steps=12,
             inds=False),
        # the advection tendency of one field in the caller's own device arrays, near the entry
        # point's size limit
        dict(name="field_f64", kind="field", ft="f64", nx=124, ny=124, nz=28, shelf=False),
        # frequent output: a few steps, then every tracer and every individual is recorded
        dict(name="record_f32", kind="steps", ft="f32", nx=96, ny=80, nz=24, nsp=2, n=100000, cap=2, steps=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["parcel", "gyre", "ocean", "shelf", "carbon", "ensemble", "parcels", "coupled", "record", "field"])
    ft = rng.choice(["f32", "f32", "f64"])
    if kind == "parcel":
        return dict(kind="steps", ft=ft, nx=1, ny=1, nz=1, nsp=rng.choice([1, 2]), n=_log(rng, 200, 8000), cap=8,
                    steps=rng.randint(60, 240))
    if kind == "gyre":
        return dict(kind="steps", ft=ft, nx=_log(rng, 16, 300), ny=_log(rng, 16, 300), nz=1, nsp=rng.choice([1, 2, 3]),
                    n=_log(rng, 1000, 100000), cap=4, steps=rng.randint(40, 120))
    if kind in ("ocean", "record"):
        nx, ny, nz = _log(rng, 24, 240), _log(rng, 24, 240), _log(rng, 6, 60)
        return dict(kind="steps", ft=ft, nx=nx, ny=ny, nz=nz, nsp=rng.choice([1, 2, 4]), n=_log(rng, 5000, 500000),
                    cap=2, steps=rng.randint(2, 8) if kind == "record" else rng.randint(20, 60), inds=kind == "record")
    if kind == "shelf":
        return dict(kind="steps", ft=ft, nx=_log(rng, 20, 130), ny=_log(rng, 20, 130), nz=_log(rng, 5, 35), nsp=rng.choice([1, 2]),
                    n=_log(rng, 2000, 80000), cap=2, steps=rng.randint(20, 80), shelf=True)
    if kind == "carbon":
        return dict(kind="steps", ft="f64", nx=_log(rng, 12, 90), ny=_log(rng, 12, 90), nz=_log(rng, 4, 40),
                    nsp=rng.choice([1, 2]), n=_log(rng, 2000, 80000), cap=2, steps=rng.randint(20, 60), mode="carbon")
    if kind == "ensemble":
        return dict(kind="batch", ft="f32", nx=0, ny=0, nz=0, nsp=1, n=0, cap=2, steps=rng.randint(20, 60),
                    members=rng.randint(2, 10), inds=False)
    if kind == "parcels":
        return dict(kind="batch", ft="f32", nx=1, ny=1, nz=1, nsp=1, n=0, cap=8, steps=rng.randint(200, 480),
                    members=_log(rng, 8, 64))
    if kind == "coupled":
        return dict(kind="coupled", ft="f32", nx=_log(rng, 24, 160), ny=_log(rng, 24, 160), nz=_log(rng, 6, 48),
                    nsp=rng.choice([1, 2]), n=_log(rng, 5000, 300000), cap=2, steps=rng.randint(4, 16), inds=False)
    # the advection tendency of one tracer field from the caller's own device arrays
    nx, ny = _log(rng, 24, 180), _log(rng, 24, 180)
    nz = max(4, min(60, (1 << 19) // ((nx + 4) * (ny + 4)) - 4))
    return dict(kind="field", ft="f64", nx=nx, ny=ny, nz=_log(rng, 4, nz), shelf=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------

INIT = dict(DIC=20.0, NH4=0.5, NO3=0.8, PO4=0.10, DFe=1.0e-6, DOC=10.0, DON=0.1, DOP=0.05, PFe_inorg=1.0e-7,
            POC=0.02, PON=3.0e-3, POP=2.0e-4, PFe_bio=1.0e-7, Dust=1.0e-8)


def _f(a):
    """torch (z, y, x) to the reference's column-major (x, y, z) array."""
    return a.detach().cpu().numpy().transpose()


def _velocity(grid, seed, snap, rms=0.05, modes=12):
    """Divergence-free C-grid velocity from random Fourier modes, as (u, v, w) in (z, y, x) order;
    no flow through a Bounded face."""
    Nx, Ny, Nz = grid.Nx, grid.Ny, grid.Nz
    bx, by = grid.topo[0] == Bounded.code, grid.topo[1] == Bounded.code
    r = np.random.default_rng([seed, 77, snap])
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
    pos = lambda n, half: np.arange(n + (0 if half else 1)) + (0.5 if half else 0.0)  # noqa: E731

    def ax(k, p, N, bounded, ph):
        return np.sin(np.pi * np.outer(k, p) / N) if bounded else np.cos(2 * np.pi * np.outer(k, p) / N + ph[:, None])

    def potential(comp):
        kx, ky, kz = r.integers(1, max(2, Nx // 8) + 1, modes), r.integers(1, max(2, Ny // 8) + 1, modes), r.integers(1, 4, modes)
        amp = np.hypot(kx, ky) ** (-11.0 / 6.0) * r.standard_normal(modes) * (1.0 if comp == 2 else 0.3)
        px, py = r.uniform(0, 2 * np.pi, modes), r.uniform(0, 2 * np.pi, modes)
        X, Y = ax(kx, pos(Nx, comp == 0), Nx, bx, px), ax(ky, pos(Ny, comp == 1), Ny, by, py)
        d = pos(Nz, comp == 2)
        Z = np.cos(np.pi * np.outer(kz - 1, d) / Nz) if comp == 2 else np.sin(np.pi * np.outer(kz, d) / Nz)
        if comp < 2:
            Z[:, 0] = Z[:, -1] = 0.0
        ZY = (t(Z * amp[:, None]).T[:, None, :] * t(Y).T[None, :, :]).reshape(-1, modes)
        return (ZY @ t(X)).reshape(Z.shape[1], Y.shape[1], X.shape[1])

    A0, A1, A2 = potential(0), potential(1), potential(2)
    dx, dy, dz = grid.Δx, grid.Δy, float(np.asarray(grid.dzF)[grid.Hz])
    u = (A2[:, 1:] - A2[:, :-1]) / dy - (A1[:-1] - A1[1:]) / dz
    v = (A0[:-1] - A0[1:]) / dz - (A2[:, :, 1:] - A2[:, :, :-1]) / dx
    w = (A1[:, :, 1:] - A1[:, :, :-1]) / dx - (A0[:, 1:] - A0[:, :-1]) / dy
    s = rms / math.sqrt(float(u.square().mean() + v.square().mean() + w.square().mean()) + 1e-300)
    return u[:, :, :Nx + bx] * s, v[:, :Ny + by] * s, w * s


def _individuals(rng, grid, p, s, N, C, carbon, zmax):
    """Sizes lognormal, quotas about half full, positions uniform in the upper water column."""
    d = empty_individuals(C)
    g = {k: (v[s] if hasattr(v, "__len__") else v) for k, v in p.items()}
    d["ac"][:N] = True
    for k, n in (("x", grid.Nx), ("y", grid.Ny), ("z", zmax)):
        d[k][:N] = rng.random(N) * n
    Bm = np.exp(rng.standard_normal(N) * 0.2) * 1.3
    d["Sz"][:N] = Bm
    Bm *= float(g["Cquota"]) * float(g["Nsuper"])
    d["Bm"][:N] = Bm
    d["gen"][:N] = 1.0
    if carbon:
        d["Chl"][:N] = Bm * float(g["Chl2C"])
        return {k: v for k, v in d.items() if k not in ("Cq", "Nq", "Pq")} | {"Bd": d["Cq"]}
    Cq = 0.5 * float(g["Cqmax"]) * Bm * rng.uniform(0.8, 1.2, N)
    d["Cq"][:N] = Cq
    d["Nq"][:N] = 0.5 * (float(g["Nqmax"]) * (Bm + Cq) - Bm * float(g["R_NC"])) * rng.uniform(0.8, 1.2, N)
    d["Pq"][:N] = 0.5 * (float(g["Pqmax"]) * (Bm + Cq) - Bm * float(g["R_PC"])) * rng.uniform(0.8, 1.2, N)
    d["Chl"][:N] = Bm * float(g["Chl2Cint"])
    return d


def _land(grid_size, rng):
    """A sloping coast on the west side and a few islands, (x, y, z) True = water."""
    Nx, Ny, Nz = grid_size
    x, y = np.arange(Nx)[:, None], np.arange(Ny)[None, :]
    depth = np.clip((x + 3.0 * np.sin(2 * np.pi * y / Ny)) / (0.35 * Nx), 0.1, 1.0) * Nz
    for _ in range(3):
        cx, cy, r = rng.uniform(0.3, 0.9) * Nx, rng.uniform(0, 1) * Ny, rng.uniform(0.02, 0.06) * (Nx + Ny)
        depth = np.where(np.hypot(x - cx, y - cy) < r, 0.0, depth)
    return np.asfortranarray(np.arange(Nz)[None, None, :] < np.ceil(depth)[:, :, None])


def _world(case, seed, member=0):
    """Grid, parameters, initial state and forcing of one model, from the seed alone."""
    rng = np.random.default_rng([seed, member])
    nx, ny, nz, n = case["nx"], case["ny"], case["nz"], case["n"]
    if case["kind"] == "batch":
        # the members' sizes belong to the case: they do not change with the seed
        size = np.random.default_rng([case["members"], member])
        n = int(round(2.0 ** size.uniform(8, 13 if nx else 17)))
        if not nx:
            nx, ny, nz = int(size.integers(24, 129)), int(size.integers(24, 129)), int(size.integers(16, 33))
    FT = np.float32 if case["ft"] == "f32" else np.float64
    carbon, shelf = case.get("mode") == "carbon", bool(case.get("shelf"))
    parcel, flat = nx * ny * nz == 1, nz == 1
    dxy, dz, dT = (128.0, 128.0, 60.0) if parcel else (1000.0, 10.0, 60.0) if flat else (50.0, 2.0, 30.0)
    topo = (Bounded, Bounded, Bounded) if shelf else (Periodic, Periodic, Bounded)
    grid = RectilinearGrid(size=(nx, ny, nz), x=(0.0, nx * dxy), y=(0.0, ny * dxy), z=(0.0, -dz * nz), FT=FT, topology=topo,
                           landmask=_land((nx, ny, nz), rng) if shelf else None)
    nsp, steps, zmax = case["nsp"], case["steps"], min(nz, 20)
    per_cell = n * nsp / (nx * ny * zmax)
    # super-individuals whose nutrient demand the water of their cell can meet, and grazing that
    # balances growth near the initial population
    over = dict(Nsuper=[500.0 / (1.8e-11 * (1.0 + per_cell))] * nsp, grz_P=[6.0e-6 / (1.0 + per_cell)] * nsp)
    phyt = update_phyt_params(over, FT, N=nsp, mode=CarbonMode() if carbon else QuotaMode())
    bgc = update_bgc_params({"κh": 1.0e-2, "κv": 1.0e-5, "κhP": 1.0e-2, "κvP": 1.0e-5} if shelf else {}, FT)
    C = n * case["cap"]
    inds = [_individuals(rng, grid, phyt, s, n, C, carbon, zmax) for s in range(nsp)]
    trs = []
    for name in tracer_names:
        a = INIT[name] * (0.9 + 0.2 * rng.random(grid.total_size[::-1], dtype=np.float32).astype(np.float64)).transpose()
        if shelf:
            a = np.asfortranarray(a * grid.landmask)
        trs.append(fill_halo_tracer(a, grid))
    hours = int(steps * dT // 3600) + 1
    sun = 250.0 + 60.0 * np.arange(hours)
    parf = np.asfortranarray(sun * (0.9 + 0.2 * rng.random((nx, ny, 1))))
    deg = 24.0 + 0.5 * np.arange(hours) - 0.01 * np.arange(nz)[:, None]
    temp = np.asfortranarray(np.broadcast_to(deg, (nx, ny, nz, hours)))
    flow = not parcel
    vels = [_velocity(grid, seed * 1000 + member, q, 0.1 if flat else 0.05) for q in range(hours)] if flow else None
    bcs = [("DOC", "west", 1.0e-4), ("NO3", "bottom", 2.0e-6), ("DFe", "top", -1.0e-11)] if shelf else []
    return SimpleNamespace(grid=grid, phyt=phyt, bgc=bgc, nsp=nsp, n=n, C=C, inds=inds, trs=trs, dT=dT, parf=parf, temp=temp,
                           vels=vels, hours=hours, bcs=bcs, carbon=carbon, seed=(seed * 7919 + member) & 0xFFFFFFFF)


def _members(case, seed):
    return [_world(case, seed, m) for m in range(case["members"] if case["kind"] == "batch" else 1)]


# ------------------------------------------------------------------------------------------
# the program
# ------------------------------------------------------------------------------------------

def _pinned(n, dtype=torch.float64):
    return torch.zeros(n, dtype=dtype, pin_memory=DEV == "cuda")


def _dp(t):
    return ct.cast(t.data_ptr(), ct.POINTER(ct.c_double))


def _names(carbon):
    return ("x", "y", "z", "Bm") + (("Bd",) if carbon else ("Cq", "Nq", "Pq")) + ("Chl", "gen", "age")


class _Record:
    """What the program reads back of its members, in page-locked buffers that it keeps."""

    def __init__(self, worlds, case):
        G = [int(np.prod(w.grid.total_size)) for w in worlds]
        self.f32, self.G = case["ft"] == "f32", G
        self.tr, self.par = _pinned(NTR * sum(G)), _pinned(sum(G))
        self.inds = None
        if case.get("inds", True):
            names = _names(worlds[0].carbon)
            self.slots = [w.C for w in worlds for _ in range(w.nsp)]
            self.inds, self.ac = _pinned(len(names) * sum(self.slots)), _pinned(sum(self.slots), torch.uint8)
            self.structs, at, at8 = [], 0, 0
            for c in self.slots:
                st = _abi.pi_individuals()
                for k in names:
                    setattr(st, k, _dp(self.inds[at:at + c]))
                    at += c
                st.ac = ct.cast(self.ac[at8:].data_ptr(), ct.POINTER(ct.c_uint8))
                at8 += c
                self.structs.append(st)

    def read(self, get_tracer, get_par, get_inds, nsp):
        at = 0
        for m, G in enumerate(self.G):
            for n in range(NTR):
                get_tracer(m, n, _dp(self.tr[NTR * at + n * G:]))
            get_par(m, _dp(self.par[at:]))
            at += G
        out = [self.tr.float() if self.f32 else self.tr, self.par.float() if self.f32 else self.par]
        if self.inds is not None:
            for q, st in enumerate(self.structs):
                get_inds(q // nsp, q % nsp, ct.byref(st))
            out += [self.inds.float() if self.f32 else self.inds, self.ac]
        return out


def _check(rc):
    if rc:
        raise RuntimeError("status %d" % rc)


def prepare(case, seed):
    if case["kind"] == "field":
        return _prepare_field(case, seed)
    ws = _members(case, seed)
    st = SimpleNamespace(case=case, w=ws[0], lib=_lib.load(), rec=_Record(ws, case))
    stack = lambda w, c: np.stack([_f(v[c]) for v in w.vels], axis=-1)  # noqa: E731
    if case["kind"] == "batch":
        st.batch = PlanktonBatch([Member(w.grid, w.bgc, w.phyt, w.C, w.seed) for w in ws], nspecies=case["nsp"])
        for m, w in enumerate(ws):
            st.batch.set_state(m, w.inds, w.trs)
            st.batch.set_series(m, vels=dict(u=stack(w, 0), v=stack(w, 1), w=stack(w, 2)) if w.vels else None, ΔT_vel=3600.0,
                                PARF=w.parf, ΔT_PAR=3600.0, temp=w.temp, ΔT_temp=3600.0, time_offset=7)
        return st
    w = ws[0]
    FT = np.float32 if case["ft"] == "f32" else np.float64
    st.model = PlanktonModel(GPU(), w.grid, FT=FT, mode=CarbonMode() if w.carbon else QuotaMode(), max_individuals=w.C,
                             bgc_params={k: v for k, v in w.bgc.items()}, phyto=phyto_setup(w.phyt, [w.n] * w.nsp, w.nsp),
                             seed=w.seed, initial_state=(w.inds, w.trs))
    for tracer, pos, value in w.bcs:
        set_bc_b(st.model, tracer=tracer, pos=pos, bc_value=value)
    if case["kind"] == "coupled":
        # the host model's fields of each step: two velocity snapshots in turn
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).pin_memory()  # noqa: E731
        st.vel = [[pin(c.cpu().numpy()) for c in _velocity(w.grid, seed * 1000, q)] for q in range(2)]
        st.parf, st.temp = pin(w.parf[:, :, 0].T), pin(w.temp[:, :, :, 0].T)
        st.count = _pinned(w.nsp * case["steps"], torch.int64)
        return st
    st.sim = PlanktonSimulation(st.model, ΔT=w.dT, iterations=case["steps"], PARF=w.parf, temp=w.temp,
                                vels=dict(u=stack(w, 0), v=stack(w, 1), w=stack(w, 2)) if w.vels else None, ΔT_vel=3600.0)
    return st


def run(state):
    case = state.case
    if case["kind"] == "field":
        return _run_field(state)
    lib, rec = state.lib, state.rec
    if case["kind"] == "batch":
        b = state.batch
        b.step(state.w.dT, case["steps"], sync=False)
        return rec.read(lambda m, n, p: _check(lib.pi_batch_get_tracer(b.h, m, n, p)),
                        lambda m, p: _check(lib.pi_batch_get_diag(b.h, m, _abi.PI_DIAG_PAR, 0, p)),
                        lambda m, s, q: _check(lib.pi_batch_get_individuals(b.h, m, s, q)), case["nsp"])
    h = state.model._native.h
    if case["kind"] == "coupled":
        ptr = lambda t: ct.c_void_p(t.data_ptr())  # noqa: E731
        for i in range(case["steps"]):
            u, v, w = state.vel[i // 6 % 2]
            _check(lib.pi_set_velocity_f32(h, ptr(u), ptr(v), ptr(w)))
            _check(lib.pi_set_PARF_f32(h, ptr(state.parf)))
            _check(lib.pi_set_temp_f32(h, ptr(state.temp)))
            _check(lib.pi_time_step_async(h, ct.c_double(state.w.dT)))
            for s in range(case["nsp"]):
                _check(lib.pi_count_active_async(h, s, ct.c_void_p(state.count[i * case["nsp"] + s:].data_ptr())))
    else:
        update_b(state.sim, time_offset=dict(vels=True, PARF=True, temp=True), sync=False)
    out = rec.read(lambda m, n, p: _check(lib.pi_get_tracer(h, n, p)),
                   lambda m, p: _check(lib.pi_get_diag(h, _abi.PI_DIAG_PAR, 0, p)),
                   lambda m, s, q: _check(lib.pi_get_individuals(h, s, q)), case["nsp"])
    return out + [state.count] if case["kind"] == "coupled" else out


def _field_inputs(case, seed):
    rng = np.random.default_rng([seed, 5])
    nx, ny, nz, shelf = case["nx"], case["ny"], case["nz"], bool(case.get("shelf"))
    topo = (Bounded, Bounded, Bounded) if shelf else (Periodic, Periodic, Bounded)
    grid = RectilinearGrid(size=(nx, ny, nz), x=(0.0, nx * 50.0), y=(0.0, ny * 50.0), z=(0.0, -2.0 * nz), FT=np.float64,
                           topology=topo, landmask=_land((nx, ny, nz), rng) if shelf else None)
    c = (1.0 + 0.2 * rng.random(grid.total_size[::-1])).transpose()
    c = fill_halo_tracer(np.asfortranarray(c * grid.landmask), grid)
    vel = _padded(grid, _velocity(grid, seed, 0))
    return grid, torch.as_tensor(c.transpose().copy(), device=DEV), vel


def _prepare_field(case, seed):
    grid, c, vel = _field_inputs(case, seed)
    g, keep = make_grid_struct(grid)
    return SimpleNamespace(case=case, lib=_lib.load(), g=g, keep=keep, c=c, vel=[x.contiguous() for x in vel], out=torch.zeros_like(c))


def _run_field(state):
    stream = ct.c_void_p(torch.cuda.current_stream().cuda_stream)
    _check(state.lib.pi_tracer_advection_noalloc(ct.byref(state.g), _dp(state.c), *(_dp(x) for x in state.vel),
                                                 ct.c_double(30.0), _dp(state.out), stream))
    return state.out


def work(case):
    """Each step reads and writes the state of every individual and the 14 tracers of every cell
    and reads the step's forcing; a pass writes its record once."""
    word = 4 if case["ft"] == "f32" else 8
    if case["kind"] == "field":
        return dict(bytes=8 * 5 * case["nx"] * case["ny"] * case["nz"], flops=0)
    cells, inds, steps = case["nx"] * case["ny"] * case["nz"], case["n"] * case["nsp"], case["steps"]
    if case["kind"] == "batch":
        cells = case["members"] * (1 if case["nx"] else 76 * 76 * 24)
        inds = case["members"] * (2200 if case["nx"] else 21000)
    state = (8 if case.get("mode") == "carbon" else 10) * 2 * word + 2
    record = word * 15 * cells + (word * 10 * inds * case["cap"] if case.get("inds", True) else 0)
    return dict(bytes=steps * (inds * state + cells * (2 * NTR + 5) * word) + record, flops=0)


# ------------------------------------------------------------------------------------------
# the time step in Float64 torch: fields are (z, y, x) tensors with halos
# ------------------------------------------------------------------------------------------

def _lit(x):
    return float(np.float32(x))


def _fill(c, grid, face=(False, False, False)):
    """The halo rule of each axis; `face`: the field has its own face on a Bounded axis."""
    for ax, N, H, b in ((-1, grid.Nx, grid.Hx, grid.topo[0]), (-2, grid.Ny, grid.Hy, grid.topo[1]), (-3, grid.Nz, grid.Hz, grid.topo[2])):
        bounded, f = b == Bounded.code, face[-1 - ax]
        lo = (c.narrow(ax, H, 1).expand_as(c.narrow(ax, 0, H)) if bounded else c.narrow(ax, N, H)).clone()
        hi = (c.narrow(ax, N + H - 1, 1).expand_as(c.narrow(ax, N + H, H)) if bounded else c.narrow(ax, H, H)).clone()
        c.narrow(ax, 0, H).copy_(lo)
        if bounded and f:
            c.narrow(ax, N + H + 1, H - 1).copy_(c.narrow(ax, N + H, 1).clone())
        else:
            c.narrow(ax, N + H, H).copy_(hi)
    return c


def _padded(grid, vel):
    out = []
    for q, v in enumerate(vel):
        a = torch.zeros(grid.total_size[::-1], dtype=torch.float64, device=DEV)
        z, y, x = v.shape
        a[grid.Hz:grid.Hz + z, grid.Hy:grid.Hy + y, grid.Hx:grid.Hx + x] = v.to(DEV)
        out.append(_fill(a, grid, tuple(q == k for k in range(3))))
    return out


def _at(c, ax, o, N, H):
    """The interior cells of axis `ax` moved by o."""
    return c.narrow(ax, H + o, N)


def _inner(c, grid, skip=None):
    for ax, N, H in ((-1, grid.Nx, grid.Hx), (-2, grid.Ny, grid.Hy), (-3, grid.Nz, grid.Hz)):
        if ax != skip:
            c = c.narrow(ax, H, N)
    return c


def _sweep(ct_, c0, vel, grid, ax, area, spacing, vol, mask, dT):
    """One DST3FL sweep of tracer_temp ct_ (original tracer c0): the new interior."""
    N, H = {-1: (grid.Nx, grid.Hx), -2: (grid.Ny, grid.Hy), -3: (grid.Nz, grid.Hz)}[ax]
    bounded = grid.topo[-1 - ax] == Bounded.code
    down = ax == -3                       # w is positive upward, the index grows downward
    cut = lambda a, o, n=N: _inner(a, grid, ax).narrow(ax, H + o, n)  # noqa: E731
    m = [cut(mask, o, N + 1) for o in (-2, -1, 0, 1)] if mask is not None else [1.0] * 4
    v = [cut(ct_, o, N + 1) for o in (-2, -1, 0, 1)]
    sp, ar = spacing.narrow(0, H, N + 1).reshape([-1 if a == ax else 1 for a in (-3, -2, -1)]) if spacing.dim() else spacing, area
    vl = cut(vel, 0, N + 1)
    cfl, tr = (vl * dT / sp).abs(), ar * vl
    sgn = -1.0 if down else 1.0
    d0, dm, dp = sgn * (v[2] - v[1]) * m[2] * m[1], sgn * (v[1] - v[0]) * m[1] * m[0], sgn * (v[3] - v[2]) * m[3] * m[2]

    def psi(num):
        big = d0.abs() * _lit(1e20) <= num.abs()
        th = torch.where(big, torch.copysign(torch.full_like(num, _lit(1e20)), num * d0), num / torch.where(big, torch.ones_like(d0), d0))
        lim = torch.minimum((2 - cfl) * (1 - cfl) / 6 + (1 - cfl * cfl) / 6 * th, torch.ones_like(th))
        return torch.clamp_min(torch.minimum(lim, th * (1 - cfl) / (cfl + _lit(1e-20))), 0.0)

    up, dn = 0.5 * (tr + tr.abs()), 0.5 * (tr - tr.abs())
    F = up * (v[2] + psi(dp) * d0) + dn * (v[1] - psi(dm) * d0) if down else up * (v[1] + psi(dm) * d0) + dn * (v[2] - psi(dp) * d0)
    if bounded:
        F = F.clone()
        F.narrow(ax, N, 1).zero_()
    both = m[3].narrow(ax, 0, N) * m[2].narrow(ax, 0, N) if mask is not None else 1.0
    a0, a1 = F.narrow(ax, 0, N), F.narrow(ax, 1, N)
    t0, t1 = tr.narrow(ax, 0, N), tr.narrow(ax, 1, N)
    dF, ft = ((a0 - a1), (t0 - t1)) if down else ((a1 - a0), (t1 - t0))
    return _inner(ct_, grid) - dT / vol * (dF * both - _inner(c0, grid) * (ft * both))


def _advect(c, vel, grid, mask, dT):
    """tracer_temp - tracer on the interior after the x, y and z sweeps."""
    dzF, dzC = (torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV) for a in (grid.dzF, grid.dzC))
    dz = dzF[grid.Hz:grid.Hz + grid.Nz].reshape(-1, 1, 1)
    one = torch.ones((), dtype=torch.float64, device=DEV)
    vol, t = grid.Δx * grid.Δy * dz, c
    for ax, area, sp, q in ((-1, grid.Δy * dz, one * grid.Δx, 0), (-2, grid.Δx * dz, one * grid.Δy, 1), (-3, one * grid.Δx * grid.Δy, dzC, 2)):
        new = torch.zeros_like(c)
        _inner(new, grid).copy_(_sweep(t, c, vel[q], grid, ax, area, sp, vol, mask, dT))
        t = _fill(new, grid)
    return _inner(t, grid) - _inner(c, grid), vol, dz


def _philox(seed, it, sp, purpose, slots):
    """Three uniforms on the 2^-24 lattice of Philox4x32-10 for every slot."""
    M = 0xFFFFFFFF

    def mul(a, b):
        lo, hi = a * (b & 0xFFFF), a * (b >> 16)
        t = (lo >> 16) + (hi & 0xFFFF)
        return (hi >> 16) + (t >> 16), ((t & 0xFFFF) << 16) | (lo & 0xFFFF)

    c = [slots.clone(), torch.full_like(slots, it), torch.full_like(slots, sp | purpose << 16), torch.full_like(slots, 0x706c6b74)]
    k0, k1 = seed & M, seed >> 32 & M
    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return [(x >> 8).double() * 2.0 ** -24 for x in c[:3]]


class _Exact:
    def __init__(self, w):
        self.w, g = w, w.grid
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
        self.names = _names(w.carbon)
        self.sp = []
        for d in w.inds:
            s = {k: t(np.asarray(d[k], dtype=np.float64)) for k in self.names}
            s |= {k: torch.zeros(w.C, dtype=torch.bool, device=DEV) for k in ("gz", "mt", "dv")}
            s["ac"], s["zi"] = t(np.asarray(d["ac"], dtype=bool)), t(np.asarray(d["zi"], dtype=np.int64))
            self.sp.append(s)
        self.tr = torch.stack([t(a.transpose()) for a in w.trs])
        self.other = torch.zeros_like(self.tr)        # tracers live in two buffers in turn
        self.diag = torch.zeros(g.total_size[::-1], dtype=torch.float64, device=DEV)
        lm = np.asarray(g.landmask)
        self.mask = None if lm.all() else t(lm.transpose().astype(np.float64))
        self.dzF, self.dzC = t(np.asarray(g.dzF, dtype=np.float64)), t(np.asarray(g.dzC, dtype=np.float64))
        self.v0 = [torch.zeros(g.total_size[::-1], dtype=torch.float64, device=DEV) for _ in range(3)]
        self.it = 0
        self.slots = torch.arange(w.C, dtype=torch.int64, device=DEV)

    def bc(self, x, q):
        N = float((self.w.grid.Nx, self.w.grid.Ny, self.w.grid.Nz)[q])
        if self.w.grid.topo[q] == Bounded.code:
            return torch.where(x > N, 2 * N - x, torch.where(x < 0, -x, x))
        return torch.where(x > N, x - N, torch.where(x < 0, x + N, x))

    def sample(self, f, q, pos):
        g = self.w.grid
        Gy, Gx = f.shape[1], f.shape[2]
        i, d = [], []
        for a, H in enumerate((g.Hx, g.Hy, g.Hz)):
            s = pos[a] + (1.0 if a == q else 0.5)
            i.append(s.trunc().long() + H - 1)
            d.append(s - s.trunc())
        base, fl, out = (i[2] * Gy + i[1]) * Gx + i[0], f.reshape(-1), 0.0
        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    wt = (d[0] if a else 1 - d[0]) * (d[1] if b else 1 - d[1]) * (d[2] if c else 1 - d[2])
                    sp = (g.Δx, g.Δy, self.dzC[i[2] + c])[q]
                    out = out + wt * fl[base + a + Gx * (b + Gy * c)] / sp
        return out

    def move(self, s, sp, v1, dT):
        w, g = self.w, self.w.grid
        on = s["ac"].nonzero().squeeze(1)
        X = [s[k][on] for k in "xyz"]
        vh = [(a + b) * 0.5 for a, b in zip(self.v0, v1)]
        sign, total, pos = (1.0, 1.0, -1.0), None, X
        for f, wt, nxt in ((self.v0, 1.0, 0.5), (vh, 2.0, 0.5), (vh, 2.0, 1.0), (v1, 1.0, None)):
            k = [self.sample(f[q], q, pos) for q in range(3)]
            total = [a * wt for a in k] if total is None else [a + b * wt for a, b in zip(total, k)]
            if nxt:
                pos = [self.bc(X[q] + sign[q] * nxt * k[q] * dT, q) for q in range(3)]
        X = [self.bc(X[q] + sign[q] * total[q] / 6.0 * dT, q) for q in range(3)]
        r = _philox(w.seed, self.it, sp, 0, self.slots[on])
        kdz = (s["zi"][on] + g.Hz).clamp(1, g.Nz + 2 * g.Hz) - 1
        for q, (kap, sc) in enumerate(((w.bgc["κhP"], g.Δx), (w.bgc["κhP"], g.Δy), (w.bgc["κvP"], self.dzC[kdz]))):
            X[q] = self.bc(X[q] + (r[q] - 0.5) * 2.0 * math.sqrt(float(kap) * dT) / sc, q)
        H = (g.Hx, g.Hy, g.Hz)
        idx = [torch.full((w.C,), h, dtype=torch.int64, device=DEV) for h in H]
        for q, k in enumerate("xyz"):
            s[k] = torch.zeros_like(s[k])
            s[k][on] = X[q]
            idx[q][on] = (X[q] + 1.0).trunc().long() + H[q]
        s["zi"] = idx[2]
        s["cell"] = ((idx[2] - 1) * (g.Ny + 2 * g.Hy) + idx[1] - 1) * (g.Nx + 2 * g.Hx) + idx[0] - 1

    def divide(self, s):
        p, d = s["dv"].nonzero().squeeze(1), (~s["ac"]).nonzero().squeeze(1)
        d = d[:len(p)]
        for k in self.names[3:-2]:
            if k == "Bd":
                s[k][d] = s[k][d] * 0.5
            else:
                s[k][d] = s[k][p] * 0.5
            s[k][p] = s[k][p] * 0.5
        for k in "xyz":
            s[k][d] = s[k][p]
        s["gen"][d] = s["gen"][p] + 1.0
        s["gen"][p] = s["gen"][p] + 1.0
        s["age"][p] = 0.0
        s["age"][d] = s["age"][d] * 0.0
        s["ac"] = s["ac"].clone()
        s["ac"][d] = True

    @staticmethod
    def dec(x, xmax, k, pw):
        f = (1.0 - x / xmax).clamp(0.0, 1.0) ** pw
        return f / (_lit(k) + f)

    def heat(self, T, p, damp):
        R, T0 = _lit(8.3145), _lit(273.15)
        ref = math.exp(-p["Ea"] / (R * (p["Topt"] + T0)))
        k = torch.exp(-p["Ea"] / (R * (T + T0)))
        if damp:
            k = k * self.dec(T - p["Topt"], p["Tmax"] - p["Topt"], damp, 4)
        return torch.clamp_max(k.clamp_min(0.0) / ref, 1.0)

    def grow(self, s, sp, p, env, ac0, dT, plk):
        names, dead = self.names, ac0 & ~s["ac"]
        if dead.any() and self.w.carbon:
            T, Bm, Bd = env["T"][s["cell"][dead]], s["Bm"][dead], s["Bd"][dead]
            TD = (T - p["Topt"]) * p["f_T2B"] * (Bm - Bd) * (T > p["Topt"]) * (Bd < Bm) * (p["thermal"] == 1.0)
            s["Bd"][dead] = Bd + torch.minimum(TD, (Bm - Bd) / dT).clamp_min(0.0) * dT
        on = s["ac"].nonzero().squeeze(1)
        c, seen = s["cell"][on], ac0[on]
        e = {k: torch.where(seen, v[c], torch.zeros((), dtype=torch.float64, device=DEV)) for k, v in env.items() if k != "inside"}
        I = {k: s[k][on] for k in names}  # noqa: E741
        tiny, one = _lit(1e-30), torch.ones_like(I["Bm"])
        T, par, pop, Bm, Chl = e["T"], e["par"], e["pop"], I["Bm"], I["Chl"]
        aI = par * p["α"] * p["Φ"]
        grid_in = env["inside"].reshape(-1)[c] & seen
        if self.w.carbon:
            Bd, th = I["Bd"], p["thermal"]
            PCm = p["PCmax"] * (self.heat(T, p, None) * th + self.heat(T, p, 1e-1) * (1 - th))
            light = 1 - torch.exp(-aI / PCm.clamp_min(tiny) * Chl / Bm.clamp_min(tiny))
            PS = PCm * (Bm - Bd).clamp_min(0.0) * (light * (1 - p["is_bact"]) + p["is_bact"])
            gam = torch.clamp_max(Bd / Bm.clamp_min(tiny) * (Bd > 0), 1.0) * (th == 1.0)
            TD = (T - p["Topt"]) * p["f_T2B"] * (Bm - Bd) * (T > p["Topt"]) * (Bd < Bm) * (th == 1.0)
            TD = torch.minimum(TD, (Bm - Bd) / dT).clamp_min(0.0)
            RS = p["respir"] * Bm * self.heat(T, p, None)
            I["Bm"] = Bm + (PS * (1 - gam) - RS) * dT
            I["Bd"] = Bd + (TD - PS * gam) * dT
            I["Chl"] = I["Bm"] * p["Chl2C"]
            take = {"DIC": (RS - PS) * dT}
        else:
            Cq, Nq, Pq, tf = I["Cq"], I["Nq"], I["Pq"], self.heat(T, p, None)
            PCm = p["PCmax"] * self.heat(T, p, 4e-2)
            PS = PCm * (1 - torch.exp(-aI / PCm.clamp_min(tiny) * Chl / Bm.clamp_min(tiny))) * Bm
            qn, qp = (Nq + Bm * p["R_NC"]) / (Bm + Cq).clamp_min(tiny), (Pq + Bm * p["R_PC"]) / (Bm + Cq).clamp_min(tiny)
            rn, rp = self.dec(qn, p["Nqmax"], 1e-4, 4), self.dec(qp, p["Pqmax"], 1e-4, 4)

            def uptake(v, reg, x, ks):
                return torch.minimum(v * reg * x / (x + ks).clamp_min(tiny) * tf * Bm, x / dT / pop.clamp_min(1.0))

            NH4, NO3, PO4, DOC = (e[k].clamp_min(0.0) for k in ("NH4", "NO3", "PO4", "DOC"))
            VNH4, VNO3 = uptake(p["VNH4max"], rn, NH4, p["KsatNH4"]), uptake(p["VNO3max"], rn, NO3, p["KsatNO3"])
            VPO4 = uptake(p["VPO4max"], rp, PO4, p["KsatPO4"])
            Cq, Pq, Nq = Cq + PS * dT, Pq + VPO4 * dT, Nq + (VNH4 + VNO3) * dT
            VDOC = uptake(p["VDOCmax"], self.dec(Cq / (Bm + Cq).clamp_min(tiny), p["Cqmax"], 1e-4, 4), DOC, p["KsatDOC"])
            ratio = PS / (VDOC + PS)
            VDOC = VDOC * ((ratio > _lit(1e-2)) | ratio.isnan())
            rchl = PS / Bm.clamp_min(tiny) * p["Chl2N"] / (aI * Chl / Bm).clamp_min(tiny) * (par > _lit(1e-1))
            resp = p["respir"] * Bm * tf
            Cq = Cq + (VDOC - resp) * dT
            lack = (0.0 - Cq).clamp_min(0.0)
            Bm, Nq, Pq, Cq = Bm - lack, Nq + lack * p["R_NC"], Pq + lack * p["R_PC"], Cq + lack
            mn = torch.minimum(torch.minimum(Cq, Nq / p["R_NC"]), Pq / p["R_PC"])
            BS, exu = mn * p["k_mtb"], (Cq - mn).clamp_min(0.0) * p["k_mtb"]
            I |= {"Bm": Bm + dT * BS, "Cq": Cq - dT * (BS + exu), "Nq": Nq - dT * BS * p["R_NC"], "Pq": Pq - dT * BS * p["R_PC"],
                  "Chl": Chl + dT * BS * p["R_NC"] * rchl}
            take = {"DIC": (resp - PS) * dT, "DOC": (exu - VDOC) * dT, "NH4": -VNH4 * dT, "NO3": -VNO3 * dT, "PO4": -VPO4 * dT}
        I["age"] = I["age"] + dT / 3600.0
        Sz = I["Bm"] / (p["Cquota"] * p["Nsuper"])
        mort = p["mort_P"] * self.dec(Sz, p["mort_reg"], 1e-5, 4)
        if self.w.carbon and p["thermal"] == 1.0:
            mort = p["mort_P"] * (1 - self.dec(I["Bd"] / I["Bm"].clamp_min(tiny), _lit(0.99) * one, 1e-6, 4))
        dvid = p["dvid_P"] * (1 - self.dec(Sz, p["dvid_reg"], 2e-3, 2))
        r = _philox(self.w.seed, self.it, sp, 1, self.slots[on])
        for k, prob, x in (("gz", pop * p["grz_P"], r[0]), ("mt", mort, r[1]), ("dv", dvid, r[2])):
            s[k] = torch.zeros_like(s[k])
            s[k][on] = x < prob * dT
        for k in names:
            s[k][on] = I[k]
        for name, v in take.items():
            plk[tracer_names.index(name)].index_add_(0, c[grid_in], v[grid_in])

    def step(self, v1, parf, temp, dT):
        w, g, tr = self.w, self.w.grid, self.tr
        n_of = tracer_names.index
        self.it += 1
        G = self.diag.numel()
        Z = lambda: torch.zeros(G, dtype=torch.float64, device=DEV)  # noqa: E731
        pop, chl, plk = Z(), Z(), torch.zeros((NTR, G), dtype=torch.float64, device=DEV)
        for k, s in enumerate(self.sp):
            self.move(s, k, v1, dT)
            on = s["ac"]
            pop.index_add_(0, s["cell"][on], torch.ones_like(s["x"][on]))
            chl.index_add_(0, s["cell"][on], s["Chl"][on])
        shape = self.diag.shape
        dz = self.dzF[g.Hz:g.Hz + g.Nz]
        par, light = torch.zeros_like(self.diag), parf
        ci = _inner(chl.reshape(shape), g)
        pin = _inner(par, g)
        for k in range(g.Nz):
            at = (ci[k] / (g.Δx * g.Δy * dz[k]) * float(w.bgc["kc"]) + float(w.bgc["kw"])) * dz[k]
            ex = torch.exp(-at)
            pin[k] = light * (1 - ex) / at
            light = light * ex
        self.diag += par
        inside = torch.zeros(shape, dtype=torch.bool, device=DEV)
        _inner(inside, g).fill_(True)
        T = torch.zeros_like(self.diag)
        _inner(T, g).copy_(temp)
        env = dict(par=par.reshape(-1), T=T.reshape(-1), pop=pop, inside=inside, **{k: tr[n_of(k)].reshape(-1) for k in ("NH4", "NO3", "PO4", "DOC")})
        for k, s in enumerate(self.sp):
            p = {a: float(b[k] if hasattr(b, "__len__") else b) for a, b in w.phyt.items()}
            ac0 = s["ac"].clone()
            gz, mt = ac0 & s["gz"], ac0 & ~s["gz"] & s["mt"]
            for lost, f in ((gz, "graz"), (mt, "mort")):
                q = (lost & inside.reshape(-1)[s["cell"]]).nonzero().squeeze(1)
                c, Bm = s["cell"][q], s["Bm"][q]
                pools = [("C", Bm if w.carbon else Bm + s["Cq"][q])]
                pools += [] if w.carbon else [("N", Bm * p["R_NC"] + s["Nq"][q]), ("P", Bm * p["R_PC"] + s["Pq"][q])]
                for el, v in pools:
                    fr = p[f + "Frac" + el]
                    plk[n_of("DO" + el)].index_add_(0, c, v * fr)
                    plk[n_of("PO" + el)].index_add_(0, c, v * (1 - fr))
            s["ac"] = ac0 & ~gz & ~mt
            s["dv"] = s["dv"] & s["ac"]
            self.divide(s)
            self.grow(s, k, p, env, ac0, dT, plk)
        new = self.other
        dt = self.tracers(v1, dT, plk.reshape((NTR,) + tuple(shape)))
        for n in range(NTR):
            _inner(new[n], g).copy_(_inner(tr[n], g) + dt[n])
            _fill(new[n], g)
        self.tr, self.other, self.v0 = new, tr, v1

    def tracers(self, v1, dT, plk):
        g, b, tr = self.w.grid, {k: float(v) for k, v in self.w.bgc.items()}, self.tr
        n_of = tracer_names.index
        m = self.mask
        both = lambda a, ax, o: 1.0 if m is None else (_inner(m, g, ax).narrow(ax, (g.Hx, g.Hy, g.Hz)[-1 - ax] + o, a) *  # noqa: E731
                                                       _inner(m, g, ax).narrow(ax, (g.Hx, g.Hy, g.Hz)[-1 - ax] + o - 1, a))
        Gc = []
        for n in range(NTR):
            d, vol, dz = _advect(tr[n], v1, g, m, dT)
            if b["κh"] or b["κv"]:
                lap = 0.0
                hz = self.dzF[g.Hz:g.Hz + g.Nz + 1].reshape(-1, 1, 1)
                for ax, N, H, kap, ar, sp in ((-1, g.Nx, g.Hx, b["κh"], g.Δy * dz, g.Δx), (-2, g.Ny, g.Hy, b["κh"], g.Δx * dz, g.Δy),
                                              (-3, g.Nz, g.Hz, b["κv"], g.Δx * g.Δy, hz)):
                    c = _inner(tr[n], g, ax)
                    df = (c.narrow(ax, H, N + 1) - c.narrow(ax, H - 1, N + 1)) * both(N + 1, ax, 0) * (ar * kap if ax > -3 else kap * ar) / sp
                    lap = lap + (df.narrow(ax, 1, N) - df.narrow(ax, 0, N)) * both(N, ax, 1)
                d = d + lap / vol * dT
            Gc.append(d)
        dzC = self.dzC[:g.Nz].reshape(-1, 1, 1)
        for name, ws in (("PFe_inorg", b["w_sink_inorg"]), ("Dust", b["w_sink_inorg"]), ("PFe_bio", b["w_sink_org"])):
            c = ws * _inner(tr[n_of(name)], g)
            up, dn = torch.zeros_like(c), c.clone()
            up[1:] = c[:-1]
            dn[-1] = 0.0
            Gc[n_of(name)] = Gc[n_of(name)] + (up - dn) / dzC * dT
        C = {k: _inner(tr[n_of(k)], g).clamp_min(0.0) for k in tracer_names}

        def add(name, v):
            Gc[n_of(name)] = Gc[n_of(name)] + v * dT

        for src, dst, rate in (("DOC", "DIC", "kDOC"), ("POC", "DOC", "kPOC"), ("DON", "NH4", "kDON"), ("PON", "DON", "kPON"),
                               ("DOP", "PO4", "kDOP"), ("POP", "DOP", "kPOP"), ("NH4", "NO3", "Nit")):
            add(dst, C[src] * b[rate])
            add(src, -C[src] * b[rate])
        free = (C["DFe"] - b["ligand"]).clamp_min(0.0) * C["DFe"] * b["DFeFrac"] * b["lambda_Fe"]
        scav = (b["lambda_min"] + b["lambda_dust"] * C["Dust"]) * C["DFe"] * b["DFeFrac"]
        onto = b["lambda_POC"] * C["POC"] * C["DFe"] * b["DFeFrac"]
        add("DFe", C["PFe_bio"] * b["kPOC"] - onto - scav + C["PFe_inorg"] * b["kdiss"] - free)
        add("PFe_bio", onto - b["kPOC"] * C["PFe_bio"])
        add("PFe_inorg", scav + free - C["PFe_inorg"] * b["kdiss"])
        for name, pos, val in self.w.bcs:
            n, v = n_of(name), Gc[n_of(name)].clone()
            if pos == "west":
                v[:, :, 0] += val * dT / g.Δx
            elif pos == "bottom":
                v[-1] += val * dT / dz[-1]
            else:
                v[0] -= val * dT / dz[0]
            Gc[n] = v
        return [Gc[n] + _inner(plk[n], g) / vol for n in range(NTR)]

    def pass_(self, case, seed):
        w, g = self.w, self.w.grid
        r = (lambda a: a.float().double()) if case["ft"] == "f32" else (lambda a: a)
        field = lambda a: torch.as_tensor(np.array(a.transpose(), order="C"), device=DEV)  # noqa: E731
        still = [torch.zeros(g.total_size[::-1], dtype=torch.float64, device=DEV) for _ in range(3)]
        coupled = case["kind"] == "coupled"
        vels = [_velocity(g, seed * 1000, q) for q in range(2)] if coupled else w.vels
        vels = [_padded(g, [r(x) for x in v]) for v in vels] if vels else [still]
        if case["ft"] == "f32":
            self.tr = r(self.tr)
        for i in range(case["steps"]):
            h = 0 if coupled else int(i * w.dT // 3600)
            self.step(vels[i // 6 % 2] if coupled else vels[min(h, len(vels) - 1)], r(field(w.parf[:, :, h])), r(field(w.temp[:, :, :, h])), w.dT)


def exact(case, seed):
    """run()'s answer for a new state, in Float64. None for the ensembles of many members, which would
    take minutes here; flags and counts have no such value."""
    if case["kind"] == "field":
        grid, c, vel = _field_inputs(case, seed)
        lm = np.asarray(grid.landmask)
        mask = None if lm.all() else torch.as_tensor(np.ascontiguousarray(lm.transpose()).astype(np.float64), device=DEV)
        out = torch.zeros_like(c)
        _inner(out, grid).copy_(_advect(c, vel, grid, mask, 30.0)[0])
        return out
    if case.get("members", 1) * case["steps"] > 700:
        return None
    ws = _members(case, seed)
    xs = [_Exact(w) for w in ws]
    for x in xs:
        x.pass_(case, seed)
    out = [torch.cat([x.tr.reshape(-1) for x in xs]).cpu(), torch.cat([x.diag.reshape(-1) for x in xs]).cpu()]
    if case.get("inds", True):
        out += [torch.cat([s[k] for x in xs for s in x.sp for k in x.names]).cpu(), None]
    return out + [None] if case["kind"] == "coupled" else out
