"""Flux conditions of the FP32 form on both sides of the level count where the walks of k32_ztail finish the
cells themselves (up to 10) and k32_close does (above), with z walks shorter than that, and in a batch where
one member has conditions and another has none: against the oracle, each tracer within 1e-5 of its largest."""
import numpy as np
import pytest

import oracle
from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals.batch import Member, PlanktonBatch
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lz", [8, 32])
@pytest.mark.parametrize("nz", [1, 9, 10, 11, 17])
def test_flux_conditions_vs_oracle(gpu_lib, nz, lz):
    rng = np.random.default_rng(nz)
    phyt, bgc = update_phyt_params({}, np.float64, N=1), update_bgc_params({"κv": 1e-3}, np.float64)
    members, states, vels = [], [], []
    for q, (nx, ny) in enumerate([(35, 6), (5, 33)]):
        size = (nx, ny, nz)
        grid = RectilinearGrid(size=size, x=(0.0, nx * 50.0), y=(0.0, ny * 50.0), z=(0.0, -2.0 * nz), FT=np.float64,
                               topology=(Bounded, Periodic if q else Bounded, Bounded), landmask=rng.random(size) < 0.9)
        inds = [W.make_individuals(grid, phyt, 0, 8, 8, rng)]
        inds[0]["ac"][:] = False                                 # tracers only
        members.append(Member(grid, bgc, phyt, 8, 3))
        states.append((inds, W.make_tracers(grid, rng)))
        shapes = [(nx + 1, ny, nz), (nx, ny + (0 if q else 1), nz), (nx, ny, nz + 1)]
        vels.append([s * rng.standard_normal(n) for s, n in zip((0.1, 0.1, 2e-3), shapes)])
    batch = PlanktonBatch(members, nspecies=1)
    batch.set_option("z_levels", lz)
    models = [oracle.OracleModel(m.grid, bgc, phyt, 1, 8, 3) for m in members]
    faces = list(_abi.FACES)
    fluxes = [(n, faces[(n + d) % 6], 1e-4 * (n + 1)) for n in range(0, _abi.NTRACERS, 2) for d in (0, 2)]
    for q, m in enumerate(models):
        batch.set_state(q, *states[q])
        m.set_state(*states[q])
        for n, face, v in fluxes if q == 0 else []:
            m.set_flux_bc(n, _abi.FACES[face], _abi.PI_BC_CONST, [v])
            batch.set_flux_bc(q, n, _abi.FACES[face], _abi.PI_BC_CONST, [v])
    for _ in range(3):
        for q, m in enumerate(models):
            g = members[q].grid
            for t, i in ((m, None), (batch, q)):
                a = () if i is None else (i,)
                t.set_velocity(*a, *vels[q])
                t.set_PARF(*a, np.full((g.Nx, g.Ny), 300.0))
                t.set_temp(*a, np.full((g.Nx, g.Ny, g.Nz), 25.0))
            m.time_step(60.0)
        batch.step(60.0, 1)
    for q, m in enumerate(models):
        g = members[q].grid
        inner = tuple(slice(h, h + n) for h, n in zip((g.Hx, g.Hy, g.Hz), (g.Nx, g.Ny, g.Nz)))
        for n, name in enumerate(_abi.tracer_names):
            a, b = m.get_tracer(n)[inner], batch.get_tracer(q, n)[inner]
            assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(a)), (q, name)
