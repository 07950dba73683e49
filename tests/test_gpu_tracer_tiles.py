"""The x-y and z tracer kernels of the FP32 form at the edges of their work items (31 columns × 16 rows;
32 columns × 32 levels), with land, tracer diffusion and flux boundary conditions on every face, against
the oracle: each tracer within 1e-5 of its largest value, the bar of the FP32 form."""
import numpy as np
import pytest

import oracle
from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._native import CModel
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("land", [False, True])
@pytest.mark.parametrize("size,topo", [((30, 15, 31), Periodic), ((31, 16, 32), Periodic), ((32, 17, 33), Bounded),
                                       ((63, 5, 65), Bounded), ((3, 33, 2), Periodic)])
def test_tiles_vs_oracle(gpu_lib, size, topo, land, general):
    rng = np.random.default_rng(sum(size))
    lm = rng.random(size) < 0.85 if land else np.ones(size, dtype=bool)
    grid = RectilinearGrid(size=size, x=(0.0, size[0] * 50.0), y=(0.0, size[1] * 50.0), z=(0.0, -2.0 * size[2]),
                           FT=np.float64, topology=(topo, topo, Bounded), landmask=lm)
    phyt = update_phyt_params({}, np.float64, N=1)
    bgc = update_bgc_params({"κh": 1.0, "κv": 1e-3} if general else {}, np.float64)
    inds = [W.make_individuals(grid, phyt, 0, 8, 8, rng)]
    inds[0]["ac"][:] = False                                     # tracers only
    trs = W.make_tracers(grid, rng)
    e = int(topo is Bounded)                                     # faces of a Bounded axis: N + 1
    shapes = [(size[0] + e, size[1], size[2]), (size[0], size[1] + e, size[2]), (size[0], size[1], size[2] + 1)]
    vel = [v * rng.standard_normal(s) for v, s in zip((0.1, 0.1, 2e-3), shapes)]
    models = [CModel(gpu_lib, "pi_", grid, bgc, phyt, 1, 8, 3, precision=_abi.PI_FP32), oracle.OracleModel(grid, bgc, phyt, 1, 8, 3)]
    for m in models:
        m.set_state(inds, trs)
        if general:
            for n, face in enumerate(_abi.FACES):
                m.set_flux_bc(n, _abi.FACES[face], _abi.PI_BC_CONST, [1e-4 * (n + 1)])
        for _ in range(4):
            m.set_velocity(*vel)
            m.set_PARF(np.full(size[:2], 300.0))
            m.set_temp(np.full(size, 25.0))
            m.time_step(60.0)
    inner = tuple(slice(h, h + n) for h, n in zip((grid.Hx, grid.Hy, grid.Hz), size))
    for n, name in enumerate(_abi.tracer_names):
        a, b = models[1].get_tracer(n)[inner], models[0].get_tracer(n)[inner]
        assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(a)), name
