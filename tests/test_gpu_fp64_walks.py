"""The walks of the FP64 tracer kernels (k64_xy: up to 16 rows, k64_ztail: up to 16 levels, as many as the
grid has blocks for) against the oracle, bit for bit, on grids whose last walk is ragged: with all
water and with land, diffusion and a flux condition on every face, on rectilinear and latitude-longitude
grids, in QuotaMode and IronEnergyMode."""
import numpy as np
import pytest

import oracle
from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._native import CModel
from PlanktonIndividuals.architectures import IronEnergyMode
from PlanktonIndividuals.grids import Bounded, LatLonGrid, Periodic, RectilinearGrid, fill_halo_tracer
from PlanktonIndividuals.init import initialize_plankton_iron
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params
from helpers import compare_states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["water", "land", "latlon", "latlon water", "iron", "iron land", "iron latlon"])
@pytest.mark.parametrize("size", [
    (40, 59, 23),      # 16 rows (the last 11), 16 levels (the last 7)
    (63, 57, 11),      # 8 rows (the last 1), 8 levels (the last 3)
    (33, 37, 9),       # 4 rows (the last 1), 4 levels (the last 1)
    (40, 59, 3),       # 2 rows, 2 levels (the last 1)
])
def test_ragged_walks_identical_to_oracle(gpu_lib, size, kind):
    rng = np.random.default_rng(sum(size))
    general, iron = kind not in ("water", "iron"), "iron" in kind
    lm = rng.random(size) < 0.85 if general and "water" not in kind else np.ones(size, dtype=bool)
    if "latlon" in kind:
        grid = LatLonGrid(size=size, lat=(30.0, 36.0), lon=(-10.0, -4.0), z=(0.0, -10.0 * size[2]), FT=np.float64, landmask=lm)
    else:
        t = Bounded if general else Periodic
        grid = RectilinearGrid(size=size, x=(0.0, size[0] * 50.0), y=(0.0, size[1] * 50.0), z=(0.0, -2.0 * size[2]),
                               FT=np.float64, topology=(t, t, Bounded), landmask=lm)
    mode = {"mode": IronEnergyMode()} if iron else {}
    phyt = update_phyt_params({}, np.float64, N=1, **mode)
    bgc = update_bgc_params({"κh": 1.0, "κv": 1e-3, "κhP": 0.1, "κvP": 1e-4} if general else {}, np.float64)
    C = 600
    inds = [initialize_plankton_iron(grid, phyt, 0, 400, C, rng) if iron else W.make_individuals(grid, phyt, 0, 400, C, rng)]
    trs = W.make_tracers(grid, rng)
    e = [int(c == _abi.PI_BOUNDED) for c in grid.topo]                # faces of a Bounded axis: N + 1
    shapes = [(size[0] + e[0], size[1], size[2]), (size[0], size[1] + e[1], size[2]), (size[0], size[1], size[2] + 1)]
    width = 10000.0 if "latlon" in kind else 50.0                     # Courant numbers up to about 0.4
    vel = [s * rng.standard_normal(n) for s, n in zip((1e-3 * width, 1e-3 * width, 2e-3), shapes)]
    kw = {"mode": "iron"} if iron else {}
    models = [CModel(gpu_lib, "pi_", grid, bgc, phyt, 1, C, 3, precision=_abi.PI_FP64, **kw),
              oracle.OracleModel(grid, bgc, phyt, 1, C, 3, **kw)]
    for m in models:
        m.set_state(inds, trs)
        if general:
            for n, face in enumerate(_abi.FACES):
                m.set_flux_bc(n, _abi.FACES[face], _abi.PI_BC_CONST, [1e-4 * (n + 1)])
        for _ in range(3):
            m.set_velocity(*vel)
            m.set_PARF(np.full(size[:2], 300.0))
            m.set_temp(np.full(size, 25.0))
            m.time_step(60.0)
    assert compare_states(models[1], models[0], 1) == []
    models[0].close()


@pytest.mark.parametrize("land", [False, True])
@pytest.mark.parametrize("odd", ["courant", "zeros", "nonfinite"])
def test_flux_shortcuts_identical_to_oracle(gpu_lib, odd, land):
    """The flux of a face leaves out the side without transport and, where a product decides it, the limiter's
    last quotient: Courant numbers above 1, faces at rest, flat and zero tracers, NaN and infinities."""
    size = (33, 37, 9)
    rng = np.random.default_rng(len(odd))
    lm = rng.random(size) < 0.8 if land else np.ones(size, dtype=bool)
    grid = RectilinearGrid(size=size, x=(0.0, size[0] * 50.0), y=(0.0, size[1] * 50.0), z=(0.0, -2.0 * size[2]),
                           FT=np.float64, topology=(Periodic, Bounded, Bounded), landmask=lm)
    phyt, bgc = update_phyt_params({}, np.float64, N=1), update_bgc_params({}, np.float64)
    inds = [W.make_individuals(grid, phyt, 0, 8, 8, rng)]
    trs = W.make_tracers(grid, rng)
    cfl = 1.5 if odd == "courant" else 0.2
    vel = [cfl * w / 60.0 * rng.standard_normal(n) for w, n in zip((50.0, 50.0, 2.0), (size, (size[0], size[1] + 1, size[2]),
                                                                                       (size[0], size[1], size[2] + 1)))]
    if odd == "zeros":
        vel = [np.where(rng.random(v.shape) < 0.4, rng.choice([0.0, -0.0], v.shape), v) for v in vel]
    for n, t in enumerate(trs):
        hit = rng.random(t.shape) < (0.3 if odd == "zeros" else 0.01)
        if odd == "zeros":
            t[hit] = rng.choice([0.0, 1.0, 1e-310, -1e-3], t.shape)[hit]
        if odd == "nonfinite" and n % 2:
            t[hit] = rng.choice([np.nan, np.inf, -np.inf], t.shape)[hit]
        fill_halo_tracer(t, grid)
    models = [CModel(gpu_lib, "pi_", grid, bgc, phyt, 1, 8, 3, precision=_abi.PI_FP64), oracle.OracleModel(grid, bgc, phyt, 1, 8, 3)]
    for m in models:
        m.set_state(inds, trs)
        for _ in range(2):
            m.set_velocity(*vel)
            m.set_PARF(np.full(size[:2], 300.0))
            m.set_temp(np.full(size, 25.0))
            m.time_step(60.0)
    for n, name in enumerate(_abi.tracer_names):
        a, b = models[1].get_tracer(n), models[0].get_tracer(n)
        assert np.array_equal(a, b, equal_nan=True), (name, int(np.sum(~((a == b) | (np.isnan(a) & np.isnan(b))))))
    models[0].close()
