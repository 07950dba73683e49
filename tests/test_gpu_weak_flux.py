"""Boundary fluxes of the FP32 form enter the tendency, as apply_bcs! does (Biogeochemistry/apply_bcs.jl:4-98,
before apply_tendency!): an increment per step far below half an ulp of the tracer (4.8e-7 at 8..16) still
adds up beside advection, instead of being rounded away on the tracer. The mass that a flux adds is the
difference of two runs with and without it, against the same difference in Float64.

Tolerance: every cell and step of the two runs rounds once by up to half an ulp, evenly spread beside the
advection (changes of 0.1 and more): sqrt(2·cells·steps)·ulp/sqrt(12) = 3.5e-4 against a gain of 6e-2, below
1 %; 5 % is eight times that."""
import numpy as np
import pytest

from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._native import CModel
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params

pytestmark = pytest.mark.gpu
STEPS, SIZE, DT = 200, (32, 32, 4), 60.0
DOC = _abi.tracer_names.index("DOC")


def mass(lib, grid, inds, trs, vel, precision, flux, face, diffusion):
    phyt = update_phyt_params({}, np.float64, N=1)
    bgc = update_bgc_params({"κh": 1e-3} if diffusion else {}, np.float64)
    m = CModel(lib, "pi_", grid, bgc, phyt, 1, 8, 3, precision=precision)
    m.set_state(inds, trs)
    if flux:
        m.set_flux_bc(DOC, _abi.FACES[face], _abi.PI_BC_CONST, [flux])
    m.set_velocity0(*vel)
    m.set_velocity(*vel)
    m.set_PARF(np.full(SIZE[:2], 300.0))
    m.set_temp(np.full(SIZE, 25.0))
    for _ in range(STEPS):
        m.time_step(DT)
    inner = tuple(slice(h, h + n) for h, n in zip((grid.Hx, grid.Hy, grid.Hz), SIZE))
    total = float(np.sum(m.get_tracer(DOC)[inner]))
    m.close()
    return total


@pytest.mark.parametrize("face,diffusion", [("bottom", False), ("bottom", True), ("top", False), ("south", False)])
def test_flux_below_an_ulp_adds_up(gpu_lib, face, diffusion):
    rng = np.random.default_rng(5)
    topo = (Periodic, Bounded, Bounded)
    grid = RectilinearGrid(size=SIZE, x=(0.0, SIZE[0] * 50.0), y=(0.0, SIZE[1] * 50.0), z=(0.0, -2.0 * SIZE[2]),
                           FT=np.float64, topology=topo)
    inds = [W.make_individuals(grid, update_phyt_params({}, np.float64, N=1), 0, 8, 8, rng)]
    inds[0]["ac"][:] = False                                     # tracers only
    trs = W.make_tracers(grid, rng)
    trs[DOC][...] = rng.uniform(9.0, 14.0, trs[DOC].shape)
    # a flow that differs from row to row, along x only: the tracer changes in every cell, no mass crosses a wall
    vel = [np.broadcast_to(rng.uniform(0.1, 0.3, (1, SIZE[1], SIZE[2])), SIZE).copy(),
           np.zeros((SIZE[0], SIZE[1] + 1, SIZE[2])), np.zeros((SIZE[0], SIZE[1], SIZE[2] + 1))]
    cells = SIZE[0] * (SIZE[2] if face == "south" else SIZE[1])
    width = 50.0 if face == "south" else 2.0                     # of a cell across the face
    step = 6e-2 / (cells * STEPS)                                # increment of a boundary cell per step
    assert step < 3e-7 or face == "south"
    flux = step * width / DT * (-1.0 if face == "top" else 1.0)
    gain = [mass(gpu_lib, grid, inds, trs, vel, p, flux, face, diffusion) - mass(gpu_lib, grid, inds, trs, vel, p, 0.0, face, diffusion)
            for p in (_abi.PI_FP32, _abi.PI_FP64)]
    assert gain[1] > 0.05
    assert abs(gain[0] - gain[1]) <= 0.05 * gain[1], gain
