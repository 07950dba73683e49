"""The FP64 form's cell lists and division lists at the sizes where their kernels change: crowded cells
(k64_order up to 2,048 individuals, k64_order_big above), slot counts around warp words and block
runs. Same bits as the oracle after steps with divisions, deaths and grazing."""
import numpy as np
import pytest

import oracle
from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._native import CModel
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params
from helpers import compare_states

pytestmark = pytest.mark.gpu


def run(lib, size, N, C, nsp, steps=5, over=None):
    rng = np.random.default_rng(N + C)
    grid = RectilinearGrid(size=size, x=(0.0, size[0] * 50.0), y=(0.0, size[1] * 50.0), z=(0.0, -2.0 * size[2]),
                           FT=np.float64, topology=(Periodic, Periodic, Bounded))
    over = over or dict(dvid_P=[3e-3], dvid_reg=[0.5], mort_P=[2e-3], mort_reg=[1.5], grz_P=[1e-7])
    phyt = update_phyt_params({k: v * nsp for k, v in over.items()}, np.float64, N=nsp)
    bgc = update_bgc_params({"κhP": 1.0e-2, "κvP": 1.0e-4}, np.float64)
    inds = [W.make_individuals(grid, phyt, s, N, C, rng) for s in range(nsp)]
    trs = W.make_tracers(grid, rng)
    models = [CModel(lib, "pi_", grid, bgc, phyt, nsp, C, 3, precision=_abi.PI_FP64),
              oracle.OracleModel(grid, bgc, phyt, nsp, C, 3)]
    for m in models:
        m.set_state(inds, trs)
        for _ in range(steps):
            m.set_velocity(np.zeros(size), np.zeros(size), np.zeros((size[0], size[1], size[2] + 1)))
            m.set_PARF(np.full(size[:2], 300.0))
            m.set_temp(np.full(size, 25.0))
            m.time_step(60.0)
    # a periodic axis with fewer cells than halo points has halos of its own (the interior counts there)
    bad = [b for b in compare_states(models[1], models[0], nsp) if not b.startswith("tracer")]
    assert not bad, bad[:5]
    inner = tuple(slice(2, 2 + n) for n in size) if min(size[:2]) < 2 else slice(None)
    for n in range(_abi.NTRACERS):
        assert np.array_equal(models[0].get_tracer(n)[inner], models[1].get_tracer(n)[inner]), n
    assert models[0].count_active(0) != int(inds[0]["ac"].sum())


@pytest.mark.parametrize("size,N,C,nsp", [
    ((1, 1, 1), 2270, 4000, 1),            # about 2,043 + daughters: crosses ORDER_BIG during the run
    ((1, 1, 1), 5000, 9000, 2),            # one crowded cell, two species
    ((2, 1, 3), 9000, 20000, 2),           # several crowded cells
    ((7, 5, 3), 31, 33, 1), ((7, 5, 3), 1000, 1503, 3), ((5, 4, 2), 20000, 32768, 1), ((5, 4, 2), 20000, 32801, 1),
])
def test_fp64_lists_identical_to_oracle(gpu_lib, size, N, C, nsp):
    over = dict(dvid_P=[0.0], mort_P=[2e-3], mort_reg=[1.5], grz_P=[1e-5]) if C < 1.2 * N else None
    run(gpu_lib, size, N, C, nsp, over=over)


def test_fp64_daughters_of_a_large_species(gpu_lib):
    """Above DIVIDE_INBLOCK slots the daughters have their own kernel."""
    run(gpu_lib, (16, 16, 4), 150000, 262145, 1, steps=3)
