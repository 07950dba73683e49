"""Crowded cells of the FP64 form, bit for bit against the oracle: cells around ORDER_CELL (64) individuals,
where the lists and the particle terms go from a thread per individual or cell to a block and a warp per
cell, cells sorted in shared memory and, above 8,192 individuals, through windows of the slots (262,144
each), with one and several species, losses in crowded cells, and IronEnergyMode."""
import numpy as np
import pytest

import oracle
from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._native import CModel
from PlanktonIndividuals.architectures import IronEnergyMode
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.init import initialize_plankton_iron
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params
from helpers import compare_states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,N,C,nsp,iron", [
    ((4, 4, 2), 2050, 4000, 1, False),         # 64 per cell, more and less
    ((4, 4, 2), 700, 1403, 3, False), ((4, 4, 2), 1300, 2600, 2, True),
    ((8, 4, 1), 4100, 8200, 1, False),         # 128 per cell
    ((2, 2, 2), 8180, 16400, 1, False),        # around 1,024 per cell
    ((1, 1, 1), 8190, 16400, 1, False),        # crosses 8,192
    ((2, 1, 2), 40000, 270000, 1, False), ((2, 1, 2), 21000, 150000, 2, True),     # two windows of slots
])
def test_crowded_cells_identical_to_oracle(gpu_lib, size, N, C, nsp, iron):
    rng = np.random.default_rng(N + C)
    grid = RectilinearGrid(size=size, x=(0.0, size[0] * 50.0), y=(0.0, size[1] * 50.0), z=(0.0, -2.0 * size[2]),
                           FT=np.float64, topology=(Periodic, Periodic, Bounded))
    over = dict(dvid_P=[3e-3], dvid_reg=[0.5], mort_P=[2e-3], mort_reg=[1.5], grz_P=[1e-6])
    phyt = update_phyt_params({k: v * nsp for k, v in over.items()}, np.float64, N=nsp, **({"mode": IronEnergyMode()} if iron else {}))
    bgc = update_bgc_params({"κhP": 1.0e-2, "κvP": 1.0e-4}, np.float64)
    inds = [initialize_plankton_iron(grid, phyt, s, N, C, rng) if iron else W.make_individuals(grid, phyt, s, N, C, rng)
            for s in range(nsp)]
    for d in inds:                             # the individuals lie all over the slots
        perm = rng.permutation(C)
        for k in d:
            d[k] = np.ascontiguousarray(np.asarray(d[k])[perm])
    trs = W.make_tracers(grid, rng)
    kw = {"mode": "iron"} if iron else {}
    models = [CModel(gpu_lib, "pi_", grid, bgc, phyt, nsp, C, 3, precision=_abi.PI_FP64, **kw),
              oracle.OracleModel(grid, bgc, phyt, nsp, C, 3, **kw)]
    for m in models:
        m.set_state(inds, trs)
        for _ in range(4):
            m.set_velocity(np.zeros(size), np.zeros(size), np.zeros((size[0], size[1], size[2] + 1)))
            m.set_PARF(np.full(size[:2], 300.0))
            m.set_temp(np.full(size, 25.0))
            m.time_step(60.0)
    # a periodic axis with fewer cells than halo points has halos of its own (the interior counts there)
    assert [b for b in compare_states(models[1], models[0], nsp) if not b.startswith("tracer")] == []
    inner = tuple(slice(2, 2 + n) for n in size) if min(size[:2]) < 2 else slice(None)
    for n in range(_abi.NTRACERS):
        assert np.array_equal(models[0].get_tracer(n)[inner], models[1].get_tracer(n)[inner]), n
    assert models[0].count_active(0) != N
    models[0].close()
