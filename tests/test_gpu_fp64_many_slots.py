"""Division lists of the FP64 form above 262,144 slots, where several blocks make them: slot counts around a
block's 65,536 slots and a word's 32, and the capacity error, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._native import CapacityError, CModel
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params
from helpers import compare_states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,N,full", [(262145, 120000, False), (327679, 150000, False), (327680, 100000, False),
                                      (393249, 380000, False), (327681, 300000, True), (262144, 200000, True)])
def test_division_lists_identical_to_oracle(gpu_lib, C, N, full):
    rng = np.random.default_rng(C)
    size = (16, 16, 4)
    grid = RectilinearGrid(size=size, x=(0.0, 800.0), y=(0.0, 800.0), z=(0.0, -8.0), FT=np.float64,
                           topology=(Periodic, Periodic, Bounded))
    over = dict(dvid_P=[1.0 if full else 3e-4], dvid_reg=[0.01 if full else 0.5], mort_P=[2e-4], mort_reg=[1.5], grz_P=[1e-8])
    phyt = update_phyt_params(over, np.float64, N=1)
    bgc = update_bgc_params({}, np.float64)
    inds = [W.make_individuals(grid, phyt, 0, N, C, rng)]
    perm = rng.permutation(C)                  # the individuals lie all over the slots
    inds = [{k: np.ascontiguousarray(np.asarray(v)[perm]) for k, v in inds[0].items()}]
    trs = W.make_tracers(grid, rng)
    models = [CModel(gpu_lib, "pi_", grid, bgc, phyt, 1, C, 3, precision=_abi.PI_FP64),
              oracle.OracleModel(grid, bgc, phyt, 1, C, 3)]
    failed = []
    for m in models:
        m.set_state(inds, trs)
        m.set_velocity(np.zeros(size), np.zeros(size), np.zeros((16, 16, 5)))
        m.set_PARF(np.full(size[:2], 300.0))
        m.set_temp(np.full(size, 25.0))
        n = 0
        try:
            for n in range(3):
                m.time_step(60.0)
        except CapacityError as e:
            failed.append((n, str(e)))
    assert len(failed) == (2 if full else 0) and len(set(failed)) <= 1
    if full:        # a step that stops has taken the decisions off its individuals; their lists are the same
        a, b = (m.get_individuals(0) for m in models)
        assert all(np.array_equal(a[k], b[k]) for k in ("ac", "x", "Bm", "gen"))
    else:
        assert compare_states(models[1], models[0], 1) == []
        assert models[0].count_active(0) != N
    models[0].close()
