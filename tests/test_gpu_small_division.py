"""Division of small segments (one block per segment beside the light) against the lists of large ones,
and the capacity check that stops every segment of a step."""
import numpy as np
import pytest

from PlanktonIndividuals._native import CapacityError
from PlanktonIndividuals.batch import Member, PlanktonBatch
from helpers import compare_states
from test_gpu_small_models import world, stepped
from PlanktonIndividuals.parameters import update_phyt_params

pytestmark = pytest.mark.gpu


# segments below, at and above one tile of bitmap words, around the 8 warps' runs (8 × 1024 slots) and
# up to the largest segment that one block divides (262,144 slots); many divisions every step. The
# other member has 262,145 slots, so the batch builds the lists with the four list kernels.
@pytest.mark.parametrize("N,C", [(20, 1024), (700, 2047), (4000, 8192), (4000, 8193), (9000, 20000), (100000, 262144)])
def test_one_block_division(gpu_lib, N, C):
    over = dict(dvid_P=[5e-3], dvid_reg=[0.5], mort_P=[2e-3], mort_reg=[1.5], grz_P=[1e-6])
    w = world((6, 5, 4), N, C, 11)
    other = world((6, 5, 4), 100, 262145, 12)
    for x in (w, other):
        x["phyt"] = update_phyt_params(over, np.float64, N=1)
    alone, mixed = stepped([w], 4), stepped([w, other], 4)
    bad = compare_states(alone.member(0), mixed.member(0), 1)
    assert not bad, bad[:5]
    assert alone.count_active() != N


# the second member overflows in its first dividing step: no member divides in that step, in either form
@pytest.mark.parametrize("C1", [3000, 262145])
def test_capacity_stops_every_segment(gpu_lib, C1):
    w1, w2 = world((6, 5, 4), 500, C1, 13), world((6, 5, 4), 400, 401, 14)
    for x in (w1, w2):
        x["phyt"] = update_phyt_params(dict(dvid_P=[1e-2], dvid_reg=[0.1], grz_P=[0.0], mort_P=[0.0]), np.float64, N=1)
    b = PlanktonBatch([Member(x["grid"], x["bgc"], x["phyt"], x["C"], x["seed"]) for x in (w1, w2)], nspecies=1)
    for m, x in enumerate((w1, w2)):
        b.set_state(m, x["inds"], x["trs"])
        b.set_series(m, PARF=x["parf"], temp=x["temp"])
    with pytest.raises(CapacityError, match="member 1"):
        b.step(60.0, 5)
    assert b.get_time()[0] == 2                  # decisions of step 1 divide in step 2
    assert b.count_active(0) == 500 and b.count_active(1) == 400
    assert float(np.max(b.get_individuals(0, 0)["gen"])) == 1.0
