"""Small FP32 models take launch shapes of their own (tiles cut into work units, one-pass halo fills of
members with fewer cells than halo points). A member computes the same bits on every one of them:
alone, and in a batch whose other member moves the whole batch to the shapes of large models."""
import numpy as np
import pytest

from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals.batch import Member, PlanktonBatch
from PlanktonIndividuals.grids import Bounded, Periodic, RectilinearGrid
from PlanktonIndividuals.parameters import update_bgc_params, update_phyt_params
from helpers import compare_states

pytestmark = pytest.mark.gpu

OVER = {"dvid_P": [2e-3], "dvid_reg": [1.0], "mort_P": [1e-3], "grz_P": [1e-5]}


def world(size, N, C, seed, topo=(Periodic, Periodic, Bounded)):
    rng = np.random.default_rng(seed)
    grid = RectilinearGrid(size=size, x=(0.0, size[0] * 50.0), y=(0.0, size[1] * 50.0), z=(0.0, -2.0 * size[2]),
                           FT=np.float64, topology=topo)
    phyt = update_phyt_params(OVER, np.float64, N=1)
    ind = W.make_individuals(grid, phyt, 0, N, C, rng)
    return dict(grid=grid, phyt=phyt, bgc=update_bgc_params({}, np.float64), C=C, seed=seed, inds=[ind],
                trs=W.make_tracers(grid, rng), parf=np.full(size[:2] + (1,), 300.0), temp=np.full(size + (1,), 25.0))


def stepped(worlds, steps):
    b = PlanktonBatch([Member(w["grid"], w["bgc"], w["phyt"], w["C"], w["seed"]) for w in worlds], nspecies=1)
    for m, w in enumerate(worlds):
        b.set_state(m, w["inds"], w["trs"])
        b.set_series(m, PARF=w["parf"], temp=w["temp"])
    b.step(60.0, steps)
    return b


# 1 × 1 × 1 and thin members take k32_halo_small alone; beside the 1 × 120 × 30 slice (21,080
# halo-padded cells) the batch takes the three passes. 20 × 7 × 1 is direct alone.
@pytest.mark.parametrize("size,topo", [((1, 1, 1), (Periodic, Periodic, Bounded)), ((1, 9, 5), (Periodic, Periodic, Bounded)),
                                       ((3, 1, 2), (Bounded, Periodic, Bounded)), ((20, 7, 1), (Periodic, Bounded, Bounded)),
                                       ((1, 1, 36), (Periodic, Periodic, Bounded))])
def test_halo_fill_of_thin_members(gpu_lib, size, topo):
    w = world(size, 300, 1500, 5, topo)
    other = world((1, 120, 30), 500, 1100, 6)
    alone, mixed = stepped([w], 7), stepped([w, other], 7)
    bad = compare_states(alone.member(0), mixed.member(0), 1)
    assert not bad, bad[:5]


# one tile, a ragged tile count and a capacity below one tile; beside 1,300,000 slots (1,270 tiles)
# the whole batch works on whole tiles
@pytest.mark.parametrize("N,C", [(1, 1), (700, 1000), (1024, 1025), (3000, 5003)])
def test_work_units_of_few_tiles(gpu_lib, N, C):
    w = world((6, 5, 4), N, C, 7)
    if C < 1.4 * N:                       # no room for divisions
        w["phyt"] = update_phyt_params(dict(OVER, dvid_P=[0.0]), np.float64, N=1)
    other = world((6, 5, 4), 2000, 1300000, 8)
    alone, mixed = stepped([w], 9), stepped([w, other], 9)
    bad = compare_states(alone.member(0), mixed.member(0), 1)
    assert not bad, bad[:5]
    assert alone.count_active() == mixed.count_active(0)
