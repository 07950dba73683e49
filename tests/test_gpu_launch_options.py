"""The launch-shape options of a batch: every default can be set again, and changes no result."""
import re

import pytest

from PlanktonIndividuals import workloads as W
from PlanktonIndividuals.batch import Member, PlanktonBatch
from helpers import compare_states

pytestmark = pytest.mark.gpu

DEFAULTS = {"move_block": 128, "move_fit": 0, "move_blocks_per_sm": 0, "physiology_block": 128, "physiology_fit": 3,
            "physiology_blocks_per_sm": 0, "xy_rows": 16, "z_levels": 32, "par_warps": 0, "tracer_fused": 0,
            "tracer_fused_levels": 32, "xy_beside_particles": -1}
OTHERS = {"move_block": 256, "move_fit": 3, "move_blocks_per_sm": 2, "physiology_block": 256, "physiology_fit": 2,
          "physiology_blocks_per_sm": 4, "xy_rows": 8, "z_levels": 8, "par_warps": 2, "tracer_fused": 1,
          "tracer_fused_levels": 8, "xy_beside_particles": 1}


def make(capacity=1500):
    wl = W.config2(nx=24, nz=8, N_per_species=600, steps=60, nmodes=8, capacity=capacity)
    b = PlanktonBatch([Member(wl.grid, wl.bgc, wl.phyt, wl.capacity, wl.seed)], nspecies=2)
    b.set_state(0, wl.individuals, wl.tracers)
    b.set_series(0, vels={c: x[..., None] for c, x in zip("uvw", wl.velocity(0))}, ΔT_vel=wl.dT * 1000, PARF=wl.parf,
                 ΔT_PAR=wl.dT_PAR, temp=wl.temp, ΔT_temp=wl.dT_temp)
    return b, wl


def test_every_default_can_be_set_again(gpu_lib):
    a, wl = make()
    b, _ = make()
    a.step(wl.dT, 9)
    for opts, steps in ((OTHERS, 4), (DEFAULTS, 5)):
        for k, v in opts.items():
            b.set_option(k, v)
        b.step(wl.dT, steps)
    assert compare_states(a.member(0), b.member(0), 2) == []


@pytest.mark.parametrize("capacity", [1500, 270000])       # division in one block, and by tiles
def test_autotune_report_is_well_formed(gpu_lib, capacity):
    b, wl = make(capacity)
    lines = b.autotune(wl.dT, steps_per_candidate=1).splitlines()
    assert len(lines) == 12 and lines[-1].startswith("tracer path = ")
    for line in lines[:-1]:
        assert re.fullmatch(r"[^=:]+( \([^)]*\))?(: not used| = \d+ \(\d+\.\d{4} ms( per step)?\))", line), line
    unused = [line for line in lines if line.endswith(": not used")]
    assert any(line.startswith("assign block") for line in unused) == (capacity == 1500)
