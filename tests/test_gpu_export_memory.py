"""pi_get_individuals brings the same columns to page-locked and to pageable memory, on both sides of the slot
counts where the way to pageable memory changes (8,192 in the FP32 form, 32,768 in the FP64 form)."""
import ctypes as ct

import numpy as np
import pytest
import torch

from PlanktonIndividuals import _abi
from PlanktonIndividuals._abi import IND_DOUBLE, IND_INT, pi_individuals
from PlanktonIndividuals._native import CModel
from test_gpu_small_models import world

pytestmark = pytest.mark.gpu
NAMES = IND_DOUBLE + IND_INT + ("ac",)


def read(m, C, names, pinned):
    st, out = pi_individuals(), {}
    for k in names:
        dt, cty = {"ac": (torch.uint8, ct.c_uint8)}.get(k, (torch.int64, ct.c_int64) if k in IND_INT else (torch.float64, ct.c_double))
        out[k] = torch.full((C,), 77, dtype=dt, pin_memory=pinned)
        setattr(st, k, ct.cast(out[k].data_ptr(), ct.POINTER(cty)))
    assert m.lib.pi_get_individuals(m.h, 0, ct.byref(st)) == 0
    return {k: v.numpy() for k, v in out.items()}


@pytest.mark.parametrize("precision", [_abi.PI_FP32, _abi.PI_FP64])
@pytest.mark.parametrize("C", [1, 257, 8192, 8193, 32768, 32769])
def test_page_locked_and_pageable_agree(gpu_lib, C, precision):
    w = world((6, 5, 4), max(1, C // 2), C, 31)
    m = CModel(gpu_lib, "pi_", w["grid"], w["bgc"], w["phyt"], 1, C, 1, precision=precision)
    inds = dict(w["inds"][0])
    rng = np.random.default_rng(6)
    for k in ("graz", "mort", "dvid"):
        inds[k] = (rng.random(C) < 0.5) * inds["ac"].astype(np.float64)
    m.set_state([inds], w["trs"])
    for names in (NAMES, ("zi", "mort", "ac"), ("ac",), ("x", "Bm")):
        a, b = read(m, C, names, True), read(m, C, names, False)
        for k in names:
            assert np.array_equal(a[k], b[k]), k
            if k in ("graz", "mort", "dvid", "xi", "yi", "zi", "ac"):
                active = inds["ac"]
                assert np.array_equal(a[k][active], np.asarray(inds[k])[active]), k
    m.close()
