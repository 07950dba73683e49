"""pi_batch_get_individuals and the FP64 form's pi_get_individuals write their columns on the device: any subset of columns, separate or adjacent
arrays, one chunk or several, against the upload (logical order) and against each other."""
import ctypes as ct

import numpy as np
import pytest

from PlanktonIndividuals import _abi, workloads as W
from PlanktonIndividuals._abi import IND_DOUBLE, IND_INT, pi_individuals
from PlanktonIndividuals._native import CModel
from PlanktonIndividuals.batch import Member, PlanktonBatch
from test_gpu_small_models import world, stepped

pytestmark = pytest.mark.gpu


def read(b, m, names, adjacent=False, C=None):
    C = C or b.members[m].capacity
    st, out = pi_individuals(), {}
    block = np.empty((len(names), C))
    for q, k in enumerate(names):
        a = block[q] if adjacent else np.empty(C)
        if k in IND_INT:
            a = a.view(np.int64)
            setattr(st, k, a.ctypes.data_as(ct.POINTER(ct.c_int64)))
        elif k == "ac":
            a = np.empty(C, np.uint8)
            st.ac = a.ctypes.data_as(ct.POINTER(ct.c_uint8))
        else:
            setattr(st, k, a.ctypes.data_as(ct.POINTER(ct.c_double)))
        out[k] = a
    assert b.lib.pi_batch_get_individuals(b.h, m, 0, ct.byref(st)) == 0
    return out


@pytest.mark.parametrize("N,C", [(1, 1), (200, 257), (3000, 5000), (600000, 600001)])     # the last in two chunks
def test_upload_and_download_agree(gpu_lib, N, C):
    w = world((6, 5, 4), N, C, 21)
    b = PlanktonBatch([Member(w["grid"], w["bgc"], w["phyt"], C, 1)], nspecies=1)
    b.set_state(0, w["inds"], w["trs"])
    got = b.get_individuals(0, 0)
    for k in IND_DOUBLE:
        want = w["inds"][0][k].astype(np.float32).astype(np.float64)
        if k in "xyz":
            assert np.max(np.abs(got[k] - w["inds"][0][k])) <= 2.0 ** -24
        elif k == "Sz":
            p = w["phyt"]
            cq = np.float32(p["Cquota"][0]) * np.float32(p["Nsuper"][0])
            assert np.array_equal(got[k], (w["inds"][0]["Bm"].astype(np.float32) / cq).astype(np.float64))
        else:
            assert np.array_equal(got[k], want), k
    assert np.array_equal(got["ac"], w["inds"][0]["ac"])


@pytest.mark.parametrize("names", [("x",), ("ac",), ("Bm", "ac"), ("xi", "zi"), ("z", "Pq", "dvid", "yi", "ac"),
                                   IND_DOUBLE + IND_INT + ("ac",)])
def test_column_subsets(gpu_lib, names):
    b = stepped([world((6, 5, 4), 3000, 5000, 22)], 6)
    full = b.get_individuals(0, 0)
    for adjacent in (False, True):
        got = read(b, 0, names, adjacent)
        for k in names:
            assert np.array_equal(got[k], full[k].astype(got[k].dtype)), k


@pytest.mark.parametrize("N,C", [(1, 1), (200, 257), (600000, 600001)])                    # the last in two chunks
def test_fp64_upload_and_download_agree(gpu_lib, N, C):
    w = world((6, 5, 4), N, C, 23)
    m = CModel(gpu_lib, "pi_", w["grid"], w["bgc"], w["phyt"], 1, C, 1, precision=_abi.PI_FP64)
    rng = np.random.default_rng(5)
    inds = dict(w["inds"][0])
    for k in ("graz", "mort", "dvid"):
        inds[k] = (rng.random(C) < 0.5).astype(np.float64)
    m.set_state([inds], w["trs"])
    got = m.get_individuals(0)
    for k in ("graz", "mort", "dvid", "xi", "yi", "zi", "ac"):
        assert np.array_equal(got[k], inds[k]), k
