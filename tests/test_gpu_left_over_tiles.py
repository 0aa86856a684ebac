"""Tiles that the ranked builder leaves to the general one, for every shape of the list.

Wide fields leave most tiles, near the grid's edge and inside, of some or of all
layers; the list holds those near the edge from its front and the others from its
back, in groups of 32 / P cells.  The model equals the general builder's alone, bit
for bit (compared as in test_gpu_ranks.py).
"""
import os

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, make_fields

from .test_gpu_ranks import _check, _prob

pytestmark = pytest.mark.gpu
os.environ["E2E_TEST_HOOKS"] = "1"  # read at the library's first allocation


@pytest.mark.parametrize("angles", [2, 3, 4, 8, 16, 32])
@pytest.mark.parametrize("g", [9, 14, 21, 40])  # all cells near the edge; no interior; odd; groups inside rows
def test_wide_fields(g, angles):
    p = _prob(g=g, nt=4, nrzns=70, nm=3, angles=angles, neighb_gsize=9)
    _check(p, make_fields(p, FieldSpec(A=0.7, sigma0=1.5, sigma_base=1.5, obstacle_frac=0.04, seed=g + angles)))


@pytest.mark.parametrize("dx", [1.0, 0.5])
def test_one_layer_of_several(dx):
    p = _prob(g=33, nt=6, nrzns=90, nm=3, angles=8, dx=dx, dy=dx, dt=dx, prob_type="energy2")
    f = make_fields(p, FieldSpec(A=0.5 * dx, sigma0=0.2 * dx, obstacle_frac=0.04, scalar=0.3, seed=5))
    f["Yi"][2] *= 9.0
    f["u"][4, 10:20, 10:20] += np.float32(30.0)  # interior tiles of another
    _check(p, f)


def test_one_re_run_for_rows_without_a_histogram():
    # more dense rows than the pool of a first run has histograms
    p = _prob(g=60, nt=8, nrzns=200, nm=3, angles=16)
    f = make_fields(p, FieldSpec(A=0.7, sigma0=1.6, sigma_base=1.5, obstacle_frac=0.04, seed=1))
    m = api.build_model(p, f)
    info, want = m.info(), m.to_host()
    V, pi, _ = m.solve(method="layered")
    m.free()
    assert info["overflow_units"] > 3 * 8192
    assert info["build_launches"] == 2
    Vf, pif, st = api.build_solve(p, f)
    assert st["launches"] == 3  # two builds, one backup
    assert np.array_equal(Vf, V) and np.array_equal(pif, pi)
    # without memory for the room that those rows may need: a third run with what they did need
    pool = 4 * p.neighb_gsize ** 2 * info["overflow_units"]
    os.environ["E2E_TEST_ALLOC_FAIL"] = f"{4 * info['nnz'] + 1024}:{pool - 1}"
    try:
        m = api.build_model(p, f)
    finally:
        os.environ.pop("E2E_TEST_ALLOC_FAIL", None)
    assert m.info()["build_launches"] == 3
    got = m.to_host()
    m.free()
    assert all(np.array_equal(want[k], got[k]) for k in ("row_ptr", "col", "cnt", "R"))
