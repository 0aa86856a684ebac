"""Which builder took a problem (e2e_model_info.general_tiles), and rules that only decide that.

The comparisons of the ranked builder with the general one (test_gpu_ranks.py)
say something where the first really was ranked: the action sets, spacings and
fields that it takes, those that it refuses whole, and those of which it leaves
some cells.
"""
import dataclasses

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, make_fields

from .test_gpu_ranks import _check, _general, _prob

pytestmark = pytest.mark.gpu


def _tiles(p, f):
    """(groups of cells that the general builder built, all groups)"""
    lanes = 1
    while lanes < p.num_actions:
        lanes *= 2
    m = api.build_model(p, f)
    n = m.info()["general_tiles"]
    m.free()
    st = api.build_solve(p, f)[2]
    assert st["general_tiles"] == n
    return n, (p.nt - 1) * -(-p.ncells // (32 // lanes))


def _fields(p, **kw):
    return make_fields(p, FieldSpec(**{**dict(A=0.6 * p.dx, sigma0=0.3 * p.dx, obstacle_frac=0.05, seed=7), **kw}))


@pytest.mark.parametrize("speeds,angles,F", [(1, 2, 1.3), (1, 8, 1.0), (1, 12, 1.3), (1, 16, 1.0), (2, 8, 2.5), (2, 12, 1.0),
                                              (4, 8, 1.0), (1, 32, 1.0), (32, 1, 1.0)])
@pytest.mark.parametrize("nm", [3, 10])
def test_action_sets_taken(speeds, angles, F, nm):
    p = _prob(g=40, nt=3, nrzns=150, nm=nm, speeds=speeds, angles=angles, F=F)
    n, total = _tiles(p, _fields(p))
    assert n < total // 4


@pytest.mark.parametrize("kind,dx,dt", [("time", 0.5, 0.5), ("energy2", 0.5, 0.5), ("custom1", 2.0, 1.5)])
def test_spacings_taken(kind, dx, dt):
    p = _prob(g=40, nt=5, nrzns=90, nm=3, speeds=2, angles=8, dx=dx, dy=dx, dt=dt, F=1.2, prob_type=kind, alpha=0.07)
    n, total = _tiles(p, _fields(p, scalar=0.3))
    assert n < total // 2  # (rows whose landings lie beyond the reward tables too)


@pytest.mark.parametrize("change", [dict(nm=11), dict(dx=0.3, dy=0.3, dt=0.3), dict(angles=32, F=1.3), dict(dt=-1.0),
                                    dict(speeds=2, dx=0.25, dy=0.25, dt=0.3, F=1.2, prob_type="energy3")])
def test_problems_refused_whole(change):
    p = _prob(**{**dict(g=20, nt=3, nrzns=60, nm=3, angles=8), **change})
    n, total = _tiles(p, _fields(p))
    assert n == total


@pytest.mark.parametrize("case", ["wide", "drift", "inf", "nan"])
def test_cells_left_over(case):
    p = _prob(g=24, nt=4, nrzns=300, nm=4, angles=8)
    f = make_fields(p, FieldSpec(A=0.7, sigma0=1.4 if case == "wide" else 0.3, sigma_base=1.5, obstacle_frac=0.04, seed=5))
    if case == "drift":
        f["u"] = f["u"] + np.linspace(-14, 14, 24, dtype=np.float32)[None, None, :]
    elif case == "inf":
        f["u"][2, 3, 4] = -np.inf
    elif case == "nan":
        f["ui"][2, 0, 4, 5] = np.nan
    n, total = _tiles(p, f)
    assert 0 < n < total
    if case in ("inf", "nan"):
        assert n < total // 4


# Time rewards of a power of two's multiples: the sums are the same in any order, and the
# counts are folded, as long as they stay below 2^24 units (here of 1/2: up to 20686
# realisations).  Layers with and without the late reward.
@pytest.mark.parametrize("dx,dt,out,term", [(0.5, 0.5, -100.0, 100.0), (2.0, 2.0, -100.0, 100.0), (0.5, 0.5, -33.7, 41.9)])
def test_order_free_time_rewards(dx, dt, out, term):
    p = _prob(g=21, nt=24, nrzns=130, nm=3, speeds=2, angles=4, dx=dx, dy=dx, dt=dt, r_outbound=out, r_terminal=term)
    f = _fields(p, A=0.9 * dx)
    _check(p, f)
    n, total = _tiles(p, f)
    assert n < total // 2


@pytest.mark.parametrize("nrzns", [20680, 20700])
def test_sums_on_both_sides_of_the_exact_range(nrzns):
    p = _prob(g=9, nt=3, nrzns=nrzns, nm=2, angles=4, dx=0.5, dy=0.5, dt=0.5, neighb_gsize=9)
    f = _fields(p, A=0.5)
    _check(p, f)
    n, total = _tiles(p, f)
    assert n < total // 2


@pytest.mark.parametrize("kind", ["energy2", "custom1"])
@pytest.mark.parametrize("where", ["Yi", "u", "ui"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38])
def test_sequential_sums_with_values_that_are_not_finite(kind, where, value):
    p = _prob(g=21, nt=4, nrzns=90, nm=3, angles=8, dx=0.5, dy=0.5, dt=0.5, F=1.1, prob_type=kind, alpha=0.07)
    f = _fields(p, scalar=0.3)
    at = {"Yi": (1, 17, 1), "u": (1, 9, 9), "ui": (1, 0, 3, 4)}[where]
    f[where][at] = np.float32(value)
    _check(p, f)


def test_models_of_both_builders_have_the_same_size():
    p = _prob(g=24, nt=4, nrzns=100, nm=4, angles=8)
    f = _fields(p)
    q, h = _general(p, f)
    a, b = api.build_model(p, f), api.build_model(q, h)
    assert a.info()["nnz"] == b.info()["nnz"]
    assert a.info()["general_tiles"] < b.info()["general_tiles"]
    a.free(), b.free()
    assert dataclasses.replace(q, nmodes=p.nmodes) == p
