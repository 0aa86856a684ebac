"""The ranked builder against the general one, bit for bit.

Problems of more than ten modes go to the general builder (k_build_tiles), so
the same problem with zero modes appended gives the model to compare: row
pointers, next states, counts, rewards and the dropped-sample counter.  Sizes at
the edges of the ranked builder's blocks (128 realisations, 32 / P cells a warp,
modes padded to even), every reward type, spacings of a power of two, action sets
from 2 to 32, grids smaller than a window, and inputs whose cells it leaves to
the general builder: wide noise, strong drift, infinities and NaN.
"""
import dataclasses

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields

pytestmark = pytest.mark.gpu


def _both(prob, fields):
    out = []
    for p, f in ((prob, fields), _general(prob, fields)):
        m = api.build_model(p, f)
        h = m.to_host()
        h["dropped"] = np.array(m.info()["dropped"])
        out.append(h)
        m.free()
    return out


def _general(prob, fields):
    more = 11 - prob.nmodes
    f = dict(fields)
    for k in ("ui", "vi"):
        f[k] = np.concatenate([fields[k], np.zeros((prob.nt, more, prob.gsize, prob.gsize), np.float32)], axis=1)
    f["Yi"] = np.concatenate([fields["Yi"], np.zeros((prob.nt, prob.nrzns, more), np.float32)], axis=2)
    return dataclasses.replace(prob, nmodes=11), f


def _check(prob, fields):
    r, g = _both(prob, fields)
    for k in ("row_ptr", "col", "cnt", "dropped"):
        assert np.array_equal(r[k], g[k]), k
    assert r["R"].tobytes() == g["R"].tobytes() or np.array_equal(r["R"], g["R"], equal_nan=True)


def _prob(g=23, nt=4, nrzns=200, nm=4, speeds=1, angles=16, **kw):
    m = kw.pop("neighb_gsize", min(21, g if g % 2 else g - 1))
    return Problem(gsize=g, nt=nt, nrzns=nrzns, nmodes=nm, num_ac_speeds=speeds, num_ac_angles=angles, i_term=(2 * g) // 3,
                   j_term=g // 3, neighb_gsize=m, **kw)


@pytest.mark.parametrize("nrzns", [1, 2, 63, 127, 128, 129, 511, 1030])
@pytest.mark.parametrize("nm", [1, 2, 3, 7, 10])
def test_realisations_and_modes(nrzns, nm):
    p = _prob(g=19, nt=3, nrzns=nrzns, nm=nm)
    _check(p, make_fields(p, FieldSpec(A=0.8, sigma_base=1.5, obstacle_frac=0.06, seed=nrzns * 11 + nm)))


@pytest.mark.parametrize("speeds,angles", [(1, 2), (1, 3), (2, 2), (1, 5), (1, 8), (3, 3), (1, 12), (2, 8), (2, 12), (4, 8), (1, 32), (32, 1)])
@pytest.mark.parametrize("F", [1.0, 1.3, 2.5])
def test_action_sets(speeds, angles, F):
    p = _prob(g=22, nt=3, nrzns=150, nm=3, speeds=speeds, angles=angles, F=F, term_subgrid_size=2)
    _check(p, make_fields(p, FieldSpec(A=0.6, obstacle_frac=0.06, seed=7)))


@pytest.mark.parametrize("g", [2, 3, 5, 7, 8, 9, 16, 31, 33, 64])
def test_grids(g):
    p = _prob(g=g, nt=3, nrzns=140, nm=2, angles=8, neighb_gsize=g if g % 2 else g - 1)
    _check(p, make_fields(p, FieldSpec(A=0.9, obstacle_frac=0.08, seed=g)))


@pytest.mark.parametrize("kind", ["time", "energy1", "energy2", "energy3", "custom1"])
@pytest.mark.parametrize("dx,dy,dt", [(1.0, 1.0, 1.0), (0.5, 0.5, 0.5), (2.0, 2.0, 1.5), (0.25, 0.5, 0.3), (0.3, 0.3, 0.3)])
def test_rewards_and_spacings(kind, dx, dy, dt):
    p = _prob(g=21, nt=23, nrzns=90, nm=3, speeds=2, angles=8, dx=dx, dy=dy, dt=dt, F=1.2, prob_type=kind, alpha=0.07,
              r_outbound=-33.7, r_terminal=41.9)
    s = FieldSpec(A=0.5 * dx, sigma0=0.3 * dx, obstacle_frac=0.05, scalar=0.3, scalar_wave=0.4, seed=3)
    _check(p, make_fields(p, s))


@pytest.mark.parametrize("speeds,angles", [(1, 2), (1, 4), (2, 2), (2, 4), (3, 4), (4, 4), (4, 8), (16, 2)])
def test_sequential_sums_of_small_and_many_speed_action_sets(speeds, angles):  # large tables of rewards a CTA
    p = _prob(g=26, nt=5, nrzns=130, nm=4, speeds=speeds, angles=angles, dx=0.5, dy=0.5, dt=0.5, F=1.1, prob_type="energy2")
    _check(p, make_fields(p, FieldSpec(A=0.5, sigma0=0.2, obstacle_frac=0.05, scalar=0.3, scalar_wave=0.4, seed=speeds + angles)))


@pytest.mark.parametrize("m", [1, 3, 5, 9])
def test_small_neighbourhoods(m):  # counted bins outside the m x m neighbourhood
    for dx in (1.0, 0.5):
        p = _prob(g=20, nt=4, nrzns=120, nm=3, angles=8, neighb_gsize=m, dx=dx, dy=dx, dt=dx, prob_type="energy1")
        _check(p, make_fields(p, FieldSpec(A=1.2 * dx, sigma0=0.5 * dx, obstacle_frac=0.05, seed=m)))


@pytest.mark.parametrize("case", ["wide", "drift", "still", "heavy", "inf", "nan", "stop_dt"])
def test_cells_left_to_the_general_builder(case):
    p = _prob(g=24, nt=4, nrzns=300, nm=4, angles=8)
    f = make_fields(p, FieldSpec(A=0.7, sigma0=1.4 if case == "wide" else 0.3, sigma_base=1.5, obstacle_frac=0.04, seed=5))
    if case == "drift":
        f["u"] = f["u"] + np.linspace(-14, 14, 24, dtype=np.float32)[None, None, :]
    elif case == "still":
        for k in ("u", "v", "Yi"):
            f[k] = np.zeros_like(f[k])
    elif case == "heavy":  # a few realisations far out: listed samples, lists that overflow
        f["Yi"][:, ::7] *= 6.0
    elif case == "inf":
        f["Yi"][1, 5, 0] = np.inf
        f["u"][2, 3, 4] = -np.inf
    elif case == "nan":
        f["Yi"][1, 17, 1] = np.nan
        f["v"][0, 9, 9] = np.nan
        f["ui"][2, 0, 4, 5] = np.nan
    elif case == "stop_dt":
        p = dataclasses.replace(p, dt=-1.0)
    _check(p, f)
