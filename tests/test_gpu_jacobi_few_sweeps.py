"""Jacobi solves that end after a few sweeps.

All sweeps of a layer at once cost the same however early the iteration ends, so
a solve that is limited to few sweeps, or whose threshold the rewards may already
meet, starts with ordinary sweeps; the sliced copy that only those need tells
which way it went.  Values, policy, iteration count, residual and status of both
ways are the same bit for bit, for results that did not converge too, and for
rewards that are infinite or NaN.
"""
import dataclasses

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200._lib import E2EError
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields

from .helpers import problem

pytestmark = pytest.mark.gpu
SWEEPS = 0x140  # one lean sweep after another
NOT_CONVERGED = 6


def _solve(m, **kw):
    """(status, values, policy, statistics): the outputs of a solve that did not converge too."""
    torch = pytest.importorskip("torch")
    ns = m.info()["ns"]
    V = torch.full((ns,), float("nan"), dtype=torch.float32, device="cuda")
    pi = torch.full((ns,), -9, dtype=torch.int32, device="cuda")
    status, st = 0, {}
    try:
        st = m.solve(method="jacobi", value=V, policy=pi, **kw)[2]
    except E2EError as e:
        status = e.status
    return status, V.cpu().numpy(), pi.cpu().numpy(), st


def _same(m, **kw):
    a, b = _solve(m, **kw), _solve(m, schedule=SWEEPS, **kw)
    assert a[0] == b[0], (kw, a[0], b[0])
    assert a[1].tobytes() == b[1].tobytes() and np.array_equal(a[2], b[2]), kw
    for k in ("iterations", "residual"):
        assert a[3].get(k) == b[3].get(k), (kw, k)
    return a


def _fresh(nt=30):
    prob = Problem(gsize=20, nt=nt, nrzns=60, nmodes=2, num_ac_angles=8, i_term=12, j_term=5, neighb_gsize=9)
    return prob, api.build_model(prob, make_fields(prob, FieldSpec(obstacle_frac=0.05, seed=nt)))


def test_a_threshold_above_the_rewards_takes_one_sweep():
    prob, m = _fresh()
    status, _, _, st = _solve(m, threshold=1e6)
    assert (status, st["iterations"]) == (0, 1)
    assert st["pack_ms"] > 0  # swept
    m.free()


def test_a_limit_of_few_sweeps_sweeps():
    prob, m = _fresh()
    assert _solve(m, threshold=0.1, max_iter=2)[0] == NOT_CONVERGED
    assert m.solve(method="layered")[2]["pack_ms"] == 0.0  # the copy is there: those sweeps made it
    m.free()
    prob, m = _fresh()
    status, _, _, st = _solve(m, threshold=0.1)
    assert status == 0 and st["pack_ms"] == 0.0  # the usual solve: all sweeps of a layer at once
    m.free()


@pytest.mark.parametrize("nt", [3, 4, 8, 30, 70])
def test_both_ways_agree_for_any_limit(nt):
    prob, m = _fresh(nt)
    for thr in (0.1, 1.5, 40.0, 1e6):
        for it in sorted({0, 1, 2, 3, nt // 3, nt // 2, nt - 1, nt, nt + 1}):
            _same(m, threshold=thr, max_iter=it)
    m.free()


@pytest.mark.parametrize("out,term", [(-np.inf, 5.0), (-1.0, -np.inf), (np.nan, 5.0), (-3.0, np.nan)])
def test_infinite_and_nan_rewards(out, term):
    base, fields = problem("t_time")
    m = api.build_model(dataclasses.replace(base, r_outbound=float(out), r_terminal=float(term)), fields)
    for thr in (0.1, 1e6):
        for it in (0, 1, 3, base.nt - 1):
            _same(m, threshold=thr, max_iter=it)
    m.free()


@pytest.mark.parametrize("out,term", [(np.inf, 1.0), (-1.0, np.inf)])
def test_rewards_without_an_upper_bound(out, term):
    # against the backups of unpadded rows: in the sliced copy a row's padding multiplies a
    # value by a weight of zero, which is NaN where the value is infinite
    base, fields = problem("t_time")
    prob = dataclasses.replace(base, r_outbound=float(out), r_terminal=float(term))
    m = api.build_model(prob, fields)
    status, V, pi, _ = _solve(m, threshold=0.1)
    m.free()
    Vf, pif, _ = api.build_solve(prob, fields)
    assert status == 0 and np.isinf(V).any()
    assert np.array_equal(V, Vf) and np.array_equal(pi, pif)
