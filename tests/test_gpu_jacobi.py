"""The Jacobi solve that takes all sweeps of a layer at once against the sweeps
one after another (e2e_vi_opts.schedule with a tuning given): values, policy,
iteration count and residual bit for bit, whatever sweep ends the iteration."""
import dataclasses

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200._lib import E2EError
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields

from .helpers import problem

pytestmark = pytest.mark.gpu
SWEEPS = 0x140  # one lean sweep after another


def _solve(m, **kw):
    try:
        V, pi, st = m.solve(method="jacobi", value=None, **kw)
        return V, pi, st["iterations"], st["residual"]
    except E2EError as e:
        return str(e)


def _same(a, b):
    if isinstance(a, str) or isinstance(b, str):
        return a == b
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("name", ["t_time", "t_custom", "t_energy2", "t_m6", "c1"])
def test_all_sweeps_of_a_layer_at_once(name):
    prob, fields = problem(name)
    m = api.build_model(prob, fields)
    for thr in (0.1, 30.0, 1e-30):
        for it in (0, 1, 2, prob.nt - 1, prob.nt, prob.nt + 1):
            assert _same(_solve(m, threshold=thr, max_iter=it), _solve(m, threshold=thr, max_iter=it, schedule=SWEEPS)), (thr, it)


@pytest.mark.parametrize("nt", [31, 33, 65, 130, 140])  # edges of 32 sweeps a block and 128 a launch
def test_sweep_blocks(nt):
    prob = Problem(gsize=9, nt=nt, nrzns=40, nmodes=2, num_ac_angles=8, i_term=6, j_term=3, neighb_gsize=9)
    m = api.build_model(prob, make_fields(prob, FieldSpec(obstacle_frac=0.05, seed=nt)))
    assert _same(_solve(m, threshold=0.1), _solve(m, threshold=0.1, schedule=SWEEPS))


@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e28])  # values outside the corrected quotient's range
def test_rewards_of_any_size(scale):
    base, fields = problem("t_time")
    prob = dataclasses.replace(base, r_outbound=-100.0 * scale, r_terminal=100.0 * scale, prob_type="custom1", alpha=1.0,
                               F=float(np.sqrt(scale)) if scale < 1 else 1.0)
    m = api.build_model(prob, fields)
    assert _same(_solve(m, threshold=1e-37), _solve(m, threshold=1e-37, schedule=SWEEPS))
