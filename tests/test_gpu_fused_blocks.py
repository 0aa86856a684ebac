"""build+solve over several blocks of layers (E2E_TEST_STAGE_BYTES sets a block's staging).

One block holds every layer of a small problem.  Larger ones take several: the
staging is reused behind the backup of the block before, a block's counters are read
with the error word of that backup, buffers grow in a later block, and the values
carry from one launch to the next.  Whatever the blocks, values, policy and counts
are those of a stored model.
"""
import os

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200._lib import E2EError
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields
from tests.helpers import problem

pytestmark = pytest.mark.gpu
E2E_ERR_DEVICE = 8


class layers_per_block:
    """Staging for n layers of p, and with unreachable waits the limit of one wait."""

    def __init__(self, p, n, unreachable=False):
        rows = p.ncells * p.num_actions
        self.env = {"E2E_TEST_STAGE_BYTES": str(rows * (4 + 4 + 4 * 6) * n)}
        if unreachable:
            self.env.update(E2E_TEST_UNREACHABLE_WAIT="1", E2E_WAIT_LIMIT_MS="50")

    def __enter__(self):
        os.environ.update(self.env)

    def __exit__(self, *exc):
        for k in self.env:
            os.environ.pop(k, None)


def _blocks(p, n):
    """Number of blocks of at most n layers, of about equal size."""
    layers = p.nt - 1
    count = -(-layers // n)
    size = -(-layers // count)
    return -(-layers // size)


def _same(p, fields, n):
    m = api.build_model(p, fields)
    info = m.info()
    V, pi, _ = m.solve(method="layered")
    m.free()
    with layers_per_block(p, n):
        Vf, pif, st = api.build_solve(p, fields)
    assert np.array_equal(Vf, V) and np.array_equal(pif, pi)
    assert (st["n_rows"], st["nnz"], st["dropped"]) == (info["n_rows"], info["nnz"], info["dropped"])
    assert st["overflow_rows"] == info["overflow_units"] and st["general_tiles"] == info["general_tiles"]
    return st


@pytest.mark.parametrize("name", ["t_time", "t_custom", "t_energy2", "t_wide", "t_m10", "t_m6", "t_half", "c1"])
@pytest.mark.parametrize("n", [1, 2, 5])
def test_blocks(name, n):
    p, fields = problem(name)
    st = _same(p, fields, n)
    # a build and a backup a block, and builds run again with larger buffers
    assert st["launches"] >= 2 * _blocks(p, n)
    if name not in ("t_wide",):
        assert st["launches"] == 2 * _blocks(p, n)


@pytest.mark.parametrize("n", [1, 3])
def test_buffers_that_grow_in_a_later_block(n):
    # the layers are built from the last to the first: quiet ones, then wide ones whose rows
    # need more entries and more dense histograms than the first block was given
    p = Problem(gsize=48, nt=10, nrzns=150, nmodes=3, num_ac_angles=16, i_term=30, j_term=11, neighb_gsize=21)
    fields = make_fields(p, FieldSpec(A=0.6, sigma_base=1.5, obstacle_frac=0.04, seed=9))
    fields["Yi"][:4] *= 8.0
    st = _same(p, fields, n)
    assert st["launches"] > 2 * _blocks(p, n) and st["overflow_rows"] > 0


def test_a_wait_of_any_block_that_runs_out():
    p, fields = problem("t_custom")
    want = api.build_solve(p, fields)[:2]
    with layers_per_block(p, 2, unreachable=True):
        with pytest.raises(E2EError) as e:
            api.build_solve(p, fields)
    assert e.value.status == E2E_ERR_DEVICE
    with layers_per_block(p, 2):
        got = api.build_solve(p, fields)[:2]
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
