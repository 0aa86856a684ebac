"""The generator's batches of time steps: a step's fields do not depend on the batch it is in."""
import os

import numpy as np
import pytest

from e2e_gpu_dp_b200 import envgen

pytestmark = pytest.mark.gpu
os.environ["E2E_TEST_HOOKS"] = "1"  # read at the library's first allocation
BY_STEP = [k for k in envgen.FILES if k not in ("all_s_mat", "obstacle_mask")]


def _generate(nt, dt):
    return envgen.build_environment_DG_with_westward_clouds(
        init_gsize=4, nt=nt, dt=dt, dxy=0.5, A=0.5, A_sc=3.0, eps=0.1, op_nrzns=10, n_wsamples=16,
        w_range=(np.pi / 10, 8 * np.pi / 10), wx=np.pi, interpolate_degree=2, n_modes=2, dyn_obstacle_data=("None",))


def test_more_steps_than_a_launch_dimension_holds():
    # the times k * 3000 * 2^-10 are exact in both runs
    many, few = _generate(33001, 2.0 ** -10), _generate(12, 3000 * 2.0 ** -10)
    for k in BY_STEP:
        assert np.array_equal(many[k][::3000], few[k]), k
    for k in ("svals_vel", "svals_phi"):
        assert np.array_equal(many[k][::3000], few[k]), k


def test_less_memory_than_one_batch_needs():
    # requests of 1 MB and more are refused: four batches instead of one of 2.5 MB
    whole = _generate(61, 0.25)
    os.environ["E2E_TEST_ALLOC_FAIL"] = f"{1 << 20}:{1 << 40}"
    try:
        parts = _generate(61, 0.25)
    finally:
        os.environ.pop("E2E_TEST_ALLOC_FAIL", None)
    for k in envgen.FILES + ("svals_vel", "svals_phi"):
        assert np.array_equal(whole[k], parts[k]), k


def test_batches_leave_room_for_every_other_buffer():
    # 39 MB of outputs and 126 MB of work arrays: with less memory than that, smaller batches
    make = lambda: envgen.build_environment_DG_with_westward_clouds(
        init_gsize=8, nt=200, dt=0.25, dxy=0.25, A=0.5, A_sc=3.0, eps=0.1, op_nrzns=10, n_wsamples=200,
        w_range=(np.pi / 10, 8 * np.pi / 10), wx=np.pi, interpolate_degree=8, n_modes=4, dyn_obstacle_data=("None",))
    whole = make()
    for mb in range(70, 301, 10):
        os.environ["E2E_TEST_ALLOC_TOTAL"] = str(mb << 20)
        try:
            parts = make()
        finally:
            os.environ.pop("E2E_TEST_ALLOC_TOTAL", None)
        for k in envgen.FILES + ("svals_vel", "svals_phi"):
            assert np.array_equal(whole[k], parts[k]), (mb, k)
