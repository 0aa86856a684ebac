"""Calls during which a device allocation is refused.

E2E_TEST_ALLOC_FAIL=lo:hi makes the library's allocator refuse every request of
lo to hi bytes, as a device without that much memory would; nothing is faulted.
A call that cannot go on returns an error and leaves nothing in flight; one that
has a way with less memory takes it and gives the same results.
"""
import os

import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200._lib import E2EError
from tests.helpers import problem

pytestmark = pytest.mark.gpu


class refuse:
    def __init__(self, lo, hi=None):
        self.v = f"{lo}:{lo if hi is None else hi}"

    def __enter__(self):
        os.environ["E2E_TEST_ALLOC_FAIL"] = self.v

    def __exit__(self, *exc):
        os.environ.pop("E2E_TEST_ALLOC_FAIL", None)


@pytest.mark.parametrize("what", ["second values", "residuals"])
def test_solve_that_fails_after_the_sliced_copy_leaves_it_complete(what):
    torch = pytest.importorskip("torch")
    prob, fields = problem("c1")
    m = api.build_model(prob, fields)
    V0, pi0, _ = m.solve(method="layered")
    m.free()
    V = torch.empty(prob.ns, dtype=torch.float32, device="cuda")
    pi = torch.empty(prob.ns, dtype=torch.int32, device="cuda")
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    m = api.build_model(prob, fields)
    with refuse(4 * prob.ns if what == "second values" else 8 * (prob.nt + 2 + 3)):
        with pytest.raises(E2EError):
            m.solve(method="layered", value=V, policy=pi, stream=s1)
    assert s1.query()  # nothing of the failed call is still running
    m.solve(method="layered", value=V, policy=pi, stream=s2)
    assert np.array_equal(V.cpu().numpy(), V0) and np.array_equal(pi.cpu().numpy(), pi0)
    m.free()
