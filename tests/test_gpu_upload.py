"""Host fields copied before the builder starts, or in ranges beside it: the same model either way."""
import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields

pytestmark = pytest.mark.gpu


# (megabytes, samples): 7.4 and 1.1e8; 8.5 and 4.5e9; 16.9 and 2.4e8; the general builder: 6 and 13
@pytest.mark.parametrize("nt,nrzns,nm,na,dx,ranges", [(8, 200, 10, 8, 1.0, 1), (8, 4000, 10, 16, 1.0, 3), (19, 200, 10, 8, 1.0, 4),
                                                       (8, 20, 8, 2, 0.3, 1), (18, 20, 8, 2, 0.3, 4)])
def test_ranges_of_an_upload(nt, nrzns, nm, na, dx, ranges):
    torch = pytest.importorskip("torch")
    p = Problem(gsize=100, nt=nt, nrzns=nrzns, nmodes=nm, dx=dx, dy=dx, dt=dx, num_ac_angles=na, i_term=50, j_term=30,
                neighb_gsize=15)
    f = make_fields(p, FieldSpec(A=0.5 * dx, sigma0=0.2 * dx, obstacle_frac=0.03, seed=1))
    host, dev = api.build_model(p, f), api.build_model(p, {k: torch.as_tensor(v).cuda() for k, v in f.items()})
    assert (host.info()["build_launches"], dev.info()["build_launches"]) == (ranges, 1)
    a, b = host.to_host(), dev.to_host()
    host.free(), dev.free()
    assert all(np.array_equal(a[k], b[k]) for k in ("row_ptr", "col", "cnt", "R"))
