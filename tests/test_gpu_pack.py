"""The sliced copy taken chunk by chunk (9 to 32 actions) through the solve that
reads it, against the Jacobi iteration over the CSR rows to its fixed point, bit
for bit: action counts at the rule's edges, partial chunks, layers smaller than a
chunk, an odd number of entries, and chunks with more entries than the copy's
shared memory holds (a calm half of the grid keeps the average low).
"""
import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angles", [8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("g,calm", [(5, False), (8, False), (23, False), (40, True)])
def test_chunks(g, calm, angles):
    p = Problem(gsize=g, nt=6, nrzns=300, nmodes=3, num_ac_speeds=1, num_ac_angles=angles, i_term=(2 * g) // 3, j_term=g // 3,
                neighb_gsize=min(21, g if g % 2 else g - 1))
    f = make_fields(p, FieldSpec(A=0.8, sigma0=1.5 if calm else 0.5, obstacle_frac=0.05, seed=g + angles))
    if calm:
        for k in ("ui", "vi"):
            f[k][:, :, : (3 * g) // 4] = 0
    m = api.build_model(p, f)
    V, pi, _ = m.solve(method="layered")
    Vj, pij, _ = m.solve(method="jacobi", threshold=1e-30)
    m.free()
    assert np.array_equal(np.asarray(V).view(np.int32), np.asarray(Vj).view(np.int32))
    assert np.array_equal(np.asarray(pi), np.asarray(pij))
