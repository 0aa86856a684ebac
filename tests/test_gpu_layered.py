"""The default layered schedule (loads ahead of the barrier) against the schedule
of one warp a chunk, bit for bit: values, policy and residual.  Action counts
around the warps' shares, layers of one partial chunk up to several rounds of
chunks a CTA, rows longer than a batch of entries.
"""
import pytest
import torch

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "g,nt,speeds,angles,spread",
    [(2, 3, 1, 2, 0.3), (5, 4, 1, 1, 0.5), (6, 5, 1, 3, 0.5), (23, 7, 1, 5, 0.5), (23, 6, 1, 13, 1.6), (40, 6, 1, 31, 0.5),
     (40, 5, 4, 8, 1.6), (40, 4, 2, 11, 0.5), (70, 4, 2, 12, 1.6), (190, 4, 1, 16, 0.5), (330, 3, 2, 4, 0.5), (330, 3, 1, 17, 0.5)],
)
def test_default_schedule(g, nt, speeds, angles, spread):
    p = Problem(gsize=g, nt=nt, nrzns=150, nmodes=3, num_ac_speeds=speeds, num_ac_angles=angles, i_term=(2 * g) // 3,
                j_term=g // 3, neighb_gsize=min(21, g if g % 2 else g - 1))
    m = api.build_model(p, make_fields(p, FieldSpec(A=0.7, sigma0=spread, obstacle_frac=0.05, seed=g)))
    out = []
    for schedule in (0, 0x101):
        V, pi, st = m.solve(method="layered", schedule=schedule)
        out.append((torch.as_tensor(V).view(torch.int32).clone(), torch.as_tensor(pi).clone(), st["residual"]))
    m.free()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]) and out[0][2] == out[1][2]
