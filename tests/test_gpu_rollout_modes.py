"""The rollout's loads ahead of a step against the oracle, bit for bit: mode counts
around the number loaded ahead, cell spacings with and without a division, and
realisation counts around a warp.  The policies are random, so that vehicles
wander for many steps before an edge or the last layer ends them.
"""
import numpy as np
import pytest

from e2e_gpu_dp_b200 import api
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields
from oracle import rollout as RO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm,nrzns", [(1, 1), (3, 31), (11, 33), (12, 64), (13, 65), (25, 20)])
@pytest.mark.parametrize("dx", [1.0, 0.5, 0.3])
def test_modes_spacings_realisations(nm, nrzns, dx):
    g = 31
    p = Problem(gsize=g, nt=24, nrzns=nrzns, nmodes=nm, num_ac_speeds=2, num_ac_angles=7, i_term=24, j_term=20, neighb_gsize=11,
                dx=dx, dy=dx, dt=dx, prob_type="energy3")
    f = make_fields(p, FieldSpec(A=0.4, sigma0=0.3, obstacle_frac=0.02, scalar=0.3, scalar_wave=0.4, seed=nm))
    pol = np.random.default_rng(nm * 100 + nrzns).integers(0, 14, size=g * g * 24).astype(np.int32)
    r = api.rollout(p, f, pol, (15, 14))
    o = RO.rollout(p, f, pol.astype(np.int64), (15, 14), dot="fma")
    for key in ("success", "travel_time", "final_tij", "energy_cons", "energy_col", "net_energy"):
        assert np.array_equal(r[key], o[key]), key
