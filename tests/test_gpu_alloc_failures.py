"""Calls during which a device allocation is refused.

E2E_TEST_ALLOC_FAIL=lo:hi makes the library's allocator refuse every request of
lo to hi bytes, as a device without that much memory would; nothing is faulted.
A call that cannot go on returns an error and leaves nothing in flight; one that
has a way with less memory takes it and gives the same results.
"""
import os

import numpy as np
import pytest

from e2e_gpu_dp_b200 import _lib, api
from e2e_gpu_dp_b200._lib import E2EError
from e2e_gpu_dp_b200.problem import FieldSpec, Problem, make_fields
from tests.helpers import problem

pytestmark = pytest.mark.gpu
os.environ["E2E_TEST_HOOKS"] = "1"  # read at the library's first allocation


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


def test_jacobi_without_memory_for_the_history_sweeps():
    torch = pytest.importorskip("torch")
    prob = Problem(gsize=9, nt=130, nrzns=40, nmodes=2, num_ac_angles=4, i_term=6, j_term=3, neighb_gsize=9)
    m = api.build_model(prob, make_fields(prob, FieldSpec(obstacle_frac=0.05, seed=2)))
    V = torch.empty(prob.ns, dtype=torch.float32, device="cuda")
    pi = torch.empty(prob.ns, dtype=torch.int32, device="cuda")
    V0, pi0, st0 = m.solve(method="jacobi")
    # everything of the size of the history; then the sizes of one array of values and of the residuals alone
    for lo, hi in ((1 << 20, 1 << 40), (4 * prob.ns, 4 * prob.ns), (8 * (130 + 2 + 130), 8 * (130 + 2 + 130))):
        V.fill_(0), pi.fill_(-5)
        with refuse(lo, hi):
            _, _, st = m.solve(method="jacobi", value=V, policy=pi)
        assert np.array_equal(V.cpu().numpy(), V0) and np.array_equal(pi.cpu().numpy(), pi0)
        assert (st["iterations"], st["residual"]) == (st0["iterations"], st0["residual"])
    m.free()


def test_build_that_fails_keeps_no_memory():
    torch = pytest.importorskip("torch")
    prob, fields = problem("c1")
    staged = prob.num_actions * prob.ncells * (prob.nt - 1) * 4 + 4096  # entries of a first attempt
    api.build_model(prob, fields).free()

    def free_bytes():
        _lib.check(_lib.lib().e2e_memory_trim())
        return torch.cuda.mem_get_info()[0]

    before = free_bytes()
    for _ in range(8):
        with refuse(2 * staged):  # the staged counts, behind the staged columns
            with pytest.raises(E2EError):
                api.build_model(prob, fields)
    assert free_bytes() >= before


@pytest.mark.parametrize("call", ["build_model", "build_solve"])
def test_failed_build_leaves_nothing_in_flight(call):
    torch = pytest.importorskip("torch")
    prob, fields = problem("c1")
    s = torch.cuda.Stream()
    dense = 4 * prob.neighb_gsize ** 2 * min(max(prob.num_actions * prob.ncells * (prob.nt - 1) // 64, 256), 8192)
    with refuse(dense):  # the dense pool: the last buffer before the first launch
        with pytest.raises(E2EError):
            getattr(api, call)(prob, fields, stream=s)
    assert s.query()
    want = api.build_model(prob, fields).to_host()
    got = api.build_model(prob, fields, stream=s).to_host()
    assert all(np.array_equal(want[k], got[k]) for k in ("row_ptr", "col", "cnt", "R"))


@pytest.mark.parametrize("call", ["build_model", "build_solve"])
def test_build_without_memory_for_the_rank_tables(call):
    prob, fields = problem("c1")
    coeffs = 4 * (prob.nt - 1) * (prob.nmodes + prob.nmodes % 2) * (-(-prob.nrzns // 128) * 128)

    def results():
        if call == "build_solve":
            return api.build_solve(prob, fields)[:2]
        h = api.build_model(prob, fields).to_host()
        return [h[k] for k in ("row_ptr", "col", "cnt", "R")]

    want = results()
    with refuse(coeffs):
        got = results()
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("call", ["build_model", "build_solve"])
def test_build_gives_the_rank_tables_back_for_the_other_buffers(call):
    torch = pytest.importorskip("torch")
    prob = Problem(gsize=44, nt=40, nrzns=12000, nmodes=10, num_ac_angles=8, i_term=25, j_term=9, neighb_gsize=15)
    spec = FieldSpec(sigma0=0.1, obstacle_frac=0.04, seed=6)
    fields = {k: torch.as_tensor(v).cuda() for k, v in make_fields(prob, spec).items()}

    def results():
        if call == "build_solve":
            *r, st = api.build_solve(prob, fields)
            return [np.asarray(torch.as_tensor(x).cpu()) for x in r], st["general_tiles"]
        m = api.build_model(prob, fields)
        h, tiles = m.to_host(), m.info()["general_tiles"]
        m.free()
        return [h[k] for k in ("row_ptr", "col", "cnt", "R")], tiles

    want, tiles = results()
    assert tiles < prob.ncells * (prob.nt - 1) // 4
    # 10 MB of staged columns, then a model of less, beside 19 MB of coefficients
    os.environ["E2E_TEST_ALLOC_TOTAL"] = str(24 << 20)
    try:
        got, tiles = results()
    finally:
        os.environ.pop("E2E_TEST_ALLOC_TOTAL", None)
    assert call == "build_solve" or tiles == prob.ncells * (prob.nt - 1) // 4  # (groups of 4 cells)
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


def test_build_solve_without_memory_for_a_block_of_layers():
    torch = pytest.importorskip("torch")
    prob = Problem(gsize=44, nt=40, nrzns=200, nmodes=2, num_ac_angles=8, i_term=25, j_term=9, neighb_gsize=15)
    fields = make_fields(prob, FieldSpec(sigma0=0.1, obstacle_frac=0.04, seed=6))
    *want, st = api.build_solve(prob, fields)
    assert st["launches"] == 2
    # 10 MB of staged columns; with the first range refused three blocks, with the second (not the dense pool's 7.4 MB) five
    for lo, hi, blocks in ((9000000, 1 << 40, 3), (3000000, 7300000, 5)):
        with refuse(lo, hi):
            *got, st = api.build_solve(prob, fields)
        assert st["launches"] == 2 * blocks
        assert all(np.array_equal(a, b) for a, b in zip(want, got))


def test_model_takes_the_place_of_the_rank_tables():
    torch = pytest.importorskip("torch")
    prob = Problem(gsize=44, nt=40, nrzns=12000, nmodes=10, num_ac_angles=8, i_term=25, j_term=9, neighb_gsize=15)
    spec = FieldSpec(sigma0=0.38, obstacle_frac=0.04, seed=6)
    fields = {k: torch.as_tensor(v).cuda() for k, v in make_fields(prob, spec).items()}
    m = api.build_model(prob, fields)
    want, nnz = m.to_host(), m.info()["nnz"]
    m.free()
    assert 4 * nnz > 8 << 20
    # 19 MB of coefficients, the staged columns and the model's
    for over in (0, 4 << 20, 8 << 20):
        os.environ["E2E_TEST_ALLOC_TOTAL"] = str((30 << 20) + over)
        try:
            m = api.build_model(prob, fields)
        finally:
            os.environ.pop("E2E_TEST_ALLOC_TOTAL", None)
        got = m.to_host()
        m.free()
        assert all(np.array_equal(want[k], got[k]) for k in ("row_ptr", "col", "cnt", "R"))


def test_build_solve_without_memory_for_one_layer_beside_the_rank_tables():
    torch = pytest.importorskip("torch")
    prob = Problem(gsize=256, nt=21, nrzns=10600, nmodes=10, num_ac_angles=8, i_term=25, j_term=9, neighb_gsize=15)
    spec = FieldSpec(sigma0=0.1, obstacle_frac=0.04, seed=6)
    fields = {k: torch.as_tensor(v).cuda() for k, v in make_fields(prob, spec).items()}
    *want, st = api.build_solve(prob, fields)
    assert st["general_tiles"] < prob.ncells * (prob.nt - 1) // 4
    # a layer's staged columns and all coefficients, 8.4 and 8.5 MB, in 12 MB
    os.environ.update(E2E_TEST_ALLOC_TOTAL=str(12 << 20), E2E_TEST_STAGE_BYTES="1")
    try:
        *got, st = api.build_solve(prob, fields)
    finally:
        os.environ.pop("E2E_TEST_ALLOC_TOTAL", None)
        os.environ.pop("E2E_TEST_STAGE_BYTES", None)
    assert st["general_tiles"] == prob.ncells * (prob.nt - 1) // 4  # (groups of 4 cells)
    assert all(np.array_equal(a, b) for a, b in zip(want, got))
