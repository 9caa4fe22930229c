"""The residual slots of the diagnostics block belong to the last solve that used them: a solve
that does not log reads zero there, whatever logged before it and on whichever route."""
import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev

pytestmark = pytest.mark.gpu

STAGES, LAST = slice(6, 12), slice(12, 14)  # include/oracle_b200.h, OB_DIAG_*


def _plan(prec, nx=48, ny=40, nz=9, **kw):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    return Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                         projection=True, autotune=False, **kw))


def _fields(p, seed=3):
    rng = np.random.default_rng(seed)
    f = [rng.standard_normal((*p.shape[:2], n)) for n in (p.shape[2],) * 2 + (p.shape[2] + 1,)]
    f[2][:, :, 0] = f[2][:, :, -1] = 0.0
    return [dev(a, p.dtype) for a in f]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("forms", ["plane", "lines"])
def test_an_unlogged_projection_clears_what_a_solve_logged(prec, forms):
    p = _plan(prec)
    p.set_variants(z_yz=int(forms == "plane"))
    u, v, w = _fields(p)
    phi = torch.empty_like(u)
    p.project(u.clone(), v.clone(), w.clone(), phi)  # the first one logs
    for logged in (lambda: p.poisson_solve(u, log_diag=True),
                   lambda: p.project(u.clone(), v.clone(), w.clone(), phi, log_diag=True)):
        p.project(u.clone(), v.clone(), w.clone(), phi)
        assert not p.read_diag()[LAST].any()
        logged()
        assert p.read_diag()[LAST].any()
        p.poisson_solve(u)  # a bare solve that does not log leaves the slots alone
        assert p.read_diag()[LAST].any()
        p.project(u.clone(), v.clone(), w.clone(), phi)
        assert not p.read_diag()[LAST].any()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_an_unlogged_projection_clears_what_a_replayed_graph_logged(prec):
    p = _plan(prec)
    a = _fields(p)
    b = [torch.empty_like(x) for x in a] + [torch.empty_like(a[0])]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        p.project_to(*a, *b, log_diag=True)  # kernels loaded before the recording
        logs, quiet = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
        stream.synchronize()
        with torch.cuda.graph(logs, stream=stream):
            p.project_to(*a, *b, log_diag=True)
        with torch.cuda.graph(quiet, stream=stream):
            p.project_to(*a, *b)
        for _ in range(2):
            p.project_to(*a, *b)
            assert not p.read_diag()[LAST].any()
            logs.replay()
            assert p.read_diag()[LAST].any()
            p.project_to(*a, *b)
            assert not p.read_diag()[LAST].any()
            logs.replay()
            quiet.replay()
            assert not p.read_diag()[LAST].any()
    del logs, quiet
    torch.cuda.synchronize()


def test_a_step_graph_clears_the_slots_of_its_own_solves_only():
    # buoyancy and projection alone: a step solves in its three stages, not for the state itself
    p = _plan("fp64", buoyancy=True, poisson_diag_every=1)
    u, v, w = _fields(p)
    s = [u, v, w, torch.ones_like(u), torch.zeros_like(u)]
    ptr = p.state_ptrs(*s)
    p.project(u, v, w, s[4], log_diag=True)
    p.step(ptr, ptr, 1.0, True)
    before = p.read_diag()
    assert before[LAST].any() and before[STAGES].any()
    g = p.step_graph(ptr, 1.0, 1)
    g.launch()
    after = p.read_diag()
    assert not after[STAGES].any()
    np.testing.assert_array_equal(after[LAST], before[LAST])
