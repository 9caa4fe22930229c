"""Fields that start on an odd element of a larger buffer, through every entry point whose x
transforms read or write the caller's fields in level pairs.

A pair wants its own size as alignment; such a field (contiguous, so it is accepted) goes level
by level, with the same arithmetic: the results are the bits of the aligned call.  Even level
counts, where pairs are used at all; lines of 3 passes, of 512 and of 1024 points.
"""
import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev

pytestmark = pytest.mark.gpu

GRIDS = [(48, 40, 8), (50, 36, 10), (512, 12, 16), (1024, 12, 10)]


def _plan(nx, ny, nz, prec, **kw):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    p = Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                      projection=True, autotune=False, **kw))
    v = p.variants()
    assert v["z_fx"] and v["z_ix"]
    return p


def _off(a):
    """The same values one element into a buffer of their own."""
    flat = torch.empty(a.numel() + 1, dtype=a.dtype, device=a.device)
    b = flat[1:].view(a.shape).copy_(a)
    assert b.is_contiguous() and b.data_ptr() % (2 * a.element_size())
    return b


def _fields(p, seed=7):
    rng = np.random.default_rng(seed)
    nx, ny, nz = p.shape
    f = [rng.standard_normal((nx, ny, n)) for n in (nz, nz, nz + 1, nz)]
    f[2][:, :, 0] = f[2][:, :, -1] = 0.0
    return [dev(a, p.dtype) for a in f]


def _same(got, want):
    for n, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), n


@pytest.mark.parametrize("nx, ny, nz", GRIDS)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_projection_and_operators(nx, ny, nz, prec):
    from oraclev8_b200 import _lib as L
    p = _plan(nx, ny, nz, prec, damping=True, epsilon=0.5)
    u, v, w, d = _fields(p)

    def project(move):
        a = [move(x.clone()) for x in (u, v, w, torch.zeros_like(u))]
        p.project(*a)
        if prec == "fp32":
            p.refine(*a)
        return a

    def project_to(ins, outs):
        a = [ins(x.clone()) for x in (u, v, w)]
        b = [outs(torch.zeros_like(x)) for x in (u, v, w, u)]
        p.project_to(*a, *b)
        return b

    keep = lambda a: a
    _same(project(_off), project(keep))
    want = project_to(keep, keep)
    for ins, outs in ((_off, keep), (keep, _off), (_off, _off)):
        _same(project_to(ins, outs), want)
    out = _off(torch.zeros_like(u))
    p.divergence(_off(u), _off(v), _off(w), out=out)
    _same([out], [p.divergence(u, v, w)])
    _same([p.poisson_solve(_off(d))], [p.poisson_solve(d)])
    _same([p.apply_operator(_off(d))], [p.apply_operator(d)])
    _same(p.phi_gradient(_off(d)), p.phi_gradient(d))
    _same(p.tendency(L.OB_TEND_DAMPING, *map(_off, (u, v, w, d)), 20.0),
          p.tendency(L.OB_TEND_DAMPING, u, v, w, d, 20.0))


@pytest.mark.parametrize("nx, ny, nz", GRIDS)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("physics", ["lh82", "damped"])
def test_steps_and_captured_steps(nx, ny, nz, prec, physics):
    kw = dict(advection=2, coriolis=1, f0=5e-5)
    kw.update(dict(buoyancy=True) if physics == "lh82" else dict(damping=True, epsilon=0.5))
    results = []
    for move in (lambda a: a, _off):
        p = _plan(nx, ny, nz, prec, **kw)
        if prec == "fp32":
            p.set_refinement(1)
        s = [move(a) for a in _fields(p)]
        s.append(move(torch.zeros_like(s[0])))
        ptr = p.state_ptrs(*s)
        p.step(ptr, ptr, 10.0, True)
        diag = p.read_diag()[:6]
        g = p.step_graph(ptr, 10.0, 2)
        g.launch()
        torch.cuda.synchronize()
        results.append((s, diag))
    _same(results[1][0], results[0][0])
    # maxima are exact; the potential's extrema are about a mean whose sum runs in another
    # order: n additions' rounding, 1e-16 n, of the potential's scale
    np.testing.assert_array_equal(results[1][1][:4], results[0][1][:4])
    n = nx * ny * nz
    scale = np.abs(results[0][1][4:6]).max()
    assert np.abs(results[1][1][4:6] - results[0][1][4:6]).max() <= 1.2e-16 * n * scale
