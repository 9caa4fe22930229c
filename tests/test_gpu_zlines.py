"""The level-paired line transforms (csrc/zfft.cuh) against the oracle.

Sizes at the edges of their rules: the shortest lines, lines of 2, 3 and 4
passes, every last radix (2, 4, 6, 8), odd strides Q, odd and even level counts
(paired and scalar accesses), one level past a chunk, grids that batch several
rows per block and grids that do not.  FP64 holds the parity bar (1e-12 of each
field's maximum); FP32 the bounds of the single-precision forms: u and v within
a few ulp of the wind (1e-6), w and phi within 1e-3 of their own scale.
"""
import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev, host

pytestmark = pytest.mark.gpu

GRIDS = [(8, 10, 9), (16, 12, 9), (50, 36, 17), (162, 40, 8), (36, 162, 33), (250, 8, 5),
         (128, 96, 16), (972, 8, 4), (8, 1000, 7), (1024, 16, 17)]


def _plan(nx, ny, nz, prec, **kw):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    p = Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                      projection=True, autotune=False, **kw))
    v = p.variants()
    assert v["z_fx"] and v["z_ix"] and v["z_fy"] and v["z_iy"]  # the forms under test
    return p, rho0


def _fields(nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    f = [rng.standard_normal((nx, ny, n)).astype(np.float32).astype(np.float64)
         for n in (nz, nz, nz + 1)]
    f[2][:, :, 0] = f[2][:, :, -1] = 0.0
    return f


def _close(got, want, bar, what):
    err = np.abs(host(got).astype(np.float64) - want).max() / max(np.abs(want).max(), 1e-300)
    assert err <= bar, (what, err)


@pytest.mark.parametrize("nx, ny, nz", GRIDS)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("plane", [1, 0])
def test_projection_and_operators_match_the_oracle(nx, ny, nz, prec, plane):
    p, rho0 = _plan(nx, ny, nz, prec, damping=True, epsilon=0.5)
    if plane and not p.variants()["z_yz"]:
        pytest.skip("the plane does not fit shared memory")
    p.set_variants(z_yz=plane)
    dt = p.dtype
    u, v, w = _fields(nx, ny, nz, seed=nx + 7 * ny + nz)
    wind, fine, rough = (1e-12,) * 3 if prec == "fp64" else (1e-6, 1e-5, 1e-3)
    ref = O.State(u.copy(), v.copy(), w.copy(), np.zeros_like(u), np.zeros_like(u))
    proj = O.Projection(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3)
    s, (rf, rh) = proj.solver, proj.rho_pair(rho0)
    d = O.anelastic_divergence(u, v, w, rf, rh, s.kx, s.ky, proj.dz)
    proj.apply(ref, rho0)
    du, dv, dw = dev(u, dt), dev(v, dt), dev(w, dt)
    phi = torch.empty_like(du)
    p.project(du, dv, dw, phi)
    scale = max(np.abs(ref.u).max(), np.abs(ref.v).max())
    for got, want in ((du, ref.u), (dv, ref.v)):
        assert np.abs(host(got).astype(np.float64) - want).max() <= wind * 10 * scale
    _close(dw, ref.w, rough, "w")
    _close(phi, ref.projection_potential, rough, "phi")
    _close(p.divergence(dev(u, dt), dev(v, dt), dev(w, dt)), d, fine, "divergence")
    # the solve takes the compatible part of its source
    _close(p.poisson_solve(dev(d, dt)), ref.projection_potential, rough, "solve")
    f = ref.projection_potential.astype(np.float32).astype(np.float64)
    for got, want, name in zip(p.phi_gradient(dev(f, dt)), O.phi_gradient(f, s.kx, s.ky, proj.dz),
                               ("gx", "gy", "gz")):
        if np.abs(want).max() > 0:
            _close(got, want, 1e-12 if prec == "fp64" else 1e-4, name)
    from oraclev8_b200 import _lib as L
    hu, hv = O.helmholtz_tendency(u, v, 0.5, 20.0, nx * 5e3, ny * 5e3)
    got = p.tendency(L.OB_TEND_DAMPING, dev(u, dt), dev(v, dt), dev(w, dt), dev(u, dt), 20.0)
    _close(got[0], hu, fine, "damper u")
    _close(got[1], hv, fine, "damper v")


@pytest.mark.parametrize("nx, ny, nz", [(36, 20, 7), (128, 40, 17), (250, 12, 16)])
@pytest.mark.parametrize("prec", ["fp64", "fp32r"])
def test_a_step_matches_the_other_forms(nx, ny, nz, prec):
    """The stage forms (and the FP64-residual correction): one buoyant step with
    the level-paired lines and with the shared-memory kernels."""
    outs = []
    for paired in (True, False):
        p, _ = _plan(nx, ny, nz, prec[:4], buoyancy=True, advection=2, coriolis=1, f0=5e-5)
        if prec == "fp32r":
            p.set_refinement(1)
        if not paired:
            p.shared_memory_forms()
            assert not any(x for k, x in p.variants().items() if k.startswith("z_"))
        u, v, w = (dev(a, p.dtype) for a in _fields(nx, ny, nz, seed=3))
        th = dev(_fields(nx, ny, nz, seed=4)[0], p.dtype)
        phi = torch.zeros_like(u)
        ptr = p.state_ptrs(u, v, w, th, phi)
        p.step(ptr, ptr, 10.0, True)
        p.read_diag()
        outs.append([host(a).astype(np.float64) for a in (u, v, w, th, phi)])
    for a, b, name in zip(*outs, ("u", "v", "w", "th", "phi")):
        bar = 1e-12 if prec == "fp64" else 2e-5 if name in ("u", "v", "th") else 2e-3
        assert np.abs(a - b).max() <= bar * np.abs(b).max(), name
