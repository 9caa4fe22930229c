"""The x-marching slow tendency (k_slow_xw, variant slow_xw = 1) against the gather form (0).

Both evaluate the same terms in the same order, so they differ where the compiler contracts a
product and a sum differently: a few ulp of the largest term of each sum, which for a random
state is some ten times the largest tendency.  1e-13 (450 ulp) in double precision, the same
number of ulp (5e-5) in single.  Sizes at the form's edges: the smallest grid that it takes,
rows and columns past a multiple of 8 and of a segment, level counts of one chunk, of equal and
of unequal chunks, a lid in a chunk of its own thread and in the level halo.
"""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import dev, host

pytestmark = pytest.mark.gpu


class Base:
    def __init__(self, nz, Lz):
        from oracle import lh82 as O
        self.z, self.rho0, self.theta0 = O.build_base_state(nz, Lz)


def _spec(nx, ny, nz, prec, physics):
    from oraclev8_b200 import _lib as L
    from oraclev8_b200._plan import PlanSpec
    from oraclev8_b200.solver import SpongeDampingComponent, SurfaceDragComponent
    from oraclev8_b200.solver.tendency import drag_fields, sponge_fields
    Lx, Ly, Lz = nx * 20e3, ny * 20e3, 16e3
    base = Base(nz, Lz)
    z = np.asarray(base.z)
    kw = dict(coriolis=L.OB_COR_FPLANE, f0=5e-5)
    mask = L.OB_TEND_CORIOLIS
    if "ws5" in physics or "c2" in physics:
        kw["advection"] = L.OB_ADV_UPWIND5H if "ws5" in physics else L.OB_ADV_CENTERED2
        mask |= L.OB_TEND_ADVECTION
    if "bih" in physics or "lap" in physics:
        bih = "bih" in physics
        kw.update(diffusion=L.OB_DIFF_BIHARMONIC if bih else L.OB_DIFF_LAPLACIAN,
                  diff_nu=1e13 if bih else 2e4, diff_dx2=(Lx / nx) ** 2, diff_dy2=(Ly / ny) ** 2,
                  cooling=True, cool_alpha=1.0 / 3600.0,
                  **drag_fields(SurfaceDragComponent(2e-3, 2000.0, -3.0, 1.0), z),
                  **sponge_fields(SpongeDampingComponent(Lz, 0.02, 0.3, -3.0, 1.0), z))
        mask |= (L.OB_TEND_DRAG | L.OB_TEND_SPONGE | L.OB_TEND_DIFFUSION | L.OB_TEND_COOLING)
    return PlanSpec(nx=nx, ny=ny, nz=nz, Lx=Lx, Ly=Ly, Lz=Lz, rho0=base.rho0,
                    theta0=base.theta0, precision=prec, projection=True, autotune=False,
                    **kw), mask


@pytest.mark.parametrize("nx, ny, nz", [(8, 10, 5), (8, 18, 31), (16, 10, 32), (30, 12, 33),
                                        (20, 50, 45), (36, 40, 64), (10, 12, 97), (150, 162, 9)])
@pytest.mark.parametrize("physics", ["ws5", "c2", "cor", "ws5+bih", "c2+bih", "c2+lap"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_the_march_matches_the_gather(nx, ny, nz, physics, prec):
    from oraclev8_b200._plan import Plan
    spec, mask = _spec(nx, ny, nz, prec, physics)
    rng = np.random.default_rng(nx + ny + nz)
    fields = [np.asarray(a, np.float32) for a in (
        10.0 * rng.standard_normal((nx, ny, nz)), 10.0 * rng.standard_normal((nx, ny, nz)),
        0.3 * rng.standard_normal((nx, ny, nz + 1)), rng.standard_normal((nx, ny, nz)))]
    bar = 1e-13 if prec == "fp64" else 5e-5
    outs = []
    for xw in (0, 1):
        p = Plan(spec)
        p.set_variants(slow_xw=xw)
        f = [dev(a, p.dtype) for a in fields]
        tend = [host(t).astype(np.float64) for t in p.tendency(mask, *f, 30.0)]
        phi = torch.zeros_like(f[0])
        ptr = p.state_ptrs(*f, phi)
        p.step(ptr, ptr, 10.0, False)  # its two half steps, state form
        outs.append((tend, [host(a).astype(np.float64) for a in (*f, phi)]))
    for name, a, b in zip(("du", "dv", "dw", "dth"), outs[1][0], outs[0][0]):
        assert np.abs(a - b).max() <= bar * np.abs(b).max(), name
    # the step's projections multiply a difference by the condition of w and phi
    for name, a, b in zip(("u", "v", "w", "th", "phi"), outs[1][1], outs[0][1]):
        far = 10 if name in ("u", "v", "th") else 100
        assert np.abs(a - b).max() <= far * bar * np.abs(b).max(), name
