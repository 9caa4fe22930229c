"""The source of a single-precision stage projection: div(rho u) of w + sdt b, the vertical part
a difference of values that may nearly cancel.

Over a uniform column of w (with a constant density its own flux difference is zero) and no
wind, the winds of a buoyant step are the projection's answer to b alone.  An ulp of w is 7.6e-6
here, sdt b about 1e-5: a source formed from w + sdt b rounded to float is wrong in its
first digits, one whose sum is held exactly through the difference is not.
"""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import dev, host

pytestmark = pytest.mark.gpu


def _winds(nx, ny, nz, prec, w0, plane):
    from oraclev8_b200._plan import Plan, PlanSpec
    p = Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, np.ones(nz), np.full(nz, 300.0),
                      precision=prec, buoyancy=True, projection=True, autotune=False))
    try:
        p.set_variants(z_yz=plane)
    except ValueError:
        pytest.skip("the plane does not fit shared memory")
    assert p.variants()["z_fxs"] and p.variants()["z_ix"]
    rng = np.random.default_rng(11)
    th = (1e-3 * rng.standard_normal((nx, ny, nz))).astype(np.float32).astype(np.float64)
    th = dev(th, p.dtype)
    u, v, phi = (torch.zeros_like(th) for _ in range(3))
    w = torch.full((nx, ny, nz + 1), w0, dtype=p.dtype, device="cuda")
    ptr = p.state_ptrs(u, v, w, th, phi)
    p.step(ptr, ptr, 1.0 / 3.0, False)  # no float, so the stage's sdt is not one either
    return [host(a).astype(np.float64) for a in (u, v)]


@pytest.mark.parametrize("nx, ny, nz", [(50, 36, 17), (96, 96, 32), (36, 250, 9), (512, 12, 16),
                                        (1024, 16, 8)])
@pytest.mark.parametrize("plane", [0, 1])
def test_a_large_w_leaves_the_response_to_buoyancy_alone(nx, ny, nz, plane):
    """1e-5 of the winds' scale, the single-precision lines' own bar (their rounding: ten passes
    of an ulp each, and the potential's differences)."""
    want = _winds(nx, ny, nz, "fp64", 100.0, plane=0)
    got = _winds(nx, ny, nz, "fp32", 100.0, plane)
    scale = max(np.abs(a).max() for a in want)
    assert scale > 0
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= 1e-5 * scale
