"""Which grids take the plane form (y, the vertical solve and y back in one launch, a kx plane
per block) without being timed: those whose planes have an SM each.  More planes run in waves,
which the autotuner may still choose: they give the separate launches' results.
"""
import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev, host

pytestmark = pytest.mark.gpu


def _plan(nx, ny, nz, prec, **kw):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    return Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                         projection=True, autotune=False))


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("ny, nz", [(12, 8), (320, 32)])
def test_the_untimed_choice_is_one_wave(prec, ny, nz):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    even = [n for n in range(8, 1000, 2)
            if max(p for p in range(2, n // 2 + 1) if (n // 2) % p == 0
                   and all(p % q for q in range(2, p))) <= 5]
    last = max(n for n in even if n // 2 + 1 <= sms)
    more = min(n for n in even if n // 2 + 1 > sms)
    assert _plan(last, ny, nz, prec).variants()["z_yz"] == 1
    p = _plan(more, ny, nz, prec)
    assert p.variants()["z_yz"] == 0
    p.set_variants(z_yz=1)  # still on offer


@pytest.mark.parametrize("nx, ny, nz", [(300, 12, 9), (972, 8, 4), (1024, 16, 17)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_planes_in_waves_match_the_separate_launches(nx, ny, nz, prec):
    """FP64: the parity bar of the separate launches, 1e-12; FP32: a few ulp of the wind (1e-6
    times 10, as the lines' own tests allow), 1e-3 of w and the potential."""
    rng = np.random.default_rng(nx)
    f = [rng.standard_normal((nx, ny, n)) for n in (nz, nz, nz + 1)]
    f[2][:, :, 0] = f[2][:, :, -1] = 0.0
    got = []
    for plane in (1, 0):
        p = _plan(nx, ny, nz, prec)
        p.set_variants(z_yz=plane)
        u, v, w = (dev(a, p.dtype) for a in f)
        phi = torch.empty_like(u)
        p.project(u, v, w, phi)
        got.append([host(a).astype(np.float64) for a in (u, v, w, phi)])
    for a, b, name in zip(*got, ("u", "v", "w", "phi")):
        bar = 1e-12 if prec == "fp64" else 1e-5 if name in ("u", "v") else 1e-3
        assert np.abs(a - b).max() <= bar * np.abs(b).max(), name
