"""A solve that logs its residuals takes the route of one that does not: the same launches, the
same bits, and residuals of the solution that it returns.

The plane form (a kx plane per block: forward y, the vertical solve and back) with the scratch
of one and of several groups of level chunks, columns beyond the block's threads, odd level
counts, and line forms other than the plane's own selected beside it, which a logged solve must
not fall back to.
"""
import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev

pytestmark = pytest.mark.gpu

COMPAT, DISC = 12, 13  # include/oracle_b200.h, OB_DIAG_LAST_*
GRIDS = [(48, 40, 9), (50, 36, 17), (16, 600, 4), (12, 240, 40), (12, 192, 64), (8, 10, 3)]


def _plan(nx, ny, nz, prec, **variants):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    p = Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                      projection=True, autotune=False))
    try:
        p.set_variants(z_yz=variants.pop("z_yz", 1), **variants)
    except ValueError as e:
        pytest.skip(f"the plane does not fit shared memory, or the plan's other forms: {e}")
    return p


def _fields(p, seed=5):
    rng = np.random.default_rng(seed)
    f = [rng.standard_normal((*p.shape[:2], n)) for n in (p.shape[2],) * 2 + (p.shape[2] + 1,)]
    f[2][:, :, 0] = f[2][:, :, -1] = 0.0
    return [dev(a, p.dtype) for a in f]


def _both(p, call):
    """(outputs, launches, diagnostics) of the call without and with logging; the plan's
    first solve, which logs, is past."""
    res = []
    for log in (False, True):
        before = p.launches
        outs = call(log)
        n = p.launches - before
        res.append((outs, n, p.read_diag()))
    return res


@pytest.mark.parametrize("nx, ny, nz", GRIDS)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("lines", [1, 0])
def test_logging_changes_neither_the_route_nor_the_bits(nx, ny, nz, prec, lines):
    p = _plan(nx, ny, nz, prec, z_fy=lines, z_iy=lines)
    u, v, w = _fields(p)

    def project(log):
        a = [u.clone(), v.clone(), w.clone(), torch.empty_like(u)]
        p.project(*a, log_diag=log)
        return a

    project(False)
    d = p.divergence(u, v, w)
    for call in (project, lambda log: [p.poisson_solve(d, log_diag=log)]):
        (a, na, da), (b, nb, db) = _both(p, call)
        assert na == nb
        for x, y in zip(a, b):
            assert torch.equal(x, y)
        assert db[DISC] > 0.0 and np.isfinite(db).all()


@pytest.mark.parametrize("nx, ny, nz", GRIDS)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_the_residuals_are_those_of_the_separate_launches(nx, ny, nz, prec):
    """The same sweeps in the same order, on spectra that differ by the rounding of the
    transforms at most.  The compatibility residual of an arbitrary source agrees to that
    rounding (log2 of the line times an ulp of the spectrum's largest value, in the plan's
    type); the discrete residual is the rms of the sweeps' roundings, thousands of values of one
    distribution and in single precision partly of another sweep (twisted or generic), hence a
    factor."""
    got = []
    for plane in (1, 0):
        p = _plan(nx, ny, nz, prec, z_yz=plane)
        u, v, w = _fields(p)
        p.poisson_solve(u, log_diag=True) if prec == "fp64" else p.project(
            u.clone(), v.clone(), w.clone(), torch.empty_like(u), log_diag=True)
        compat = p.read_diag()[COMPAT]
        a = [u.clone(), v.clone(), w.clone(), torch.empty_like(u)]
        p.project(*a, log_diag=True)
        got.append((compat, p.read_diag()[DISC]))
    (c1, d1), (c0, d0) = got
    dz = 16e3 / nz
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    # the zero mode is a sum of nx ny unit values a level (a divergence: over dz), nz of them
    peak = nx * ny * nz * (dz if prec == "fp64" else 1.0) * 3.0
    assert abs(c1 - c0) <= 32 * eps * peak
    assert d0 / 2.0 <= d1 <= 2.0 * d0
