"""Choosing an older kernel form by name (Plan.set_variants, oracle_b200_plan_set_variants) runs
it: the level-paired form of its class, on by default, does not run instead."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev, host

pytestmark = pytest.mark.gpu


def _plan(nx, ny, nz, prec):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    return Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                         projection=True, autotune=False))


def _old_forms(p):
    """The plan's choices of older forms, each with a value its grid allows."""
    from oraclev8_b200 import _lib as L
    cur = p.variants()
    for z, older in L.OLDER_FORMS.items():
        for k in older:
            if cur[k]:
                yield z, k, cur[k]


@pytest.mark.parametrize("nx, ny, nz", [(96, 60, 9), (512, 40, 16), (40, 512, 16), (1024, 16, 8),
                                        (16, 1024, 8)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_a_named_form_turns_the_level_paired_one_off(nx, ny, nz, prec):
    p = _plan(nx, ny, nz, prec)
    base = p.variants()
    seen = 0
    for z, name, value in _old_forms(p):
        p.set_variants(**base)
        assert p.variants() == base
        p.set_variants(**{name: value})
        now = p.variants()
        assert now[name] == value and now[z] == 0
        p.set_variants(**{**base, name: value})  # named too: as named
        assert p.variants() == base
        seen += 1
    assert seen >= 2


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_an_array_that_ends_before_the_level_paired_entries_is_the_whole_choice(prec):
    from oraclev8_b200 import _lib as L
    p = _plan(96, 60, 9, prec)
    n = L.VARIANTS.index("z_fx")
    base = p.variants()
    assert base["z_fx"] and base["z_yz"]
    vals = (ctypes.c_int * n)(*[base[k] for k in L.VARIANTS[:n]])
    L.check(p.lib.oracle_b200_plan_set_variants(p.handle, vals, 0))
    assert p.variants() == base
    L.check(p.lib.oracle_b200_plan_set_variants(p.handle, vals, 3))  # zc2_fx, zc2_fxs, zc2_ix
    now = p.variants()
    assert [k for k in base if now[k] != base[k]] == ["z_fx", "z_fxs", "z_ix"]
    L.check(p.lib.oracle_b200_plan_set_variants(p.handle, vals, n))
    now = p.variants()
    assert not any(v for k, v in now.items() if k.startswith("z_"))
    assert all(now[k] == base[k] for k in L.VARIANTS[:n])


def test_the_named_form_is_the_one_that_runs():
    """The forms round differently, so a projection tells them apart: naming the 512-point x
    forms gives the bits of a plan without level-paired forms, not those of the default."""
    rng = np.random.default_rng(4)
    nx, ny, nz = 512, 12, 16
    f = [rng.standard_normal((nx, ny, n)) for n in (nz, nz, nz + 1)]
    f[2][:, :, 0] = f[2][:, :, -1] = 0.0
    outs = []
    for how in ("default", "named", "none"):
        p = _plan(nx, ny, nz, "fp32")
        p.set_variants(z_yz=0, z_fy=0, z_iy=0)
        if how == "named":
            p.set_variants(zc3_fx=8, zc3_ix=8)
        elif how == "none":
            p.set_variants(z_fx=0, z_ix=0)
        u, v, w = (dev(a, p.dtype) for a in f)
        phi = torch.empty_like(u)
        p.project(u, v, w, phi)
        outs.append(host(u))
    assert np.array_equal(outs[1], outs[2]) and not np.array_equal(outs[0], outs[1])
