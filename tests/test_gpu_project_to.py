"""The projection into new fields against the one in place, in every form of the inverse x
transform that a grid allows, and the component on fields that need a copy first.

The kernels and their arithmetic are the same, so the results are the same bits; the outputs
start as NaN, so a level that nothing writes shows.
"""
import numpy as np
import pytest
import torch

from oracle import lh82 as O
from tests.gpu_helpers import dev

pytestmark = pytest.mark.gpu


def _fields(nx, ny, nz, dtype, lid=0.0):
    rng = np.random.default_rng(nx + ny + nz)
    u, v, w = (rng.standard_normal((nx, ny, n)) for n in (nz, nz, nz + 1))
    w[:, :, 0] = w[:, :, -1] = lid
    return [dev(a, dtype) for a in (u, v, w)]


@pytest.mark.parametrize("nx, ny, nz", [(8, 10, 9), (50, 36, 17), (64, 48, 32), (512, 12, 16),
                                        (1024, 12, 8)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_into_new_fields(nx, ny, nz, prec):
    from oraclev8_b200._plan import Plan, PlanSpec
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    for shared, off in ((False, ()), (False, ("z_ix",)), (False, ("z_ix", "zc4_ix", "zc3_ix")),
                        (True, ())):
        p = Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=prec,
                          projection=True, autotune=False))
        if shared:
            p.shared_memory_forms()
        for name in off:
            p.set_variants(**{name: 0})
        u, v, w = _fields(nx, ny, nz, p.dtype, lid=0.5)
        outs = [torch.full_like(a, float("nan")) for a in (u, v, w, u)]
        kept = [a.clone() for a in (u, v, w)]
        p.project_to(u, v, w, *outs)
        for a, b in zip((u, v, w), kept):
            assert torch.equal(a, b)
        phi = torch.empty_like(u)
        p.project(u, v, w, phi)
        for a, b, name in zip(outs, (u, v, w, phi), ("u", "v", "w", "phi")):
            assert torch.equal(a, b), (name, shared, off)


def test_the_component_copies_what_the_kernels_cannot_read():
    from oraclev8_b200.production_config import BaseState
    from oraclev8_b200.solver import AnelasticProjection, State
    nx, ny, nz = 48, 40, 9
    base = BaseState(nz, 16e3)
    fields = _fields(nx, ny, nz, torch.float64)
    results = []
    for case in ("plain", "level slices", "off 16 bytes"):
        ins = []
        for a in fields:
            if case == "level slices":
                a = torch.cat([a, a], dim=2)[:, :, :a.shape[2]]
                assert not a.is_contiguous()
            elif case == "off 16 bytes":
                flat = torch.empty(a.numel() + 1, dtype=a.dtype, device=a.device)
                a = flat[1:].view(a.shape).copy_(a)
                assert a.data_ptr() % 16
            ins.append(a)
        st = State(*ins, torch.zeros_like(fields[0]), torch.zeros_like(fields[0]), 0.0)
        st = AnelasticProjection(nx, ny, nz, nx * 1e4, ny * 1e4, 16e3).apply_projection(
            st, None, None, base, 10.0)
        results.append((st.u, st.v, st.w, st.projection_potential))
        for a, b in zip(ins, fields):
            assert torch.equal(a, b)  # the caller's fields stay
    for got in results[1:]:
        for a, b in zip(got, results[0]):
            assert torch.equal(a, b)
