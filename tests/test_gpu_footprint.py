"""The memory of a served run against the rule that admits it (serving.footprint_bytes): the
state and all that its plan allocates, the plane form's pivots among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", ["lh82", "production"])
@pytest.mark.parametrize("precision", ["fp64", "fp32r"])
@pytest.mark.parametrize("n, nz", [(128, 64), (192, 48), (256, 32), (384, 48)])
def test_a_run_holds_what_the_rule_counts(n, nz, precision, physics):
    """Without the rule's allowance (5% and 8 MB), but for what it rounds off: the extra level of
    the w-level fields (the state's, the anchor's, the stage's and the buoyancy), the extra
    plane of 2 (n / 2 + 1) / n that makes the pivots of single precision outgrow a field, and
    1 MB of tables."""
    from oraclev8_b200.serving import RunRequest, build_run, footprint_bytes
    req = RunRequest(0, n, nz, 45.0, 40e3, 1.5, 20.0, 0.1, precision, physics=physics)
    integ, state, _ = build_run(req)
    held = sum(getattr(state, f).numel() * getattr(state, f).element_size()
               for f in ("u", "v", "w", "theta_prime", "projection_potential"))
    held += integ.plan.scratch_bytes
    counted = (footprint_bytes(req) - (8 << 20)) / 1.05
    size = 8 if precision == "fp64" else 4
    assert held <= counted + 4 * n * n * size + 8 * n * nz + (1 << 20)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_plan_without_damping_ignores_its_terms(precision):
    """No damper, no second temporary: the damping term of such a plan is none, in a call of
    its own and beside others, and the operators that use the first one are unchanged."""
    from oracle import lh82 as O
    from oraclev8_b200 import _lib as L
    from oraclev8_b200._plan import Plan, PlanSpec
    nx, ny, nz = 48, 40, 32
    z, rho0, th0 = O.build_base_state(nz, 16e3)
    p, q = (Plan(PlanSpec(nx, ny, nz, nx * 5e3, ny * 5e3, 16e3, rho0, th0, precision=precision,
                          advection=2, projection=True, autotune=False, damping=d, epsilon=0.5))
            for d in (False, True))
    g = torch.Generator(device="cuda").manual_seed(2)
    u, v, th = (torch.randn(nx, ny, nz, device="cuda", dtype=p.dtype, generator=g)
                for _ in range(3))
    w = torch.zeros(nx, ny, nz + 1, device="cuda", dtype=p.dtype)
    for t in p.tendency(L.OB_TEND_DAMPING, u, v, w, th, 20.0):
        assert not t.any()
    both = L.OB_TEND_DAMPING | L.OB_TEND_ADVECTION
    for a, b in zip(p.tendency(both, u, v, w, th, 20.0),
                    q.tendency(L.OB_TEND_ADVECTION, u, v, w, th, 20.0)):
        assert torch.equal(a, b)
    assert torch.equal(p.apply_operator(th), q.apply_operator(th))
