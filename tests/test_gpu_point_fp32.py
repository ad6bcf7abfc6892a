"""The FP32 point kernels against FP64 on the same random state, quantity by
quantity: velocity and stress rates, velocities, stresses and memory variables
apart (in one norm the stresses of a random state hide the rest).

Tolerances: a rate is a sum of at most 27 products of comparable size (nine taps
on three axes) with a handful of factors; each rounds at 6e-8, so errors of 3e-7
to 6e-7 relative in the norm are expected, and 5e-6 leaves a factor of ten, far
below the 1e-3 or more of a missed tap, mechanism or face term.  Memory
variables also subtract strength products of comparable size (a few times more):
2e-5.  The FP64 side is held to the oracle at 1e-12 in the other stage tests."""
import pytest

from cases import random_state, rel_l2, small_case

pytestmark = pytest.mark.gpu

RESPONSES = ["elastic", "anelastic-Q4", "anelastic-Q8", "anelastic-fQ8"]


def _compare(p):
    from waveqlab3d_q_gpu_b200.domain import Domain
    (F, DF), = random_state(p)
    g, s = Domain(p), Domain(p, precision="fp32")
    for d in (g, s):
        d.set_fields(F)
        d.set_rates_array(DF)
        for st in (1, 2):
            d.stage(st, p.dt())
    for get in ("rates", "fields"):
        a, b = getattr(s, get)(), getattr(g, get)()
        assert rel_l2(a[:3], b[:3]) < 5e-6, get
        assert rel_l2(a[3:6], b[3:6]) < 5e-6, get
        assert rel_l2(a[6:], b[6:]) < 5e-6, get
    if p.response != "elastic":
        a, b = s.eta(), g.eta()
        for c in range(6):
            assert abs(b[c]).max() > 0
            assert rel_l2(a[c], b[c]) < 2e-5, c
    g.close()
    s.close()


@pytest.mark.parametrize("pml", [False, True])
@pytest.mark.parametrize("response", RESPONSES)
@pytest.mark.parametrize("mesh", ["cartesian", "curvilinear"])
def test_traditional(wql3d_lib, mesh, response, pml):
    _compare(small_case(mesh=mesh, response=response, pml=pml, n=(33, 16, 19)))


@pytest.mark.parametrize("op", [("upwind", 4), ("upwind", 6), ("upwind_drp", 6)])
@pytest.mark.parametrize("response", RESPONSES)
@pytest.mark.parametrize("mesh", ["cartesian", "curvilinear"])
def test_upwind(wql3d_lib, mesh, response, op):
    p = small_case(mesh=mesh, response=response, n=(33, 16, 19))
    p.fd_type, p.order = op
    _compare(p)
