"""Curvilinear blocks on both sides of the launch rules: with PML the point
kernels take three launches a stage (face terms, both roles, auxiliary
velocities) and the fused kernel two.  FP64 fQ8 with PML, small blocks with PML
and FP32 elastic ones below 1.2 million points run the fused kernel; elastic
rows of 96 points and more are mapped to warps row by row.

Tolerances are those of the single-stage parity tests: 1e-12 relative on rates
and fields, 1e-11 on memory variables, after two stages from a random state;
FP32 2e-5 on the fields, velocities and stresses apart."""
import pytest

from cases import random_state, rel_l2, small_case

pytestmark = pytest.mark.gpu

EL, Q4, Q8, FQ8 = "elastic", "anelastic-Q4", "anelastic-Q8", "anelastic-fQ8"


@pytest.mark.parametrize("response,precision,n,launches", [
    (FQ8, "fp64", (33, 21, 22), 2),      # fQ8 with PML: fused at every size
    (FQ8, "fp64", (48, 41, 40), 2),
    (EL, "fp64", (40, 40, 40), 2),       # 2^16 = 65536 points
    (EL, "fp64", (41, 40, 40), 3),
    (EL, "fp64", (95, 27, 28), 3),       # rows of 95 and 96 points
    (EL, "fp64", (96, 27, 28), 3),
    (Q8, "fp64", (25, 25, 26), 3),       # 2^14 = 16384 points
    (Q8, "fp64", (26, 25, 26), 2),
    (Q4, "fp64", (40, 40, 40), 2),
    (Q4, "fp64", (41, 40, 40), 3),
    (EL, "fp32", (41, 40, 40), 2),       # 1.2 million points
    (EL, "fp32", (106, 106, 107), 3),
    (EL, "fp32", (93, 113, 115), 3),     # 1.21 million in short rows
])
def test_pml_routes(wql3d_lib, oracle_lib, response, precision, n, launches):
    from waveqlab3d_q_gpu_b200.domain import Domain
    p = small_case(mesh="curvilinear", response=response, pml=True, n=n)
    (F, DF), = random_state(p)
    o, g = oracle_lib.OracleDomain(p), Domain(p, precision=precision)
    for d in (o, g):
        d.set_fields(F)
    o.set_rates(DF)
    g.set_rates_array(DF)
    count = []
    for st in (1, 2):
        o.stage(st, p.dt())
        before = g.kernel_launches()
        g.stage(st, p.dt())
        count.append(g.kernel_launches() - before)
    assert count[1] == launches          # the first stage also computes the fluxes
    if precision == "fp64":
        assert rel_l2(g.rates(), o.rates()) < 1e-12
        assert rel_l2(g.fields(), o.fields()) < 1e-12
        if response != EL:
            assert rel_l2(g.eta(), o.eta()) < 1e-11
    else:
        Fg, Fo = g.fields(), o.fields()
        assert rel_l2(Fg[:3], Fo[:3]) < 2e-5
        assert rel_l2(Fg[3:], Fo[3:]) < 2e-5
    g.close()
