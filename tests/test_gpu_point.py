"""The two-role point kernels (full stages of separable Cartesian and of
curvilinear blocks) against the CPU oracle at the sizes where their work maps
turn: the smallest block (13 points: every row a closure), odd row counts (a
row pair's second row missing), and the row lengths where the boundary columns
of a row change their place: 32 (no whole warp of central columns), 33 (the
remainder fills a warp of its own), 44 / 48 / 49 (two rows' boundary columns in
one warp up to 16 columns a row, one row per warp from 17).

Tolerances are those of the other single-stage and short-run parity tests:
1e-12 relative on rates and fields after stages from a random state, 1e-11
after a run with sources, stations and graph replays; FP32 against FP64 on the
same state 2e-5."""
import numpy as np
import pytest

from cases import random_state, rel_l2, small_case

pytestmark = pytest.mark.gpu

SIZES = [(13, 13, 13), (32, 15, 14), (33, 14, 13), (44, 13, 15), (48, 17, 13), (49, 16, 14)]


def _domain(p, **kw):
    from waveqlab3d_q_gpu_b200.domain import Domain
    return Domain(p, **kw)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("response,pml", [("elastic", False), ("elastic", True), ("anelastic-Q4", True),
                                          ("anelastic-Q8", False), ("anelastic-fQ8", False)])
@pytest.mark.parametrize("mesh", ["cartesian", "curvilinear"])
def test_stages_from_a_random_state(wql3d_lib, oracle_lib, mesh, response, pml, n):
    p = small_case(mesh=mesh, response=response, pml=pml, n=n)
    if pml:
        p.blocks[0].npml = 6   # the two slabs of a 13-point axis do not overlap
    (F, DF), = random_state(p)
    dt = p.dt()
    o = oracle_lib.OracleDomain(p)
    g = _domain(p)
    s = _domain(p, precision="fp32")
    for d in (o, g, s):
        d.set_fields(F)
    o.set_rates(DF)
    g.set_rates_array(DF)
    s.set_rates_array(DF)
    for st in (1, 2):
        for d in (o, g, s):
            d.stage(st, dt)
    assert rel_l2(g.rates(), o.rates()) < 1e-12
    assert rel_l2(g.fields(), o.fields()) < 1e-12
    assert rel_l2(s.fields(), g.fields()) < 2e-5
    if response != "elastic":
        assert rel_l2(g.eta(), o.eta()) < 1e-11


@pytest.mark.parametrize("n", [(16, 17, 18), (33, 16, 19)])
@pytest.mark.parametrize("op", [("upwind", 4), ("upwind", 6), ("upwind_drp", 6)])
@pytest.mark.parametrize("mesh,response", [("cartesian", "anelastic-fQ8"), ("curvilinear", "elastic")])
def test_upwind_stages_from_a_random_state(wql3d_lib, oracle_lib, mesh, response, op, n):
    """The upwind pairs at 16 points, twice the widest closure."""
    p = small_case(mesh=mesh, response=response, n=n)
    p.fd_type, p.order = op
    (F, DF), = random_state(p)
    dt = p.dt()
    o, g = oracle_lib.OracleDomain(p), _domain(p)
    for d in (o, g):
        d.set_fields(F)
    o.set_rates(DF)
    g.set_rates_array(DF)
    for st in (1, 2):
        o.stage(st, dt)
        g.stage(st, dt)
    assert rel_l2(g.rates(), o.rates()) < 1e-12
    assert rel_l2(g.fields(), o.fields()) < 1e-12


@pytest.mark.parametrize("mesh", ["cartesian", "curvilinear"])
def test_run_after_every_way_of_setting_fields(wql3d_lib, oracle_lib, mesh):
    """Graph-replayed steps, fields set again, the split operations in between,
    and steps again: nothing of an earlier state is left behind."""
    p = small_case(mesh=mesh, response="anelastic-Q8", n=(45, 15, 14))
    (F, _), (F2, _) = random_state(p, seed=3)[0], random_state(p, seed=4)[0]
    o = oracle_lib.OracleDomain(p)
    g = _domain(p, nsteps_hint=16)
    for d in (o, g):
        d.set_fields(F)
        d.run(4)
        d.set_fields(F2)
        d.run(3)
    assert rel_l2(g.fields(), o.fields()) < 1e-11
    dt = p.dt()
    h = _domain(p, nsteps_hint=16)
    h.set_fields(g.fields())
    k = _domain(p, nsteps_hint=16)
    k.set_fields(g.fields())
    from waveqlab3d_q_gpu_b200.problem import RK_A, RK_B
    h.begin_step(1)
    h.stage(1, dt)
    k.begin_step(1)
    k.scale_rates(RK_A[0])
    k.set_rates()
    k.enforce_bound_iface_conditions(1)
    k.update_fields(RK_B[0] * dt)
    assert rel_l2(k.fields(), h.fields()) < 1e-13
    h.stage(2, dt)
    k.stage(2, dt)
    assert rel_l2(k.fields(), h.fields()) < 1e-13
    assert np.abs(h.fields()).max() > 0.0
