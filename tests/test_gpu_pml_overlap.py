"""Blocks whose PML slabs meet or cross against the CPU oracle: both slabs of
an axis covering the same points (2 npml > n), and a slab that reaches the
closure rows of the other end.  Such blocks have no strict interior on that
axis; the Cartesian ones run the near-boundary kernel for every point, the
curvilinear ones the generic point update.

Tolerances are those of the single-stage parity tests: 1e-12 relative on rates
and fields, 1e-11 on memory variables, after two stages from a random state."""
import pytest

from cases import random_state, rel_l2, small_case

pytestmark = pytest.mark.gpu


def _stages(oracle, p):
    from waveqlab3d_q_gpu_b200.domain import Domain
    (F, DF), = random_state(p)
    o, g = oracle.OracleDomain(p), Domain(p)
    for d in (o, g):
        d.set_fields(F)
    o.set_rates(DF)
    g.set_rates_array(DF)
    for st in (1, 2):
        o.stage(st, p.dt())
        g.stage(st, p.dt())
    assert rel_l2(g.rates(), o.rates()) < 1e-12
    assert rel_l2(g.fields(), o.fields()) < 1e-12
    if p.response != "elastic":
        assert rel_l2(g.eta(), o.eta()) < 1e-11
    g.close()


# small_case has slabs at both ends of y and z and at the end of x
@pytest.mark.parametrize("n,npml", [((13, 13, 13), 7),    # y and z cross by a row
                                    ((17, 13, 20), 7),    # y only, with planes between the z slabs
                                    ((34, 21, 15), 9)])   # z by three rows
@pytest.mark.parametrize("response", ["elastic", "anelastic-Q4"])
@pytest.mark.parametrize("mesh", ["cartesian", "curvilinear"])
def test_overlapping_slabs(wql3d_lib, oracle_lib, mesh, response, n, npml):
    p = small_case(mesh=mesh, response=response, pml=True, n=n)
    p.blocks[0].npml = npml
    _stages(oracle_lib, p)


@pytest.mark.parametrize("literal", [False, True])
def test_slab_reaches_the_other_closure(wql3d_lib, oracle_lib, literal):
    """npml = 9 at one end of a 13-point axis: 9 + 6 > 13.  With the
    single-precision closure literal the metric is full and the block runs the
    near-boundary kernel, without it the point kernel."""
    p = small_case(response="anelastic-Q4", pml=True, n=(13, 13, 20))
    b = p.blocks[0]
    b.npml = 9
    b.pml_lqrs, b.pml_rqrs = (False, False, True), (True, True, False)
    p.closure_f32_literal = literal
    _stages(oracle_lib, p)
