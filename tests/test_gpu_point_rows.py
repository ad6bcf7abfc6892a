"""Elastic Cartesian blocks on both sides of the launch rules that depend on
their size: rows of 96 (with PML) and 125 points and more are mapped to warps
row by row, shorter ones as flattened points; FP64 blocks without PML whose
shortest axis has 139 points, and blocks with little shell and thin PML, run the
interior tiles beside the shell (two launches a stage instead of one).

Tolerances are those of the single-stage parity tests: 1e-12 relative on rates
and fields after two stages from a random state; FP32 against FP64 on the same
state 2e-5, velocities and stresses apart."""
import pytest

from cases import random_state, rel_l2, small_case

pytestmark = pytest.mark.gpu


def _stages(oracle, p, precisions):
    from waveqlab3d_q_gpu_b200.domain import Domain
    (F, DF), = random_state(p)
    o = oracle.OracleDomain(p)
    ds = [Domain(p, precision=q) for q in precisions]
    launches = ds[0].kernel_launches()
    for d in [o] + ds:
        d.set_fields(F)
    o.set_rates(DF)
    for d in ds:
        d.set_rates_array(DF)
    for st in (1, 2):
        for d in [o] + ds:
            d.stage(st, p.dt())
    launches = (ds[0].kernel_launches() - launches) / 2
    Fo = o.fields()
    for d, q in zip(ds, precisions):
        if q == "fp64":
            assert rel_l2(d.rates(), o.rates()) < 1e-12
            assert rel_l2(d.fields(), Fo) < 1e-12
        else:
            assert rel_l2(d.fields()[:3], Fo[:3]) < 2e-5
            assert rel_l2(d.fields()[3:], Fo[3:]) < 2e-5
    for d in ds:
        d.close()
    return launches


@pytest.mark.parametrize("nx,pml", [(95, True), (96, True), (97, True), (128, True), (124, False), (125, False),
                                    (126, False), (140, False)])
def test_row_lengths(wql3d_lib, oracle_lib, nx, pml):
    p = small_case(response="elastic", pml=pml, n=(nx, 15, 16))
    assert _stages(oracle_lib, p, ("fp64", "fp32")) == 1


@pytest.mark.parametrize("n,launches", [((139, 139, 139), 2), ((139, 138, 140), 1)])
def test_tiles_from_139_points_an_axis(wql3d_lib, oracle_lib, n, launches):
    assert _stages(oracle_lib, small_case(response="elastic", n=n), ("fp64",)) == launches


# shares of the points: shell / PML slabs
@pytest.mark.parametrize("n,faces,npml,precisions,launches", [
    ((101, 101, 101), 1, 5, ("fp64",), 2),     # 0.316 / 0.05
    ((102, 101, 100), 2, 10, ("fp64",), 2),    # 0.376 / 0.19
    ((102, 101, 100), 3, 10, ("fp64",), 1),    # 0.405 / 0.27
    ((81, 79, 83), 1, 5, ("fp64",), 1),        # 0.382 / 0.06
    ((94, 101, 99), 3, 8, ("fp64",), 2),       # 0.377 / 0.23, short rows
    ((97, 101, 99), 3, 8, ("fp64",), 1),       # 0.373 / 0.23
    ((141, 141, 140), 1, 5, ("fp32", "fp64"), 2),   # 0.236 / 0.04
    ((141, 130, 140), 1, 5, ("fp32", "fp64"), 1),   # 0.241 / 0.04 in FP32
])
def test_tiles_with_thin_pml(wql3d_lib, oracle_lib, n, faces, npml, precisions, launches):
    p = small_case(response="elastic", pml=True, n=n)
    b = p.blocks[0]
    b.npml = npml
    b.pml_rqrs, b.pml_lqrs = (True, faces >= 2, faces >= 3), (False, False, False)
    assert _stages(oracle_lib, p, precisions) == launches


def test_slabs_on_the_tiles_equal_the_whole_block(wql3d_lib):
    """Two s-slabs of 139 planes: each runs the tiles, whose strict interior reaches
    the open face.  Equal to the whole block to rounding, 1e-12 as in the other
    slab tests."""
    import numpy as np
    from waveqlab3d_q_gpu_b200.domain import Domain
    from waveqlab3d_q_gpu_b200.slabs import SlabSet
    p = small_case(response="elastic", n=(139, 139, 278))
    (F, _), = random_state(p, scale=1e-3)
    g = Domain(p, nsteps_hint=4)
    g.set_fields(F)
    g.run(3)
    ss = SlabSet(p, 2, nsteps_hint=4, cuts=(139, 139))
    for part, d in zip(ss.parts, ss.domains):
        d.set_fields(F[:, part.z0:part.z0 + 139])
    before = ss.domains[0].kernel_launches()
    ss.run(3)
    # a step: sample, per stage two stage kernels, a halo pack and an unpack, advance
    assert ss.domains[0].kernel_launches() - before == 3 * (2 + 5 * 4)
    Fw = g.fields(0)
    assert np.abs(Fw).max() > 0
    assert rel_l2(ss.fields(), Fw) < 1e-12
    ss.close()
    g.close()
