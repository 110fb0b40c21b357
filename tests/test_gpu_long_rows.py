"""Rows of more than 255 entries on one side of the diagonal, which the sweeps
serve from their ring (tests/test_sweep_records.py replays their records): the
factors bit for bit and the iterates of every solver against the oracle, on the
tiles that the analysis chooses.

Tolerance: the scaled matrix is diagonally dominant by a tenth (condition number
below 21) and the iterates differ from the oracle's through FMA and the order of
the sums only, 1e-16 * 600 * 21 < 2e-12 over five iterations; 1e-10."""
import numpy as np
import pytest

import sweep_cases as cases

pytestmark = pytest.mark.gpu

SHAPES = [(300, 64, 0), (300, 64, 12), (600, 40, 0), (256, 9, 3), (255, 9, 0)]


@pytest.fixture(params=SHAPES, ids=lambda s: "%d-%d-%d" % s)
def system(request, ctx):
    ia, ja, dg, a = cases.blocks_coupled(*request.param)
    ctx.pattern_forget()
    yield ia + 1, ja + 1, a, dg + 1
    ctx.pattern_forget()


@pytest.mark.parametrize("kind", ["dic", "dilu"])
def test_factors(system, ctx, oracle, kind):
    ia, ja, a, dg = system
    d = ctx.precond_setup(kind, ia, ja, a, dg)
    assert np.array_equal(d, oracle.dic_setup(ia, ja, a, dg, dilu=(kind == "dilu")))


@pytest.mark.parametrize("solver", ["iccg", "bicgstab", "gauss-seidel", "dpcg"])
def test_iterates(system, ctx, oracle, solver):
    ia, ja, a, dg = system
    b = np.random.default_rng(6).uniform(-1.0, 1.0, len(dg))
    args = (ia, ja, a, dg, np.zeros(len(dg)), b, 5, 1e-30, 1e-30)
    xo, r0o, info_o, _ = oracle.solve(solver, *args)
    x, r0, info, st = ctx.csrsolve(solver, *args)
    assert st >= 0 and info.itr_used == int(info_o[0])
    assert r0 == pytest.approx(r0o, rel=1e-12)
    np.testing.assert_allclose(x, xo, rtol=0, atol=1e-10 * np.abs(xo).max())


def test_mixed_iccg_reaches_the_tolerance(system, ctx, oracle, fc):
    ia, ja, a, dg = system
    b = np.random.default_rng(7).uniform(-1.0, 1.0, len(dg))
    ctx.set_precision(fc.FC_PREC_MIXED, 1e-4, 0)
    try:
        x, _, info, st = ctx.csrsolve("iccg", ia, ja, a, dg, np.zeros(len(dg)), b, 1000, 0.0, 1e-10)
    finally:
        ctx.set_precision(fc.FC_PREC_FP64)
    assert st == 0
    # r is formed again here: its entries cancel to 1e-10 of |b|, so that its sum is good to 1e-2
    assert np.abs(b - oracle.spmv(ia, ja, a, x)).sum() < 1.02e-10 * np.abs(b).sum()
