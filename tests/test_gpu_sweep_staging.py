"""Structures whose sweeps get four stage buffers of one or two steps
(tests/sweep_cases.py; tests/test_sweep_staging.py shows that they do), against
the oracle: the factors bit for bit, and the iterates.

Tolerance: the systems are diagonally dominant by a tenth (condition number below
100) and the iterates differ from the oracle's through FMA and the order of the
sums only: 1e-16 * sqrt(n) * 100 < 1e-11 over five iterations, 1e-10 leaves a
digit."""
import numpy as np
import pytest

import sweep_cases as cases

pytestmark = pytest.mark.gpu


@pytest.fixture(params=sorted(cases.STAGED))
def system(request, ctx):
    box, tiles, _, _ = cases.STAGED[request.param]
    ia, ja, dg, a = cases.red_black(**box)
    ctx.set_sweep_tiles(tiles)
    ctx.pattern_forget()
    try:
        yield ia + 1, ja + 1, a, dg + 1, tiles
    finally:
        ctx.set_sweep_tiles(0)
        ctx.pattern_forget()


@pytest.mark.parametrize("kind", ["dic", "dilu"])
def test_factors(system, ctx, oracle, kind):
    ia, ja, a, dg, tiles = system
    d = ctx.precond_setup(kind, ia, ja, a, dg)
    assert ctx.sweep_stats(1)["tiles"] == tiles
    assert np.array_equal(d, oracle.dic_setup(ia, ja, a, dg, dilu=(kind == "dilu")))


@pytest.mark.parametrize("solver", ["iccg", "bicgstab", "gauss-seidel"])
def test_iterates(system, ctx, oracle, solver):
    ia, ja, a, dg, tiles = system
    rng = np.random.default_rng(5)
    args = (ia, ja, a, dg, np.zeros(len(dg)), rng.uniform(-1.0, 1.0, len(dg)), 5, 1e-30, 1e-30)
    xo, r0o, info_o, _ = oracle.solve(solver, *args)
    for _ in range(3):
        x, r0, info, st = ctx.csrsolve(solver, *args)
        assert st >= 0 and info.itr_used == int(info_o[0])
        assert r0 == pytest.approx(r0o, rel=1e-12)
        np.testing.assert_allclose(x, xo, rtol=0, atol=1e-10 * np.abs(xo).max())
    assert ctx.sweep_stats(1)["tiles"] == tiles


@pytest.mark.parametrize("solver", ["iccg", "bicgstab", "gauss-seidel"])
@pytest.mark.parametrize("name", sorted(cases.DENSE))
def test_densely_coupled_rows(ctx, oracle, name, solver):
    make, tiles = cases.DENSE[name]
    ia, ja, dg, a = make()
    b = np.random.default_rng(8).uniform(-1.0, 1.0, len(dg))
    args = (ia + 1, ja + 1, a, dg + 1, np.zeros(len(dg)), b, 5, 1e-30, 1e-30)
    xo, r0o, info_o, _ = oracle.solve(solver, *args)
    ctx.set_sweep_tiles(tiles)
    ctx.pattern_forget()
    try:
        x, r0, info, st = ctx.csrsolve(solver, *args)
    finally:
        ctx.set_sweep_tiles(0)
        ctx.pattern_forget()
    assert st >= 0 and info.itr_used == int(info_o[0])
    assert r0 == pytest.approx(r0o, rel=1e-12)
    np.testing.assert_allclose(x, xo, rtol=0, atol=1e-10 * np.abs(xo).max())
