"""The persistent loop of the coloured inner ICCG (one launch for all
iterations) at the sizes and layouts where it can go wrong: fewer rows than a
block, one block and one more, several rows a thread; two colours with rows
of up to 4, 6, 8 and more entries; more than two colours.  Both value types.

The refinement around it stops at sum |b - A x| < tol * sum |b - A x0| in FP64;
the same sums formed here differ by rounding only: 1e-12 relative of r, whose
entries cancel to 1e-10 of |b|, is 1e-2, hence the 1.02.  Five digits a
refinement and a condition number below 100 keep the outer iterations few."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OFFSETS = {"path": (1,), "four": (1, 3), "six": (1, 3, 5), "eight": (1, 3, 5, 7), "ten": (1, 3, 5, 7, 9),
           "colours": (1, 2, 5)}


def even_ring(n, kind):
    """Symmetric ring with the given offsets (odd ones and even n: two colours)."""
    rng = np.random.default_rng(n)
    rows = [[] for _ in range(n)]
    for i, j in sorted({(min(i, (i + o) % n), max(i, (i + o) % n)) for o in OFFSETS[kind] for i in range(n)}):
        v = -rng.uniform(0.5, 1.5)
        rows[i].append((j, v))
        rows[j].append((i, v))
    ia, ja, a, diag = [1], [], [], []
    for i, row in enumerate(rows):
        for j, v in sorted(row + [(i, 1.1 * sum(abs(v) for _, v in row))]):
            if j == i:
                diag.append(len(ja) + 1)
            ja.append(j + 1)
            a.append(v)
        ia.append(len(ja) + 1)
    return np.array(ia, np.int32), np.array(ja, np.int32), np.array(a), np.array(diag, np.int32), rng.uniform(-1, 1, n)


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("kind", sorted(OFFSETS))
@pytest.mark.parametrize("n", [34, 1022, 1026, 2050, 65540])
def test_coloured_loop_reaches_the_tolerance(ctx, oracle, fc, mode, kind, n):
    ia, ja, a, diag, b = even_ring(n, kind)
    ctx.set_precision(fc.FC_PREC_MIXED_COLOURED if mode == "mixed" else fc.FC_PREC_COLOURED_FP64, 1e-5, 0)
    try:
        x, _, info, st = ctx.csrsolve("iccg", ia, ja, a, diag, np.zeros(n), b, 2000, 0.0, 1e-10)
    finally:
        ctx.set_precision(0)
    assert st == 0 and 2 <= info.outer_iterations <= 6
    r = b - oracle.spmv(ia, ja, a, x)
    assert np.abs(r).sum() < 1.02e-10 * np.abs(b).sum()
