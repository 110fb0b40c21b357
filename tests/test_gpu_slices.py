"""The solvers' matrix passes by slices of 32 rows and their 16-byte vector
passes, against the oracle, where these have remainders: systems of one row
below, at and above a slice, of odd sizes, at the last size that a single block
solves and the first that takes more, with rows of 5 entries, of 7 (the widths
whose loads are unrolled), and with one long row among short ones.

Tolerance: the passes keep each row's order of terms, so the iterates differ
from the oracle's only through FMA and the order of the FP64 sums.  The
systems are diagonally dominant by a tenth (condition number below 100),
so four iterations carry a relative 1e-16 * sqrt(n) * 100 < 1e-12 of each sum on;
1e-10 leaves two digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ring_system(n, kind, symmetric):
    rng = np.random.default_rng(n)
    pairs = set()
    for off in {"five": (1, 7), "seven": (1, 7, 29), "arrow": (1,)}[kind]:
        pairs |= {(min(i, (i + off) % n), max(i, (i + off) % n)) for i in range(n) if off % n}
    if kind == "arrow":
        pairs |= {(n // 2, j) if j > n // 2 else (j, n // 2) for j in range(0, n, max(3, n // 150)) if j != n // 2}
    rows = [[] for _ in range(n)]
    for i, j in sorted(pairs):
        v = -rng.uniform(0.5, 1.5)
        rows[i].append((j, v))
        rows[j].append((i, v if symmetric else -rng.uniform(0.5, 1.5)))
    ia, ja, a, diag = [1], [], [], []
    for i, row in enumerate(rows):
        for j, v in sorted(row + [(i, 1.1 * sum(abs(v) for _, v in row))]):
            if j == i:
                diag.append(len(ja) + 1)
            ja.append(j + 1)
            a.append(v)
        ia.append(len(ja) + 1)
    b = rng.uniform(-1.0, 1.0, n)
    return (np.array(ia, np.int32), np.array(ja, np.int32), np.array(a), np.array(diag, np.int32), np.zeros(n), b)


@pytest.mark.parametrize("solver", ["iccg", "bicgstab"])
@pytest.mark.parametrize("kind", ["five", "seven", "arrow"])
@pytest.mark.parametrize("n", [31, 32, 33, 63, 2560, 2561, 4999])
def test_slices_match_oracle(ctx, oracle, solver, kind, n):
    args = ring_system(n, kind, solver == "iccg") + (4, 1e-30, 1e-30)
    xo, r0o, info_o, _ = oracle.solve(solver, *args)
    x, r0, info, st = ctx.csrsolve(solver, *args)
    assert st >= 0 and info.itr_used == int(info_o[0])
    assert r0 == pytest.approx(r0o, rel=1e-12)
    np.testing.assert_allclose(x, xo, rtol=0, atol=1e-10 * np.abs(xo).max())
