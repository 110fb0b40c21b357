"""The persistent loop of the coloured inner ICCG where a thread has more than one
row of a colour and more than one group of four rows, and where the blocks of a
whole wave exchange their sums: a grid in the plane (rows of up to four entries)
and one in space (six), odd sizes, both value types.

Tolerance as in test_gpu_coloured_loop.py: the refinement stops at sum |b - A x| <
tol * sum |b| in FP64, and the same sum formed here differs by rounding, 1e-12 of
r, whose entries cancel to 1e-10 of |b|: 1e-2, hence the 1.02.  Five digits a
refinement and a condition number below 100 keep the outer iterations few."""
import numpy as np
import pytest

import sweep_cases as cases

pytestmark = pytest.mark.gpu

BLOCK = 512  # rows of a block, at most two blocks an SM


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("box", [(791, 789, 1), (101, 97, 65)])
def test_loop_with_several_rows_a_thread(ctx, oracle, fc, mode, box):
    import torch
    wave = 2 * BLOCK * torch.cuda.get_device_properties(0).multi_processor_count
    ia, ja, dg, a = cases.grid(*box)
    n = len(dg)
    assert n // 4 > wave and n % 4 and n % (2 * wave)
    b = np.random.default_rng(4).uniform(-1.0, 1.0, n)
    ctx.set_precision(fc.FC_PREC_MIXED_COLOURED if mode == "mixed" else fc.FC_PREC_COLOURED_FP64, 1e-5, 0)
    try:
        x, _, info, st = ctx.csrsolve("iccg", ia + 1, ja + 1, a, dg + 1, np.zeros(n), b, 2000, 0.0, 1e-10)
        assert ctx.mixed_colours(1) == 2
    finally:
        ctx.set_precision(fc.FC_PREC_FP64)
        ctx.pattern_forget()
    assert st == 0 and 2 <= info.outer_iterations <= 6
    assert np.abs(b - oracle.spmv(ia + 1, ja + 1, a, x)).sum() < 1.02e-10 * np.abs(b).sum()
