"""Tile widths past the 160 out-directions that the tensor-core kernel's tiles
hold, as callers or schedule tables of builds with wider tiles give them."""
import numpy as np
import pytest

from relativistic_solver_hllc_gb300 import PHASE_HG, Batch
from relativistic_solver_hllc_gb300._native import problem_desc

pytestmark = pytest.mark.gpu


def run(ctx, M, bn):
    before = ctx.hbm_used()
    with Batch(ctx) as b:
        pid = b.add_synthetic(problem_desc(2000, M, 1, PHASE_HG, 0.5, bn=bn), 3, 0.0, 1.0, 0.1, 1.0, [0.7])
        held = ctx.hbm_used() - before
        for _ in range(2):
            b.step(True)
        S, _ = b.read(pid)
    return held, S.copy()


@pytest.mark.parametrize("M,bn", [(200, 208), (200, 176), (330, 240), (500, 256)])
def test_widths_past_the_tile_are_balanced(ctx, tmp_path, M, bn):
    """Such a width counts as none: the same operands' memory and bits as the
    balanced default, not tiles cut to 160 with a last one nearly empty."""
    default = run(ctx, M, 0)
    wide = run(ctx, M, bn)
    assert wide[0] == default[0] and np.array_equal(wide[1], default[1])
    table = tmp_path / "schedule.txt"
    table.write_text(f"{M} 2 1 -1 {bn} 0 1.0\n{M} 2 2 -1 {bn} 0 1.0\n")
    ctx.autotune_load(table)
    loaded = run(ctx, M, 0)
    assert loaded[0] == default[0] and np.array_equal(loaded[1], default[1])
