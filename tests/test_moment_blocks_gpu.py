"""The moment kernels' block sizes (64 or 128 cells, by the cell count and the
SMs): a cell's sums run over the directions in order whatever the block, so
each size gives the same bits."""
import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import STREAM_PARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [9728, 58368, 60000, 82944])  # 128, 128, 64 and 64 cells a block on 152 SMs
def test_block_sizes_agree(ctx, N):
    M = 7
    rng = np.random.default_rng(N)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = rng.uniform(0.1, 1.0, (M, N, 4))
    nrm, fS, vol = oracle.cell_geometry(43, N)
    nrm, fS, vol = np.asarray(nrm).reshape(N, 12), np.asarray(fS).reshape(N, 4), np.asarray(vol)

    def run(a, b):
        n = b - a
        ctx.init(xyz, area, fa, n)
        ctx.copy_illum(np.ascontiguousarray(il[:, a:b]).ravel())
        ctx.set_geometry(*(np.ascontiguousarray(x[a:b]).ravel() for x in (nrm, fS, vol)))
        parts = list(ctx.illum_params(STREAM_PARAMS)) + list(ctx.moments(STREAM_PARAMS))
        return [np.asarray(p).reshape(n, -1).copy() for p in parts]

    whole = run(0, N)
    for a, b in ((0, 65), (N - 130, N)):
        for w, p in zip(whole, run(a, b)):
            assert np.array_equal(w[a:b], p), (a, b)
