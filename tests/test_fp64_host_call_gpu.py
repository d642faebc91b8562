"""The FP64 host-buffer calls on pinned arrays, which copy and compute in ranges
of cells where the strided copies of a range allow it."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 contract, relative


def rel_err(a, b):
    return float(np.max(np.abs(a - b) / np.abs(b)))


def test_rows_past_the_pitch_of_a_strided_copy(ctx):
    """2^26 cells: a direction's 2^31 bytes exceed the largest pitch, 2^31 - 1."""
    N, M, period = 1 << 26, 2, 1009
    xyz, area, fa = oracle.fibonacci_directions(M)
    ctx.init(xyz, area, fa, N)
    il, S = ctx.host_illum(), ctx.host_scattering()
    some = oracle.illum(3, 0.0, 1.0, period, M, independent_faces=True)
    for j in range(M):
        il[4 * N * j:4 * N * (j + 1)] = np.resize(some[4 * period * j:4 * period * (j + 1)], 4 * N)
    S[:] = 0.0
    ctx.scattering_update("fp64", il, None, 1.0, S)
    ref = oracle.calculate_int_cpu(period, xyz, area, fa, some)
    for k in range(M):
        assert rel_err(S[k * N:(k + 1) * N], np.resize(ref[k], N)) <= TOL
