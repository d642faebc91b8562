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


@pytest.mark.parametrize("M,N,lo,hi", [(40, 40001, 0, 40),      # FP64 kernel
                                       (100, 21003, 0, 100),    # digits, four ranges, a ragged last one
                                       (161, 6500, 30, 161)])   # digits, two ranges, some of the out-directions
def test_ranges_of_cells_match_one_piece(ctx, M, N, lo, hi):
    """Pinned arrays (ranges) and pageable ones (one piece) give the same bits,
    rows that the digits leave to the FP64 kernel in every range among them."""
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(7, 0.0, 1.0, N, M, independent_faces=True).reshape(M, N, 4)
    il[M // 3, 3::211] *= 1e7  # one direction carries these rows
    il[:, 5::307] = 0.0
    il = np.ascontiguousarray(il).ravel()
    B = oracle.uniform(2, 2, 0.1, 1.0, N)
    ctx.init(xyz, area, fa, N, lo, hi)
    pinned_il, pinned_S = ctx.host_illum(), ctx.host_scattering()
    pinned_il[:] = il
    for b, lam in ((None, 1.0), (B, 0.7)):
        one = ctx.scattering_update("fp64", il, b, lam, np.zeros((hi - lo) * N))
        pinned_S[:] = 0.0
        ctx.scattering_update("fp64", pinned_il, b, lam, pinned_S)
        assert np.array_equal(pinned_S, one)
        ref = oracle.calculate_int_cpu(N, xyz, area, fa, il, lo, hi - lo)
        if b is not None:
            ref = (1.0 - lam) * b[None, :] + lam * ref
        live = np.abs(ref) > 0
        assert rel_err(one.reshape(hi - lo, N)[live], ref[live]) <= TOL
        assert np.all(one.reshape(hi - lo, N)[~live] == 0.0)
