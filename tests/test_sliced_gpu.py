"""The FP64 integral on the tensor cores (digits of both operands, exact
products, 64-bit totals) against the oracle: sizes at the edges of its tiles
(128 cells x up to 128 out-directions, 32 in-directions a chunk), ranges of
out-directions, and the inputs it has to leave to the FP64 kernel -- rows with
infinities, NaN, values far above the rest, cancelling signs, exponents out of
range, zeros.

Tolerance 1e-12 relative, the FP64 contract; the digits carry 54 bits below a
row's largest value and outputs under half of that scale are recomputed, so
the error is of the order of 1e-15."""
import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import PHASE_HG, STREAM_SCATTERING_1, STREAM_SCATTERING_2

pytestmark = pytest.mark.gpu
TOL = 1e-12
WORK = 1.0e7  # cells x directions x out-directions from which the tensor cores run


def rel_err(a, b):
    return float(np.max(np.abs(a - b) / np.abs(b)))


def cells_for(M, extra):
    return int(WORK) // (M * M) + extra


@pytest.mark.parametrize("M,extra", [(48, 1), (64, 77), (65, 128), (127, 3), (128, 1), (129, 130), (160, 129), (257, 5)])
def test_sizes_match_the_oracle(ctx, M, extra):
    N = cells_for(M, extra)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, 1.5, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N)
    S = ctx.scattering(il).reshape(M, N)
    assert rel_err(S, oracle.calculate_int_cpu(N, xyz, area, fa, il)) <= TOL
    # any range of out-directions, on either stream, gives the same bits
    a, b = M // 3, M - 7
    out = np.zeros(M * N)
    ctx.scattering_async(a, b, STREAM_SCATTERING_2, out)
    ctx.scattering_async(0, a, STREAM_SCATTERING_1, out)
    ctx.scattering_async(b, M, STREAM_SCATTERING_1, out)
    ctx.wait()
    assert np.array_equal(out.reshape(M, N), S)


def test_shard_and_henyey_greenstein(ctx):
    M, lo, hi = 150, 20, 150
    N = cells_for(M, 301)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(3, 0.0, 1.0, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N, lo, hi)
    S = ctx.scattering(il).reshape(hi - lo, N)
    assert rel_err(S, oracle.calculate_int_cpu(N, xyz, area, fa, il, lo, hi - lo)) <= TOL
    ctx.set_phase(PHASE_HG, 0.4)  # new weights: the digits of W are built again
    S = ctx.scattering(il).reshape(hi - lo, N)
    mu = xyz @ xyz.T
    w = area[:, None] * (1 - 0.16) / (4 * np.pi * (1.16 - 0.8 * mu) ** 1.5)
    w /= w.sum(axis=0, keepdims=True)
    assert rel_err(S, w[:, lo:hi].T @ oracle.face_mean(il, N, M)) <= TOL


@pytest.mark.parametrize("M", [100])
def test_inputs_left_to_the_fp64_kernel(ctx, M):
    N = cells_for(M, 57)
    rng = np.random.default_rng(5)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(9, 0.0, 1.0, N, M, independent_faces=True).reshape(M, N, 4)
    cells = rng.permutation(N)
    part = {}
    for i, name in enumerate(("zero", "one", "huge", "tiny", "subnormal", "mixed", "signed", "inf", "nan", "overflow")):
        part[name] = cells[8 * i:8 * i + 8]
    il[:, part["zero"]] = 0.0
    il[:, part["one"]] = 0.0
    il[M // 2, part["one"]] = 1e3  # a single direction carries the row
    il[:, part["huge"]] *= 1e290
    il[:, part["tiny"]] *= 1e-290
    il[:, part["subnormal"]] *= 1e-310
    il[::7, part["mixed"]] *= 1e12
    il[:, part["signed"]] *= rng.choice([-1.0, 1.0], size=(M, 8, 1))
    il[3, part["inf"], 1] = np.inf
    il[M - 1, part["nan"], 2] = np.nan
    il[0, part["overflow"]] = 1.7e308  # the face sum overflows
    ctx.init(xyz, area, fa, N)
    with np.errstate(all="ignore"):
        S = ctx.scattering(il.ravel()).reshape(M, N)
        ref = oracle.calculate_int_cpu(N, xyz, area, fa, il.ravel())
    rest = np.setdiff1d(np.arange(N), np.concatenate([part[k] for k in ("zero", "signed", "inf", "nan", "overflow",
                                                                       "subnormal")]))
    assert rel_err(S[:, rest], ref[:, rest]) <= TOL
    assert np.all(S[:, part["zero"]] == 0.0)
    assert np.array_equal(np.isnan(S), np.isnan(ref)) and np.array_equal(np.isinf(S), np.isinf(ref))
    assert np.allclose(S[:, part["subnormal"]], ref[:, part["subnormal"]], rtol=1e-6, atol=0.0)
    W = oracle.weights_thomson(xyz, area, fa)
    scale = W.T @ np.abs(oracle.face_mean(il.ravel(), N, M)[:, part["signed"]])
    assert float(np.max(np.abs(S[:, part["signed"]] - ref[:, part["signed"]]) / scale)) <= TOL


def test_relaxed_iteration(ctx):
    """Update, residual and relaxation, with rows that take the FP64 kernel."""
    M, lam, steps = 120, 0.9, 3
    N = cells_for(M, 200)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(6, 0.0, 1.0, N, M, independent_faces=True).reshape(M, N, 4)
    il[0, 5::97] *= 1e5
    il[:, 7::101] = 0.0
    il = np.ascontiguousarray(il).ravel()
    B = oracle.uniform(2, 2, 0.1, 1.0, N)
    ctx.init(xyz, area, fa, N)
    ctx.copy_illum(il)
    ctx.solve_setup("fp64", B, lam)
    res = [ctx.solve_step(True) for _ in range(steps)]
    W = oracle.weights_thomson(xyz, area, fa)
    S_ref, res_ref, _ = oracle.iterate(W, oracle.face_mean(il, N, M), B, lam, steps, True)
    assert rel_err(ctx.solve_read(), S_ref) <= TOL
    assert np.max(np.abs(np.array(res) - np.array(res_ref)) / np.array(res_ref)) <= 1e-11
