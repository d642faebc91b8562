"""What the FP64 integrals' digit products report of themselves: that they ran,
which rows they left to the FP64 cores, and contractions that gave up."""
from fractions import Fraction

import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import PHASE_HG, STREAM_SCATTERING_1, RtsError, _native

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 contract, relative


def rel_err(a, b):
    return float(np.max(np.abs(a - b) / np.abs(b)))


def hg_weights(xyz, area, g):
    w = area[:, None] * (1 - g * g) / (4 * np.pi * (1 + g * g - 2 * g * (xyz @ xyz.T)) ** 1.5)
    return w / w.sum(axis=0, keepdims=True)


def rows_left(W, il, N, M):
    """Rows with an output below half of 2^(exponent of the row's largest face
    sum + exponent of the column's largest weight), or without digits."""
    sums = 4.0 * oracle.face_mean(il, N, M)
    top = sums.max(axis=0)
    bad = (sums.min(axis=0) < 0) | ~np.isfinite(top) | (np.abs(np.frexp(top)[1]) > 900)
    e_row, e_col = np.frexp(top)[1], np.frexp(W.max(axis=0))[1]
    with np.errstate(all="ignore"):
        low = (W.T @ sums < 0.5 * np.ldexp(1.0, e_row[None, :] + e_col[:, None])).any(axis=0)
    return int((bad | (low & (top > 0))).sum())


@pytest.mark.parametrize("M,N,g,sigma", [(64, 4001, None, 1.0), (100, 3000, None, 1.5), (257, 300, None, 1.0),
                                         (200, 1001, 0.5, 1.0), (200, 1001, 0.6, 1.5)])
def test_digits_run_and_list_their_rows(ctx, M, N, g, sigma):
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, sigma, N, M, independent_faces=True).reshape(M, N, 4)
    il[M // 2, 11::401] *= 1e6   # one direction carries these rows
    il[0, 7::301, 1] *= -1e5     # and these have a negative value
    il[:, 5::211] = 0.0
    il = np.ascontiguousarray(il).ravel()
    ctx.init(xyz, area, fa, N)
    if g is not None:
        ctx.set_phase(PHASE_HG, g)
    W = hg_weights(xyz, area, g) if g is not None else oracle.weights_thomson(xyz, area, fa)
    left = rows_left(W, il, N, M)
    assert left > 0
    assert ctx.fp64_stats() == (0, 0, 0)
    ctx.scattering(il)
    assert ctx.fp64_stats() == (1, left, 0)
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 0)
    ctx.scattering(il)
    assert ctx.fp64_stats() == (1, left, 0)


@pytest.mark.parametrize("M,N", [(100, 1500), (200, 700)])
def test_a_contraction_that_gives_up(ctx, M, N):
    """Its outputs are computed again as the FP64 cores' chain; a step's residual
    is reported as lost, until the next set-up."""
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, 1.0, N, M, independent_faces=True)
    B = oracle.uniform(2, 2, 0.1, 1.0, N)
    ctx.init(xyz, area, fa, N)
    S = {}
    for mode in (0, 2):
        ctx.set_tuning(_native.TUNE_FP64_DIGITS, mode)
        S[mode] = ctx.scattering(il)
    assert np.array_equal(S[0], S[2])
    assert rel_err(S[2], oracle.calculate_int_cpu(N, xyz, area, fa, il)) <= TOL
    assert ctx.fp64_stats() == (1, 0, 1)
    ctx.copy_illum(il)
    ctx.solve_setup("fp64", B, 0.9)
    with pytest.raises(RtsError) as err:
        ctx.solve_step(True)
    assert err.value.status == _native.ERR_DEVICE_WAIT
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 1)
    ctx.solve_step_async(True)
    with pytest.raises(RtsError):
        ctx.solve_residual_history(2)
    ctx.copy_illum(il)
    ctx.solve_setup("fp64", B, 0.9)
    W = oracle.weights_thomson(xyz, area, fa)
    _, ref, _ = oracle.iterate(W, oracle.face_mean(il, N, M), B, 0.9, 2, True)
    res = [ctx.solve_step(True) for _ in range(2)]
    assert np.max(np.abs(np.array(res) - np.array(ref)) / np.array(ref)) <= 1e-11
    assert ctx.fp64_stats()[2] == 2


@pytest.mark.parametrize("M,N", [(64, 2600), (100, 1500), (159, 500)])
def test_shards_take_the_route_of_the_whole(ctx, M, N):
    """Just above the size limit of the whole direction set: a shard of the
    out-directions gives the bits that all of them give."""
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, 1.0, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N)
    whole = ctx.scattering(il)
    for lo, hi in ((0, M // 2), (M // 2, M - 3), (M - 3, M)):
        ctx.init(xyz, area, fa, N, lo, hi)
        assert np.array_equal(ctx.scattering(il), whole[lo:hi])


def test_less_scratch_takes_more_passes(ctx):
    """A tight budget cuts a call into passes with the same bits; without room for
    a tile per SM the FP64 cores run, within the same tolerance."""
    M, N = 200, 60001
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(8, 0.0, 1.0, N, M, independent_faces=True).reshape(M, N, 4)
    il[M // 2, 11::4001] *= 1e6  # rows left to the FP64 cores, in every pass
    il = np.ascontiguousarray(il).ravel()
    ctx.init(xyz, area, fa, N)
    S = ctx.scattering(il)
    used = ctx.hbm_used()
    one, listed, _ = ctx.fp64_stats()
    assert one == 1 and listed == len(range(11, N, 4001))
    ctx.set_hbm_budget(used + (50 << 20))  # the digit rows of all cells take 161 MB
    assert np.array_equal(ctx.scattering(il), S)
    assert ctx.fp64_stats() == (5, 2 * listed, 0)
    ctx.set_hbm_budget(used + (4 << 20))
    chain = ctx.scattering(il)
    assert ctx.fp64_stats() == (5, 2 * listed, 0)
    ctx.set_hbm_budget(1 << 36)
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 0)
    assert np.array_equal(chain, ctx.scattering(il)) and rel_err(chain, S) <= TOL


def test_a_capturing_stream_takes_the_chain(ctx):
    torch = pytest.importorskip("torch")
    M, N = 100, 1500
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(4, 0.0, 1.0, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N)
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 0)
    chain = ctx.scattering(il)
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 1)
    out = ctx.host_scattering()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(ctx.stream_handle(STREAM_SCATTERING_1))):
        ctx.scattering_async(0, M, STREAM_SCATTERING_1, out)
    out[:] = 0.0
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.reshape(M, N), chain)
    assert ctx.fp64_stats() == (0, 0, 0)


@pytest.mark.parametrize("M,N", [(80, 32001), (96, 33000), (100, 22501), (120, 19600), (128, 19457),  # waves of large tiles
                                 (97, 1300), (161, 77)])                                              # small tiles only
def test_listed_rows_get_the_chain(ctx, M, N):
    """Rows with a negative value are computed whole on the FP64 cores: with all of
    them listed every output and the residual have the chain's bits, in the large,
    the narrow and the small tiles, and for a range of out-directions."""
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, 1.0, N, M, independent_faces=True).reshape(M, N, 4)
    il[M // 3] *= -1.0
    il = np.ascontiguousarray(il).ravel()
    B = oracle.uniform(2, 2, 0.1, 1.0, N)
    ctx.init(xyz, area, fa, N)
    got = {}
    for mode in (0, 1):
        ctx.set_tuning(_native.TUNE_FP64_DIGITS, mode)
        S = ctx.scattering(il)
        part = np.zeros(M * N)
        ctx.scattering_async(7, M - 1, STREAM_SCATTERING_1, part)
        ctx.wait()
        ctx.solve_setup("fp64", B, 0.9)
        res = [ctx.solve_step(False) for _ in range(2)]
        got[mode] = (S, part, ctx.solve_read(), np.array(res))
    assert ctx.fp64_stats() == (4, 4 * N, 0)
    for a, b in zip(got[0], got[1]):
        assert np.array_equal(a, b)


def test_kernel_timing_covers_the_listed_rows(ctx):
    """With every row listed an integral's time is the FP64 cores' and more."""
    M, N = 200, 20000
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, 1.0, N, M, independent_faces=True).reshape(M, N, 4)
    il[M // 3] *= -1.0
    ctx.init(xyz, area, fa, N)
    ctx.copy_illum(il.ravel())
    ms = {}
    for mode in (0, 1):
        ctx.set_tuning(_native.TUNE_FP64_DIGITS, mode)
        ctx.solve_setup("fp64", np.ones(N), 0.9)
        ctx.solve_step(False)
        ctx.kernel_timing(True)
        for _ in range(3):
            ctx.solve_step(False)
        ms[mode], launches = ctx.kernel_timing(False)
        assert launches == 3
    assert ms[1] > 0.9 * ms[0]


@pytest.mark.parametrize("g", [None, 0.0, 0.4])
def test_error_bound_of_the_digits(ctx, g):
    """Rows of one direction, of equal values and of lognormal ones against exact
    sums of the device's own W, output by output: in units of 2^-54 of the row's and
    the column's powers of two, 1.26 a direction (the products left out), half of
    both scaled operands a direction (their last digits), 0.75 per 32 directions
    (D_5), and half a unit in the last place of S."""
    M, N = 161, 200
    xyz, area, fa = oracle.fibonacci_directions(M)
    ctx.init(xyz, area, fa, N)
    if g is not None:
        ctx.set_phase(PHASE_HG, g)
    il = np.zeros((M, N, 4))
    il[np.arange(M), np.arange(M), 0] = 4.0  # Ibar is the unit matrix: the chain gives W itself
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 0)
    W = ctx.scattering(il.ravel())[:, :M].T.copy()
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 1)
    rng = np.random.default_rng(2)
    ibar = rng.lognormal(0.0, 1.0, (M, N))
    ibar[:, :8] = 0.0
    ibar[rng.integers(0, M, 8), np.arange(8)] = rng.uniform(0.5, 1.0, 8)
    ibar[:, 8:12] = rng.uniform(0.5, 1.0, 4)
    il[:] = 0.0
    il[..., 2] = 4.0 * ibar
    S = ctx.scattering(il.ravel())
    assert ctx.fp64_stats()[0] == 1
    e_col = np.frexp(W.max(axis=0))[1]
    taken = 0
    for c in range(16):
        e_row = int(np.frexp(ibar[:, c].max())[1])
        used = np.flatnonzero(ibar[:, c])
        a = {j: Fraction(float(ibar[j, c])) for j in used}
        for k in range(M):
            exact = sum((a[j] * Fraction(float(W[j, k])) for j in used), Fraction(0))
            scale = Fraction(2) ** (e_row + int(e_col[k]))
            if exact < scale / 2:
                continue  # the chain's
            taken += 1
            last = float((ibar[:, c] / 2.0 ** e_row + W[:, k] / 2.0 ** int(e_col[k])).sum()) / 2
            bound = Fraction(1.26 * M + last + 0.75 * -(-M // 32)) * scale / 2 ** 54
            bound += Fraction(float(np.spacing(S[k, c]))) / 2
            assert abs(Fraction(float(S[k, c])) - exact) <= bound, (c, k)
    assert taken > 8 * M
