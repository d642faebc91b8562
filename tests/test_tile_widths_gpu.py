"""The tensor-core kernel's tiles at the widths where its column slices change
(one slice, two unequal ones, the widest tile, a second tile), and CTAs that
walk several tiles, whose accumulators, finished sums and row buffers take
turns.

Tolerances: relaxed iterations agree with the FP64 oracle to the split
formats' 2^-20 (FP16, TF32) and 2^-14 (BF16) relative, the error of their
products and sums; a cell's iteration does not depend on the other cells, so
a large problem and a small one agree bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL = {"fp16x3": 2.0 ** -20, "tf32x3": 2.0 ** -20, "bf16x3": 2.0 ** -14}


def iterate(ctx, prec, xyz, area, fa, il, B, N, steps=3):
    ctx.init(xyz, area, fa, N)
    ctx.copy_illum(il)
    ctx.solve_setup(prec, B, 0.9)
    for _ in range(steps):
        ctx.solve_step(True)
    return ctx.solve_read().copy().reshape(len(area), N)


@pytest.mark.parametrize("prec", ["fp16x3", "bf16x3", "tf32x3"])
@pytest.mark.parametrize("M", [15, 16, 31, 47, 79, 80, 111, 143, 159, 160, 322])
def test_widths(ctx, prec, M):
    N = 300
    rng = np.random.default_rng(M)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il, B = rng.uniform(0.1, 1.0, M * N * 4), rng.uniform(0.1, 1.0, N)
    S = iterate(ctx, prec, xyz, area, fa, il, B, N)
    W = oracle.weights_thomson(xyz, area, fa)
    ref, _, _ = oracle.iterate(W, oracle.face_mean(il, N, M), B, 0.9, 3, True)
    assert np.max(np.abs(S - ref) / np.abs(ref)) <= TOL[prec]


@pytest.mark.parametrize("prec,N,M", [("fp16x3", 60000, 47), ("tf32x3", 60000, 47), ("bf16x3", 30000, 200)])
def test_several_tiles_per_cta(ctx, prec, N, M):
    rng = np.random.default_rng(N)
    xyz, area, fa = oracle.fibonacci_directions(M)
    il, B = rng.uniform(0.1, 1.0, (M, N, 4)), rng.uniform(0.1, 1.0, N)
    S = iterate(ctx, prec, xyz, area, fa, il.ravel(), B, N)
    for a, b in ((0, 300), (N // 2 + 5, N // 2 + 400), (N - 130, N)):
        part = iterate(ctx, prec, xyz, area, fa, np.ascontiguousarray(il[:, a:b]).ravel(), B[a:b].copy(), b - a)
        assert np.array_equal(part, S[:, a:b]), (a, b)
