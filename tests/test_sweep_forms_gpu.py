"""The transport sweep's launch forms (128, 192, 256 and 512 threads per
direction, chosen from the number of directions and the mean size of a step;
with the most directions 128 and three factors an item), against the oracle,
and a face that two cells write.

Tolerance: 1e-12 relative for Illum and the norm, the FP64 contract of the
sweep (the longest dependency chain below has under 100 steps, each a few
units in the last place)."""
import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import LOCX0_DTYPE, _native, medium, mesh_cube

pytestmark = pytest.mark.gpu
TOL = 1e-12


def start(ctx, n, M):
    vert, pairs, normals = mesh_cube(n, 1, True)
    xyz, area, fa = oracle.fibonacci_directions(M)
    N = vert.shape[0]
    ctx.init(xyz, area, fa, N)
    ctx.sweep_set_mesh(vert, pairs, normals)
    ctx.sweep_build()
    rng = np.random.default_rng(n + M)
    a, b, q = rng.uniform(0.5, 3.0, N), rng.uniform(0.0, 2.0, N), rng.uniform(0.0, 1.5, N)
    ctx.sweep_set_medium(medium(), a, b, q, (0.75, 0.25, 1.0, 0.5))
    return vert, pairs, normals, xyz, N, rng, a, b, q


@pytest.mark.parametrize("n,M", [(6, 3), (10, 5), (14, 3), (10, 160), (9, 310), (5, 461), (5, 767)])
def test_sweep_forms_match_oracle(ctx, n, M):
    vert, pairs, normals, xyz, N, rng, a, b, q = start(ctx, n, M)
    il0 = rng.uniform(0.1, 1.0, (M, N, 4))
    S = ctx.scattering(il0.ravel()).reshape(M, N)
    st = oracle.SweepStructures(vert, pairs, normals, xyz)
    il = il0.copy()
    for form in ("store", "read", "evaluate"):
        ref = oracle.sweep(st, S, a, b, q, il, bc=(0.75, 0.25, 1.0, 0.5))
        ctx.set_tuning(_native.TUNE_SWEEP_CACHE, form != "evaluate")
        norm = ctx.sweep()
        got = np.empty(M * N * 4)
        ctx.read_illum(got)
        assert np.max(np.abs(got - il.ravel()) / il.ravel()) <= TOL, form
        # the second and third sweep repeat the first: their norm is 0 up to its rounding
        assert abs(norm - ref) <= TOL * max(1.0, ref), (form, norm, ref)


def test_face_that_two_cells_write(ctx):
    """An out-face shared with a cell for which it is an out-face too (a file
    may say so of a face that the direction lies in): the later cell's value
    stays, and its change is measured against what the earlier cell wrote."""
    vert, pairs, normals, xyz, N, rng, a, b, q = start(ctx, 3, 1)
    pairs = np.asarray(pairs).reshape(N, 4)
    order, states, recs = ctx.sweep_export_direction(0)
    lev = oracle.SweepStructures(vert, pairs.ravel(), normals, xyz).levels[0]
    step = np.empty(N, int)
    for L in range(len(lev) - 1):
        step[order[lev[L]:lev[L + 1]]] = L
    il0 = rng.uniform(0.1, 1.0, N * 4)
    ctx.scattering(il0)
    ctx.sweep()
    first = np.empty(N * 4)
    ctx.read_illum(first)
    # an in-face g of cell c from an earlier cell, where another in-face keeps c in a later step than that cell
    pick = None
    for c in order[::-1]:
        ins = [f for f in range(4) if (states[c] >> f) & 1 and pairs[c, f] >= 0]
        for g in ins:
            u = pairs[c, g] >> 2
            if any(step[pairs[c, f] >> 2] >= step[u] and f != g for f in ins):
                pick = pick or (int(c), g, int(pairs[c, g]), [f for f in ins if f != g][0])
    c, g, face, other = pick
    states2 = states.copy()
    states2[c] &= ~(1 << g)
    out, at = [], 0
    for x in order:
        for f in range(4):
            if (states2[x] >> f) & 1:
                continue
            if (states[x] >> f) & 1:  # the new out-face: three nodes fed by the other in-face
                extra = np.zeros(3, LOCX0_DTYPE)
                extra["s"], extra["in_face_id"] = (0.1, 0.2, 0.3), other
                out.append(extra)
                continue
            block = recs[at:at + 3].copy()
            if x == c:
                block["in_face_id"] = other
            out.append(block)
            at += 3
    ctx.sweep_import_direction(0, order, states2, np.concatenate(out))
    ctx.copy_illum(il0)
    ctx.sweep()
    ctx.sweep()
    norm = ctx.sweep()
    got = np.empty(N * 4)
    ctx.read_illum(got)
    early, late = first[face], got[4 * c + g]
    assert got[face] == late != early
    expect = max(abs(late - early) / early, abs(early - late) / late)
    assert abs(norm - expect) <= TOL * max(1.0, expect)
