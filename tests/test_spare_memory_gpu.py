"""Memory that a context can do without -- the digits of W of the FP64 integrals,
the sweep's copy words and attenuation factors -- gives way to allocations that
it needs, under the tightest budgets that hold everything else."""
import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import Context, RtsError, medium, mesh_cube

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 contract, relative
SLACK = 4096


def mesh_context(ctx, n, M):
    vert, pairs, normals = mesh_cube(n, 1, True)
    xyz, area, fa = oracle.fibonacci_directions(M)
    N = vert.shape[0]
    ctx.init(xyz, area, fa, N)
    ctx.sweep_set_mesh(vert, pairs, normals)
    return N


def two_sweeps(ctx, N, M):
    rng = np.random.default_rng(3)
    ctx.sweep_set_medium(medium(), rng.uniform(0.5, 1.5, N), rng.uniform(0.5, 1.5, N), rng.uniform(0.1, 1.0, N))
    ctx.copy_illum(rng.uniform(0.1, 1.0, M * N * 4))
    ctx.send_scattering(rng.uniform(0.1, 1.0, M * N))
    norms = [ctx.sweep() for _ in range(2)]
    il = np.empty(M * N * 4)
    ctx.read_illum(il)
    return il, norms


@pytest.mark.parametrize("n,M", [(6, 8), (5, 160)])
def test_structures_fit_without_their_words(ctx, n, M):
    """Building and importing succeed in the memory that they need without copy
    words, and the sweeps give the same bits."""
    N = mesh_context(ctx, n, M)
    records, _ = ctx.sweep_build()
    words = 4 * records // 3 + 8 * M           # and their table
    build = ctx.hbm_used() - words
    temporary = M * N + 16 * 8 * 4 * N         # states and face frames while the structures are built
    exported = [ctx.sweep_export_direction(d) for d in range(M)]
    ref, ref_norms = two_sweeps(ctx, N, M)
    for way in ("build", "import"):
        with Context(0) as tight:
            mesh_context(tight, n, M)
            if way == "build":
                tight.set_hbm_budget(build + temporary + SLACK)
                tight.sweep_build()
            else:
                tight.set_hbm_budget(build + 64 * M + SLACK)  # blocks of a direction are at least 16 bytes
                for d in range(M):
                    tight.sweep_import_direction(d, *exported[d])
            il, norms = two_sweeps(tight, N, M)
            assert np.array_equal(il, ref) and norms == ref_norms


def test_factors_give_way(ctx):
    n, M = 6, 8
    N = mesh_context(ctx, n, M)
    ctx.sweep_build()
    ref, ref_norms = two_sweeps(ctx, N, M)
    ctx.set_hbm_budget(ctx.hbm_used())
    rng = np.random.default_rng(1)
    ctx.set_geometry(rng.uniform(-1, 1, (N, 4, 3)), rng.uniform(0.5, 1.0, (N, 4)), rng.uniform(0.5, 1.0, N))
    il, norms = two_sweeps(ctx, N, M)
    assert np.array_equal(il, ref) and norms == ref_norms


def test_digits_of_w_give_way(ctx):
    M, N = 200, 1000
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(5, 0.0, 1.0, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N)
    before = ctx.hbm_used()
    S = ctx.scattering(il)
    assert ctx.hbm_used() > before  # the digits of W
    ctx.set_hbm_budget(ctx.hbm_used())
    rng = np.random.default_rng(1)
    ctx.set_geometry(rng.uniform(-1, 1, (N, 4, 3)), rng.uniform(0.5, 1.0, (N, 4)), rng.uniform(0.5, 1.0, N))
    again = ctx.scattering(il)
    assert np.max(np.abs(again - S) / S) <= TOL
    # and to a budget as low as before them
    ctx.set_hbm_budget(1 << 34)
    assert np.array_equal(ctx.scattering(il), S)
    geometry = 17 * 8 * N
    ctx.set_hbm_budget(before + geometry)
    with pytest.raises(RtsError):
        ctx.set_hbm_budget(before)


def test_unused_scratch_is_held_within_the_budget(ctx):
    torch = pytest.importorskip("torch")
    M, N = 200, 100000
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(5, 0.0, 1.0, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N)
    S = ctx.scattering(il)  # 270 MB of digit rows
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.set_hbm_budget(ctx.hbm_used() + (40 << 20))
    assert torch.cuda.mem_get_info()[0] - before >= 200 << 20
    assert np.array_equal(ctx.scattering(il), S)  # in passes
    before = torch.cuda.mem_get_info()[0]
    rng = np.random.default_rng(1)
    ctx.set_geometry(rng.uniform(-1, 1, (N, 4, 3)), rng.uniform(0.5, 1.0, (N, 4)), rng.uniform(0.5, 1.0, N))  # 14 MB
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20  # out of what the pool held unused
