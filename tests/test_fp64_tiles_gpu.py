"""The FP64 kernels' two tile sizes: a call large enough for 128 x 64 tiles
against calls on parts of its cells, which take the 32 x 32 ones.

Both make every output by the same chain of FP64 multiply-adds over the
in-directions, so the outputs are equal bit for bit."""
import ctypes as C

import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import _native

pytestmark = pytest.mark.gpu


def call(lib, torch, il, d_xyz, d_area, fa):
    """rts_scattering_noalloc on Illum [M][N][4]."""
    M, N = il.shape[:2]
    d_S = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    fn = lib.rts_scattering_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64, C.c_int64, C.c_double, C.c_void_p, C.c_void_p]
    assert fn(il.data_ptr(), d_xyz.data_ptr(), d_area.data_ptr(), N, M, fa, d_S.data_ptr(),
              torch.cuda.current_stream().cuda_stream) == _native.OK
    torch.cuda.synchronize()
    return d_S


@pytest.mark.parametrize("N,M", [(77830, 33), (38950, 70), (25999, 130)])
def test_tile_sizes_agree(native_lib, N, M):
    import torch

    xyz, area, fa = oracle.fibonacci_directions(M)
    d_xyz, d_area = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (xyz, area))
    il = torch.rand((M, N, 4), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(N))
    S = call(native_lib, torch, il, d_xyz, d_area, fa)
    assert torch.isfinite(S).all()
    for a, b in ((0, 1), (1, 34), (N // 2, N // 2 + 1000), (N - 129, N)):
        part = call(native_lib, torch, il[:, a:b].contiguous(), d_xyz, d_area, fa)
        assert torch.equal(part, S[:, a:b]), (a, b)
