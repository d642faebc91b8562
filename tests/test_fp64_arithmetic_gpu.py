"""The switch between the two arithmetics of the FP64 integrals: the tensor
cores' digit products, and the chain of FP64 multiply-adds."""
import ctypes as C

import numpy as np
import pytest

import oracle
from relativistic_solver_hllc_gb300 import _native
from test_compat_gpu import _run_driver, build_driver

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the FP64 contract, relative


def rel_err(a, b):
    return float(np.max(np.abs(a - b) / np.abs(b)))


def noalloc(lib, il, xyz, area, fa, N, M):
    """rts_scattering_noalloc, which always runs the chain."""
    torch = pytest.importorskip("torch")
    d = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda") for a in (il, xyz, area)]
    S = torch.zeros(M * N, dtype=torch.float64, device="cuda")
    fn = lib.rts_scattering_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p] * 3 + [C.c_int64] * 2 + [C.c_double] + [C.c_void_p] * 2
    assert fn(*(t.data_ptr() for t in d), N, M, fa, S.data_ptr(), torch.cuda.current_stream().cuda_stream) == _native.OK
    torch.cuda.synchronize()
    return S.cpu().numpy().reshape(M, N)


@pytest.mark.parametrize("M,N", [(100, 1500), (200, 300), (260, 9000)])
def test_chain_on_request(ctx, native_lib, M, N):
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(M, 0.0, 1.0, N, M, independent_faces=True)
    ctx.init(xyz, area, fa, N)
    digits = ctx.scattering(il)
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 0)
    chain = ctx.scattering(il)
    assert np.array_equal(chain, noalloc(native_lib, il, xyz, area, fa, N, M))
    assert not np.array_equal(chain, digits) and rel_err(digits, chain) <= TOL
    ctx.set_tuning(_native.TUNE_FP64_DIGITS, 1)
    assert np.array_equal(ctx.scattering(il), digits)
    with pytest.raises(_native.RtsError):
        ctx.set_tuning(_native.TUNE_FP64_DIGITS, 5)


def test_chain_through_the_shim(native_lib, tmp_path):
    exe = build_driver(tmp_path)
    N, M = 1500, 100
    xyz, area, fa = oracle.fibonacci_directions(M)
    il = oracle.illum(13, 0.0, 1.0, N, M, independent_faces=True)
    out = {}
    for precision in ("fp64", "fp64_chain"):
        (tmp_path / precision).mkdir()
        a, b = _run_driver(exe, tmp_path / precision, xyz, area, fa, il, N, 3, {"RTS_SCATTER_PRECISION": precision})
        assert np.array_equal(a, b)
        out[precision] = a
    assert np.array_equal(out["fp64_chain"], noalloc(native_lib, il, xyz, area, fa, N, M))
    assert not np.array_equal(out["fp64"], out["fp64_chain"])
