"""What a result looks like when a bounded wait of its kernel runs out: a build of
the product and solve kernels in which every wait that may give up gives up at
once (copies and products in flight are still waited for).  No result may come out
as finite numbers, and the status word says MGT_ERR_TIMEOUT where
mgt_workspace_status reads it."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WRAPPER = r"""
#include "zgemm_tc.cuh"
namespace mgt {
int tri_solve(const float2*, int64_t, float2*, int64_t, int, int, void*, bool, cudaStream_t);
size_t tri_solve_workspace_bytes(int64_t n);
}
using namespace mgt;
extern "C" size_t t_bytes(int what, int64_t m, int64_t n, int64_t k) {
  return what == 0 ? zgemm_wide_bytes(m, n, k) + 256 : what == 1 ? zsolve_workspace_bytes(m, n) : tri_solve_workspace_bytes(m);
}
extern "C" int t_wide(const void* A, int M, const void* B, int N, int K, void* out, void* work) {
  return zgemm_wide((const double2*)A, K, M, (const double2*)B, N, N, K, nullptr, 0, (double2*)out, N, (char*)work + 256,
                    (int*)((char*)work + kStatusOffset), 0);
}
extern "C" int t_zsolve(const void* F, void* X, int n, int r, void* work) {
  return zsolve((const double2*)F, n, (double2*)X, r, n, r, work, 0);
}
extern "C" int t_trisolve(const void* F, void* X, int n, int r, void* work) {
  return tri_solve((const float2*)F, n, (float2*)X, r, n, r, work, false, 0);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from magreete_gb300 import build
    d = tmp_path_factory.mktemp("expired")
    (d / "wrapper.cu").write_text(WRAPPER)
    out = str(d / "libexpired.so")
    src = [str(d / "wrapper.cu")] + [os.path.join(build.CSRC, f) for f in
                                     ("zgemm_tc.cu", "zsolve.cu", "trsolve.cu", "diag.cu")]
    subprocess.run([build.nvcc_path()] + build.ARCH +
                   ["-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", build.INCLUDE, "-I", build.CSRC,
                    "--expt-relaxed-constexpr", "-DMGT_ROLE_WAIT_LIMIT=0", "--threads", "5"] + src +
                   ["-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.t_bytes.restype = ctypes.c_size_t
    lib.t_bytes.argtypes = [ctypes.c_int] + [ctypes.c_int64] * 3
    return lib


def _work(lib, what, m, n, k=0):
    return torch.zeros(lib.t_bytes(what, m, n, k), dtype=torch.uint8, device="cuda")


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _status(work):
    torch.cuda.synchronize()
    return int(work[8:12].view(torch.int32).item())


def test_product(lib):
    from magreete_gb300 import _lib as L
    M, N, K = 300, 70, 200
    A, B = torch.randn(M, K, dtype=torch.complex128).cuda(), torch.randn(K, N, dtype=torch.complex128).cuda()
    out, work = torch.zeros(M, N, dtype=torch.complex128, device="cuda"), _work(lib, 0, M, N, K)
    assert lib.t_wide(_p(A), M, _p(B), N, K, _p(out), _p(work)) == 0
    assert _status(work) == L.MGT_ERR_TIMEOUT
    assert torch.isnan(torch.view_as_real(out)).all()


@pytest.mark.parametrize("complex64", [False, True])
def test_solves(lib, complex64):
    """Orders of several block rows: everything but the first block row of the last
    triangle depends on a product."""
    from magreete_gb300 import _lib as L
    n, R = 700, 40
    dt = torch.complex64 if complex64 else torch.complex128
    F = (0.01 * torch.randn(n, n, dtype=dt) + torch.eye(n)).cuda()
    X, work = torch.randn(n, R, dtype=dt).cuda(), _work(lib, 2 if complex64 else 1, n, R)
    fn = lib.t_trisolve if complex64 else lib.t_zsolve
    assert fn(_p(F), _p(X), n, R, _p(work)) == 0
    assert _status(work) == L.MGT_ERR_TIMEOUT
    assert not torch.isfinite(torch.view_as_real(X)).any()


def test_refined_solve(tmp_path):
    """A refined solve whose triangular solves ran out of waiting says so, instead of
    not having converged: the library with its solve steps alone built that way."""
    import glob
    from magreete_gb300 import _lib as L
    from magreete_gb300 import build
    from magreete_gb300 import engine as E
    # the other files as the library has them, their objects where the build left them
    others = [f for f in glob.glob(os.path.join(build.CSRC, "*.cu")) if os.path.basename(f) != "trsolve.cu"]
    objects = [os.path.join(build.BUILD, os.path.basename(f) + ".o") for f in others]
    for src, obj in zip(others, objects):
        if not os.path.exists(obj):
            subprocess.run([build.nvcc_path()] + build.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I",
                            build.INCLUDE, "--expt-relaxed-constexpr", "-c", src, "-o", str(tmp_path / os.path.basename(obj))],
                           check=True)
            objects[objects.index(obj)] = str(tmp_path / os.path.basename(obj))
    out = str(tmp_path / "libexpired_steps.so")
    subprocess.run([build.nvcc_path()] + build.ARCH +
                   ["-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", build.INCLUDE, "-I", build.CSRC,
                    "--expt-relaxed-constexpr", "-DMGT_ROLE_WAIT_LIMIT=0", os.path.join(build.CSRC, "trsolve.cu")] +
                   objects + ["-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.mgt_solve_refined.argtypes = L.SIGNATURES["mgt_solve_refined"][1]
    n, R = 600, 5
    pts = torch.rand(n, 3, dtype=torch.float64, generator=torch.Generator().manual_seed(1)).cuda()
    Mdf, M32 = E.assemble_system("3d_scalar", pts, 9.0, 0.05, 0.0, ("cdf", "c64"))
    f = E.lu_factor(M32)
    B = torch.randn(n, R, dtype=torch.complex128).cuda()
    X = torch.zeros_like(B)
    nb = ctypes.c_size_t()
    L.check(L.load().mgt_refine_workspace_bytes(n, R, ctypes.byref(nb)))
    work = torch.zeros(nb.value, dtype=torch.uint8, device="cuda")
    st = lib.mgt_solve_refined(E._ptr(Mdf), n, E._ptr(f.lu), f.lu.stride(0), E._ptr(f.perm), n, E._ptr(B), R, E._ptr(X),
                               R, R, 1e-10, 10, E._ptr(work), nb.value, None, None, E._stream())
    assert st == L.MGT_ERR_TIMEOUT
    assert not torch.isfinite(torch.view_as_real(X)).any()
