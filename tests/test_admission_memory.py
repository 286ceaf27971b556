"""What a request is admitted with against what it takes: many detectors before
few scatterers, where the propagation's workspace is most of it, and large systems
with few, in both precisions."""
import os

import pytest
import torch


def _problem(kind, N, R, T):
    from types import SimpleNamespace
    d = 2 if kind == "2d_vector" else 3 if kind == "3d_vector" else 1
    return SimpleNamespace(kind=kind, n=d * N, nrhs=R, d=d, detectors=torch.zeros(T, 2))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,N,R,T", [("2d_vector", 1000, 64, 22_500), ("2d_vector", 500, 64, 301 * 301),
                                        ("2d_scalar", 150, 1, 90_000), ("3d_vector", 4000, 64, 1024)])
def test_estimate_covers_the_precisions_own_workspaces(kind, N, R, T, precision):
    """Host-only queries: no GPU needed."""
    import ctypes
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    from magreete_gb300 import serve
    if not os.path.exists(L.LIB_PATH):
        pytest.skip("library not built")
    lib = L.load()
    prob = _problem(kind, N, R, T)
    nb = ctypes.c_size_t()
    need = {}
    for code in (L.MGT_C128, L.MGT_CDF):
        L.check(lib.mgt_propagate_workspace_bytes_for(E.KIND_CODE[kind], code, T, N, R, ctypes.byref(nb)))
        need[code] = nb.value
    L.check(lib.mgt_propagate_workspace_bytes(E.KIND_CODE[kind], T, N, R, ctypes.byref(nb)))
    assert nb.value == max(need.values())
    own = need[L.MGT_C128 if precision == "fp64" else L.MGT_CDF]
    fields = 16 * prob.d * R * (N + 2 * T)
    assert serve.matrix_bytes(prob, precision) >= (16 if precision == "fp64" else 24) * prob.n ** 2 + own + fields
    assert lib.mgt_propagate_workspace_bytes_for(E.KIND_CODE[kind], L.MGT_C64, T, N, R, ctypes.byref(nb)) == L.MGT_ERR_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N,T", [(1000, 22_500), (500, 301 * 301), (3000, 360)])
def test_estimate_covers_a_request(N, T, precision):
    """A served request's largest allocation, its inputs on the device already."""
    import dataclasses
    import math
    from magreete_gb300 import serve
    from magreete_gb300 import workloads as W
    prob = W.disk_problem(N, 5, 9.0, n_angles=64)
    t = torch.arange(T, dtype=torch.float64) / T * 2 * math.pi
    prob = dataclasses.replace(prob, detectors=2.0 * torch.stack([torch.cos(t), torch.sin(t)], 1))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    (r,) = serve.serve_sequential([prob], precision)
    torch.cuda.synchronize()
    assert torch.isfinite(torch.view_as_real(r.E_det)).all()
    assert torch.cuda.max_memory_allocated() - base <= serve.matrix_bytes(prob, precision)


@pytest.mark.gpu
def test_small_workspace_runs_matrix_free():
    """The plain method in a workspace that holds the matrix-free kernel's partial
    sums only; less than that is refused."""
    import ctypes
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    lib = L.load()
    T, S, R = 400, 700, 64
    gen = torch.Generator().manual_seed(1)
    tg, src = torch.rand(T, 3, dtype=torch.float64, generator=gen).cuda() + 1.5, torch.rand(S, 3, dtype=torch.float64,
                                                                                              generator=gen).cuda()
    Ek = torch.randn(3 * S, R, dtype=torch.complex128, generator=gen).cuda()
    ref = E.propagate("3d_vector", tg, src, 11.0, 1.0, Ek)
    out = torch.zeros(3 * T, R, dtype=torch.complex128, device="cuda")

    def run(nbytes):
        work = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        return lib.mgt_propagate(L.MGT_3D_VECTOR, L.MGT_C128, E._ptr(tg), T, E._ptr(src), S, 11.0, 1.0, 0.0, 0, 0.0,
                                 E._ptr(Ek), R, None, R, E._ptr(out), R, R, E._ptr(work), nbytes, E._stream())

    nb = ctypes.c_size_t()
    L.check(lib.mgt_propagate_workspace_bytes_for(L.MGT_3D_VECTOR, L.MGT_C128, T, S, R, ctypes.byref(nb)))
    partial = 64 * 3 * T * R * 16            # at most 64 source ranges
    assert partial < nb.value
    assert run(partial) == L.MGT_OK
    assert (torch.linalg.norm(out - ref) / torch.linalg.norm(ref)).item() < 1e-13
    assert run(1024) == L.MGT_ERR_WORKSPACE
