"""The plain method's propagation in workspaces smaller than it asks for: chunks of fewer
detectors with the same result, the matrix-free kernel where nothing else fits, and
the engine's answer to a device that has no room."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

T, S, R = 3000, 700, 20


def _inputs():
    gen = torch.Generator().manual_seed(1)
    tg = torch.rand(T, 3, dtype=torch.float64, generator=gen).cuda() + 1.5
    src = torch.rand(S, 3, dtype=torch.float64, generator=gen).cuda()
    return tg, src, torch.randn(3 * S, R, dtype=torch.complex128, generator=gen).cuda()


def test_smaller_workspaces():
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    lib = L.load()
    tg, src, Ek = _inputs()
    ref = E.propagate("3d_vector", tg, src, 11.0, 1.0, Ek)
    nb = ctypes.c_size_t()
    L.check(lib.mgt_propagate_workspace_bytes_for(L.MGT_3D_VECTOR, L.MGT_C128, T, S, R, ctypes.byref(nb)))
    for share in (0.7, 0.3, 0.05, 0.02):
        out = torch.zeros(3 * T, R, dtype=torch.complex128, device="cuda")
        work = torch.empty(int(nb.value * share), dtype=torch.uint8, device="cuda")
        L.check(lib.mgt_propagate(L.MGT_3D_VECTOR, L.MGT_C128, E._ptr(tg), T, E._ptr(src), S, 11.0, 1.0, 0.0, 0, 0.0,
                                  E._ptr(Ek), R, None, R, E._ptr(out), R, R, E._ptr(work), work.numel(), E._stream()))
        assert (torch.linalg.norm(out - ref) / torch.linalg.norm(ref)).item() < 1e-14


def test_engine_without_room(monkeypatch):
    from magreete_gb300 import engine as E
    tg, src, Ek = _inputs()
    ref = E.propagate("3d_vector", tg, src, 11.0, 1.0, Ek)
    real, asked = E.workspace, []

    def limited(nbytes, device):
        asked.append(nbytes)
        if nbytes > 150 << 20:
            raise torch.cuda.OutOfMemoryError("no room")
        return real(nbytes, device)

    monkeypatch.setattr(E, "workspace", limited)
    out = E.propagate("3d_vector", tg, src, 11.0, 1.0, Ek)
    assert len(asked) > 1
    assert (torch.linalg.norm(out - ref) / torch.linalg.norm(ref)).item() < 1e-14
    with pytest.raises(torch.cuda.OutOfMemoryError):
        monkeypatch.setattr(E, "workspace", lambda nbytes, device: limited(1 << 40, device))
        E.propagate("3d_vector", tg, src, 11.0, 1.0, Ek)
