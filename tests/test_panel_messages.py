"""The messages of the complex128 panel (csrc/zpanel_msg.cuh), compiled for the
host: no two columns of a factorisation share a tag, nothing that can stand in a
slot before (zeros, an earlier column's words) carries a column's tag, and
numbers and candidates come back bit for bit."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "magreete_gb300", "csrc")

PROGRAM = r"""
#include "zpanel_msg.cuh"
#include <cstdio>
#include <vector>
using namespace mgt::zp;
int main() {
  // every order that the panel takes columns of, up to 2^20: distinct tags, none of them a cleared slot's
  std::vector<char> seen(1 << 21, 0);
  for (int c = 0; c < (1 << 20); ++c) {
    const uint64_t t = column_tag(c) >> kTagShift;
    if (t == 0 || t >= seen.size() || seen[t] || has_tag(column_tag(c), 0)) return std::printf("tag of column %d\n", c), 1;
    seen[t] = 1;
  }
  if (column_tag(kMaxColumns) >> kTagShift != seen.size() - 1) return std::puts("last tag"), 1;
  const uint64_t vals[] = {0, 1, ~0ull, 0x7FF0000000000000ull, 0x8000000000000001ull, 0x3FF0000000000000ull,
                           0x0123456789ABCDEFull, 0xFEDCBA9876543210ull, 0x7FF8000000000000ull};
  const int cols[] = {0, 1, 31, 127, 128, 129, 251, 19455, 65535, kMaxColumns};
  for (int c : cols)
    for (uint64_t x : vals)
      for (uint64_t y : vals) {
        uint64_t w[3], a, b;
        pack_number(column_tag(c), x, y, w);
        for (int t = 0; t < 3; ++t)
          for (int o : cols)
            if (has_tag(column_tag(o), w[t]) != (o == c)) return std::printf("number of column %d\n", c), 1;
        unpack_number(w, &a, &b);
        if (a != x || b != y) return std::puts("number"), 1;
        for (int pos : {0, 1, 127, 65535, kNoPos - 1, kNoPos}) {
          int p;
          pack_key(column_tag(c), x, pos, w);
          for (int t = 0; t < 2; ++t)
            for (int o : cols)
              if (has_tag(column_tag(o), w[t]) != (o == c)) return std::printf("key of column %d\n", c), 1;
          unpack_key(w[0], w[1], &a, &p);
          if (a != x || p != pos) return std::puts("key"), 1;
        }
      }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_messages(tmp_path):
    src = tmp_path / "messages.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "messages"
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4984, 5000])
def test_panels_of_varying_grids(n):
    """Orders at which the last CTA leaves the panel's grid and comes back some
    panels later, with a matrix whose pivot is always the last row: the factors
    have the bits of the shared-memory panel's."""
    import torch
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    lib = L.load()
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = 0.01 * torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=gen)
    i = torch.arange(n, device="cuda")
    A[i, (i + 1) % n] += 10
    outs = []
    try:
        for mode in (0, 1):
            lib.mgt_set_tuning(L.MGT_TUNE_PANEL_REGISTERS, mode)
            outs.append(E.lu_factor(A.clone()))
    finally:
        lib.mgt_set_tuning(L.MGT_TUNE_PANEL_REGISTERS, 1)
    assert int(outs[1].perm[0]) == n - 1 and int(outs[1].perm[1]) == 0
    assert torch.equal(outs[0].perm, outs[1].perm)
    assert torch.equal(outs[0].lu, outs[1].lu)


@pytest.mark.gpu
@pytest.mark.parametrize("n,ctas", [(1100, 8), (2112, 8)])
@pytest.mark.parametrize("scale", [1.0, 1e6, 1e-290])
def test_panels_of_two_kernels(n, ctas, scale):
    """Panels too tall for the CTAs allowed go to the shared-memory kernel, which
    leaves raw rows where the others' messages lie.  The workspace comes
    from a factorisation with the same sequence numbers, and its flags are not
    taken for this one's either: the factors have the bits of the
    shared-memory kernel's for every panel."""
    import ctypes
    import torch
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    lib = L.load()
    gen = torch.Generator(device="cuda").manual_seed(n)
    mats = [scale * torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=gen) for _ in range(2)]
    nb = ctypes.c_size_t()
    L.check(lib.mgt_lu_workspace_bytes(L.MGT_C128, n, ctypes.byref(nb)))
    work = torch.zeros(nb.value, dtype=torch.uint8, device="cuda")

    def factor(A, **options):
        lu, perm = A.clone(), torch.empty(n, dtype=torch.int32, device="cuda")
        opt = L.LuOptions(**options)
        L.check(lib.mgt_lu_factor_ex(L.MGT_C128, E._ptr(lu), n, n, E._ptr(perm), E._ptr(work), nb.value,
                                     ctypes.byref(opt), E._stream()))
        return lu, perm

    epoch = work[40:48].clone()
    factor(mats[0], panel_max_ctas=ctas)
    torch.cuda.synchronize()
    work[40:48] = epoch          # the next call counts as the last one did
    lu, perm = factor(mats[1], panel_max_ctas=ctas)
    try:
        lib.mgt_set_tuning(L.MGT_TUNE_PANEL_REGISTERS, 0)
        ref = E.lu_factor(mats[1].clone())
    finally:
        lib.mgt_set_tuning(L.MGT_TUNE_PANEL_REGISTERS, 1)
    assert torch.equal(perm, ref.perm)
    assert torch.equal(lu, ref.lu)
