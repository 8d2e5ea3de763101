"""The dense GEMM's work plan (csrc/gemm_plan.h, host code without CUDA), compiled with the host compiler."""
import ctypes
import os
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ako4x_b200" / "csrc"
SRC = """
#include "gemm_plan.h"
extern "C" unsigned long long workspace(long long m, long long n, long long k, int sms) {
  return ako_gemm::workspace_bytes(m, n, k, sms);
}
extern "C" int choose(long long m, long long n, long long k, int have_ws, unsigned long long bytes, int sms, int resident,
                      int* plan) {
  ako_gemm::Plan pl;
  const bool ok = ako_gemm::choose(m, n, k, have_ws != 0, bytes, sms, [&](int) { return resident; }, pl);
  plan[0] = pl.bn; plan[1] = pl.splits; plan[2] = pl.cg;
  return ok;
}
"""
SHAPES = [(m, n, k) for m in (1, 100, 128, 129, 256, 300, 512, 640, 969, 1024, 1100, 1153, 2048, 4096, 16294)
          for n in (256, 2048, 8192) for k in (64, 192, 1024, 4096)]


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SRC)
    so = d / "plan.so"
    subprocess.run([os.environ.get("CXX") or "g++", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(d / "plan.cpp"), "-o", str(so)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    f, lib.workspace.restype = lib.choose, ctypes.c_ulonglong
    f.argtypes = [ctypes.c_longlong] * 3 + [ctypes.c_int, ctypes.c_ulonglong, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]

    def call(m, n, k, bytes_, resident):
        plan = (ctypes.c_int * 3)()
        ok = f(m, n, k, bytes_ is not None, bytes_ or 0, 148, resident, plan)
        return tuple(plan) if ok else None
    call.workspace = lambda m, n, k: lib.workspace(*[ctypes.c_longlong(x) for x in (m, n, k)], 148)
    return call


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_without_resident_pairs_a_call_runs_on_single_ctas(choose, m, n, k):
    """Where no pair of CTAs can be resident the same calls are accepted, with the same workspaces."""
    for workspace in (False, True):
        need = 0
        if workspace:
            bn, splits, cg = choose(m, n, k, 1 << 60, 148)
            need = choose.workspace(m, n, k)
            assert need >= (splits * m * n * 4 if splits > 1 else 0)
            if need:
                assert choose(m, n, k, need - 1, 148) is None
        plan = choose(m, n, k, need if workspace else None, 0)
        assert plan is not None and plan[2] == 1
        bn, splits, cg = plan
        assert n % bn == 0 and (k // 64) % splits == 0
        assert splits == 1 or splits * m * n * 4 <= need


# one shape for every form of the kernel that a plan can name: tile width, pieces of K, CTAs per tile
FORMS = {(128, 1, 1): (1100, 2048, 512), (128, 2, 1): (1100, 1024, 4096), (128, 4, 1): (200, 2048, 2048), (128, 8, 1): (300, 512, 4096),
         (128, 1, 2): (640, 2048, 4096), (128, 2, 2): (512, 2048, 4096), (128, 4, 2): (256, 2048, 4096), (128, 8, 2): (260, 512, 8192),
         (256, 1, 1): (1000, 4096, 256), (256, 1, 2): (1153, 2048, 4096), (256, 2, 2): (1481, 1024, 8192), (256, 4, 2): (1444, 512, 8192)}


@pytest.mark.parametrize("form", FORMS)
def test_form_of_a_shape(choose, form):
    assert choose(*FORMS[form], 1 << 60, 148) == form


def test_a_missed_wave_and_short_k_loops(choose):
    """144 single CTAs in one wave instead of 80 pairs for 74 places; no pairs and no pieces for short K loops."""
    assert choose(1100, 4096, 4096, 1 << 60, 148)[2] == 1
    assert choose(130, 32768, 64, 1 << 60, 148)[2] == 1
    assert choose(300, 2048, 512, 1 << 60, 148) == (128, 1, 1)
    assert choose(300, 2048, 4096, 1 << 60, 148)[2] == 2
