"""Launch statuses on the host: none is dropped, and a cooperative launch that
does not fit (a context with fewer SMs than its device) falls back to the
launches per half-step.

The step launchers are linked with a stand-in for the one-launch step that fails
with a given status; no GPU is needed, and none may be there: every other
launch then fails with its own status, which tells the two ways apart.
"""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
INCLUDES = [f"-I{ROOT / 'include'}", f"-I{ROOT / 'gmes_gb300' / 'csrc'}"]

PROGRAM = r'''
#include <cstdio>
#include <cstring>
#include "gmes_internal.cuh"

static cudaError_t status = cudaSuccess;
static int calls = 0;
namespace gmes {
bool persist_takes(const Plan&, int) { return true; }
cudaError_t launch_persist(const Plan&, const Meeting&, int, int, cudaStream_t) {
  ++calls;
  return status;
}
}  // namespace gmes

static cudaError_t step(bool incident, cudaError_t st) {
  static gmes::Slot slot;
  gmes_grid_desc g;
  std::memset(&g, 0, sizeof(g));
  g.precision = GMES_FP64;
  gmes::Plan p, inc;
  std::memset((void*)&p.re, 0, sizeof(p.re));
  for (int a = 0; a < 3; ++a) p.re.n[a] = 4;
  for (int c = 0; c < 6; ++c)
    for (int a = 0; a < 3; ++a) p.re.sh[c][a] = 5;
  p.im = p.re;
  p.cplx = p.disp = false;
  p.precision = GMES_FP64;
  p.incident = nullptr;
  inc = p;
  if (incident) {
    inc.meet.at = &slot;
    p.incident = &inc;
  } else {
    p.meet.at = &slot;
  }
  status = st;
  calls = 0;
  return gmes::launch_step(g, p, 2, nullptr);
}

int main() {
  int n = 0;
  if (cudaGetDeviceCount(&n) == cudaSuccess && n > 0) {
    std::printf("gpu\n");
    return 0;
  }
  const cudaError_t none = cudaGetLastError();  // what every launch fails with here
  bool good = none != cudaSuccess;
  const cudaError_t full[] = {cudaErrorCooperativeLaunchTooLarge, cudaErrorLaunchOutOfResources};
  for (cudaError_t e : full) {
    good = good && step(false, e) != e && calls == 1;
    good = good && step(true, e) != e && calls >= 1;
  }
  good = good && step(false, cudaErrorInvalidValue) == cudaErrorInvalidValue && calls == 1;
  good = good && step(true, cudaErrorInvalidValue) == cudaErrorInvalidValue && calls == 1;
  good = good && step(false, cudaSuccess) == cudaSuccess && calls == 1;
  std::printf(good ? "ok\n" : "bad\n");
  return good ? 0 : 1;
}
'''


def test_failed_one_launch_steps(tmp_path):
    from gmes_gb300 import build
    try:
        exe = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    build.build()
    flags = build.ARCH + build.COMMON
    obj = build.BUILD / f"gmes_step-{build._digest(build.CSRC / 'gmes_step.cu', flags)}.o"
    src = tmp_path / "status.cu"
    src.write_text(PROGRAM)
    out = tmp_path / "status"
    subprocess.run([exe, *build.ARCH, "-std=c++17", *INCLUDES, str(src), str(obj), "-o", str(out),
                    "-lcudart"], check=True, capture_output=True)
    run = subprocess.run([str(out)], capture_output=True, text=True)
    if run.stdout == "gpu\n":
        pytest.skip("needs a host without a GPU")
    assert run.stdout == "ok\n"


def test_dropped_status_does_not_build(tmp_path):
    from gmes_gb300 import build
    try:
        exe = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    src = tmp_path / "dropped.cu"
    code = ('#include "gmes_internal.cuh"\ncudaError_t f(const gmes::Plan& p) {\n  %s'
            'gmes::launch_persist(p, p.meet, 1, 0, nullptr);\n  return cudaSuccess;\n}\n')
    for before, builds in (("return ", True), ("", False)):
        src.write_text(code % before)
        r = subprocess.run([exe, *build.ARCH, *build.COMMON, *INCLUDES, "-c", str(src), "-o",
                            str(tmp_path / "dropped.o")], capture_output=True, text=True)
        assert (r.returncode == 0) is builds, r.stderr
