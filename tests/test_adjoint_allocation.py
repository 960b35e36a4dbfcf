"""A forward run of the adjoint that fails for want of device memory leaves no run
to differentiate, whichever buffer was refused; and the engine works again after.
Runs on the host: the engine's object file is linked with a runtime whose memory
is the host's, whose kernels do nothing and whose n-th allocation fails."""
import os
import subprocess
from pathlib import Path

import pytest

from bromoc_gb300 import build

SRC = Path(__file__).resolve().parents[1] / "bromoc_gb300" / "csrc"

RUNTIME = r"""
#include <cstdlib>
#include <cstring>
#include <map>
int fail_at = -1;  // allocations to come before the refused one
std::map<void *, size_t> held;
extern "C" {
int cudaMalloc(void **p, size_t n) {
  if (fail_at >= 0 && fail_at-- == 0) return 2;
  *p = std::calloc(n, 1);
  held[*p] = n;
  return 0;
}
int cudaFree(void *p) {
  if (p && !held.erase(p)) std::abort();
  std::free(p);
  return 0;
}
int cudaMemcpy(void *d, const void *s, size_t n, int) { std::memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *) { std::memcpy(d, s, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *) { std::memset(d, v, n); return 0; }
int cudaStreamSynchronize(void *) { return 0; }
int cudaGetLastError() { return 0; }
const char *cudaGetErrorString(int) { return "refused"; }
int cudaLaunchKernelExC(const void *, const void *, void **) { return 0; }
int __cudaLaunchKernel() { return 0; }
int __cudaGetKernel(void **k, const void *) { *k = nullptr; return 0; }
unsigned __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction() {}
char __cudaInitModule(void **) { return 0; }
}
"""

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <vector>
#include "../../include/bromoc_gpu.h"
#include "kparams.cuh"
using namespace bgpu;
extern int fail_at;

// a prototype of one ion type with a tabulated law
static int nwtype[2] = {0, 1}, pidx[1] = {0};
static PairParamF law;
static KP kp;
bool bromoc_ctx_pair_view(const bromoc_ctx *, const KP **k, cudaStream_t *s, int *precision) {
  *k = &kp;
  *s = nullptr;
  *precision = BROMOC_FP64;
  return true;
}
int bromoc_ctx_prepare_f32(bromoc_ctx *, const KP **, cudaStream_t *) { return BROMOC_E_STATE; }
int bromoc_ctx_fail(bromoc_ctx *, int code, const char *) { return code; }
void bromoc_ctx_attach(bromoc_ctx *, int *) {}
void bromoc_ctx_detach(bromoc_ctx *, int *) {}

#define WANT(x) do { if (!(x)) { std::fprintf(stderr, "line %d: %s (case %d)\n", __LINE__, #x, at); return 1; } } while (0)

int main() {
  law.flags = kEfp;
  kp.nwtype = nwtype;
  kp.pidx = pidx;
  kp.ppf = &law;
  kp.ntype = kp.nttyp = kp.nion_t = kp.ntc = kp.cnt = 1;
  kp.shape = BROMOC_BOX;
  double x[2] = {0.0, 3.0}, o[2] = {0.0, 0.0};
  int32_t t[2] = {1, 1};
  std::vector<double> hist(64), dl(64), gep(3), gsc(3);
  // the second run is kept whole in more memory, or falls back to checkpoints, or has
  // them for its limit; each of its allocations is refused in turn
  for (int kind = 0; kind < 3; ++kind)
    for (int at = 0;; ++at) {
      bromoc_adj *a = nullptr;
      WANT(bromoc_adj_create((bromoc_ctx *)&kp, 2, BROMOC_FP64, &a) == BROMOC_OK);
      WANT(bromoc_adj_set_particles(a, 2, x, o, o, t) == BROMOC_OK);
      auto forward = [&](int steps, int nbins) {
        return bromoc_adj_forward(a, steps, 3, 1, 0, nbins, 0.0, 0.1, 0.1, hist.data());
      };
      auto backward = [&] { return bromoc_adj_backward(a, dl.data(), gep.data(), gsc.data()); };
      WANT(forward(4, 8) == BROMOC_OK);
      WANT(backward() == BROMOC_OK);
      if (kind == 2) WANT(bromoc_adj_set_keep(a, 33 * 2 * 4) == BROMOC_OK);
      fail_at = at;
      const int rc = forward(kind == 1 ? 4 : 40, kind == 1 ? 16 : 12);
      const bool refused = fail_at < 0;
      fail_at = -1;
      if (!refused) {  // every allocation has had its turn
        WANT(rc == BROMOC_OK && at >= 2);
        bromoc_adj_destroy(a);
        break;
      }
      if (rc == BROMOC_OK)  // no room to keep the run: it has checkpoints
        WANT(kind == 0 && at == 0 && backward() == BROMOC_OK);
      else
        WANT(rc == BROMOC_E_NOMEM && backward() == BROMOC_E_STATE);
      WANT(forward(4, 8) == BROMOC_OK && backward() == BROMOC_OK);
      WANT(forward(40, 12) == BROMOC_OK && backward() == BROMOC_OK);
      WANT(bromoc_adj_destroy(a) == BROMOC_OK);
    }
  return 0;
}
"""


def test_a_refused_allocation_leaves_no_run(tmp_path):
    try:
        nv = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    build.build()
    (tmp_path / "runtime.cpp").write_text(RUNTIME)
    (tmp_path / "program.cu").write_text(PROGRAM)
    exe = tmp_path / "program"
    subprocess.run([nv, *build.ARCH, "-std=c++17", "-cudart", "none", "-Xcompiler",
                    "-fsanitize=address", f"-I{SRC}", "-o", str(exe),
                    str(tmp_path / "program.cu"), str(tmp_path / "runtime.cpp"),
                    str(build.OBJ / "adjoint.cu.o")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True,
                       env={**os.environ, "ASAN_OPTIONS": "detect_leaks=0"})
    assert r.returncode == 0, r.stderr[-3000:]
