"""A recording of batched steps that an error cuts short leaves the batch as it
was: the host code of lbm_batch.cu against stand-ins for the CUDA calls that it
makes while it records (no GPU)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cuda_runtime.h>
#include <cstdio>
static int launches_left, destroyed;
static cudaError_t fake_launch(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  return launches_left-- > 0 ? cudaSuccess : cudaErrorLaunchFailure;
}
static cudaError_t fake_begin(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
static cudaError_t fake_end(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
static cudaError_t fake_instantiate(cudaGraphExec_t* out, cudaGraph_t, unsigned long long) { *out = nullptr; return cudaSuccess; }
static cudaError_t fake_destroy(cudaGraph_t) { destroyed++; return cudaSuccess; }
#define cudaLaunchKernel fake_launch
#define cudaStreamBeginCapture fake_begin
#define cudaStreamEndCapture fake_end
#define cudaGraphInstantiate fake_instantiate
#define cudaGraphDestroy fake_destroy
#include "lbm_batch.cu"
namespace lbm_internal { void set_last_error(const char*) {} }
int main() {
  for (int rest = 0; rest < 2; rest++)
    for (int left = 0; left <= 6; left++) {
      lbm_batch b;
      b.storage = STORE_F32;
      b.cfg.multi = true;
      b.rest_i = rest;
      b.cur = 1;
      b.steps = 7;
      launches_left = left;
      destroyed = 0;
      const int rc = capture_graph(&b);
      printf("%d %d %d %d %d %llu %llu %d\n", left, rc != 0, b.rest_i == rest, b.cur, b.clock_pending,
             (unsigned long long)b.steps, (unsigned long long)b.launches, destroyed);
    }
}
"""


def test_a_recording_cut_short_leaves_the_rest_planes(tmp_path):
    from lbm_gb300 import build
    src, exe = tmp_path / "harness.cu", tmp_path / "harness"
    src.write_text(HARNESS)
    csrc = os.path.join(ROOT, "lbm_gb300", "csrc")
    # host code only matters: PTX, not machine code, for the kernels
    r = subprocess.run([build.nvcc(), "-gencode", "arch=compute_103a,code=compute_103a", "-G", "-O0", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", csrc, "-o", str(exe), str(src)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail(r.stderr[-3000:])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    rows = [tuple(int(v) for v in line.split()) for line in out.stdout.splitlines()]
    assert len(rows) == 14, out.stderr
    for left, failed, same_rest, cur, pending, steps, launches, destroyed in rows:
        assert failed == (left < 6)  # a run is six launches
        assert same_rest and cur == 1 and pending == 0 and steps == 7 and launches == 0
        assert destroyed == 1
