"""The host code of lbm_batch.cu against stand-ins for the CUDA calls that it
makes (no GPU): a recording that an error cuts short leaves the batch as it was;
the steps per launch follow the rounding mode and what was chosen for it; the
autotuner's choice between one and three steps does not depend on its trials' length."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
// launches of the one-step and of the three-step kernel (the first takes 14
// arguments' worth of block, the second one warp) are told apart by block size
static int launches_left = 1 << 30, destroyed, singles, triples, recorded[2], recording, captures;
template <class F> static cudaError_t fake_launch(F, dim3, dim3 block, void**, size_t, cudaStream_t) {
  if (launches_left-- <= 0) return cudaErrorLaunchFailure;
  (recording ? recorded[block.x == 32] : block.x == 32 ? triples : singles)++;
  return cudaSuccess;
}
struct Run { int singles, triples; };
static cudaError_t fake_begin(cudaStream_t, cudaStreamCaptureMode) {
  recording = 1;
  recorded[0] = recorded[1] = 0;
  return cudaSuccess;
}
static cudaError_t fake_end(cudaStream_t, cudaGraph_t* g) { recording = 0; *g = nullptr; return cudaSuccess; }
static cudaError_t fake_instantiate(cudaGraphExec_t* out, cudaGraph_t, unsigned long long) {
  *out = (cudaGraphExec_t) new Run{recorded[0], recorded[1]};
  captures++;
  return cudaSuccess;
}
static cudaError_t fake_replay(cudaGraphExec_t g, cudaStream_t) {
  singles += ((Run*)g)->singles;
  triples += ((Run*)g)->triples;
  return cudaSuccess;
}
static cudaError_t fake_exec_destroy(cudaGraphExec_t g) { delete (Run*)g; return cudaSuccess; }
static cudaError_t fake_destroy(cudaGraph_t) { destroyed++; return cudaSuccess; }
template <class T> static cudaError_t fake_malloc(T** p, size_t n) { *p = (T*)calloc(1, n + 1); return cudaSuccess; }
static cudaError_t fake_free(void* p) { free(p); return cudaSuccess; }
static cudaError_t fake_attr(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
template <class F> static cudaError_t fake_func_attr(F, cudaFuncAttribute, int) { return cudaSuccess; }
template <class F> static cudaError_t fake_occupancy(int* v, F, int, size_t) { *v = 2; return cudaSuccess; }
static cudaError_t fake_capturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
template <class... A> static cudaError_t fine(A...) { return cudaSuccess; }
static cudaError_t fake_copy(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t = nullptr) { memcpy(d, s, n); return cudaSuccess; }
// a clock that moves by each launch's cost and by each recording's
static float single_ms = 1.0f, triple_ms = 1.5f, stamps[2];
static int stamped;
static cudaError_t fake_event(cudaEvent_t*) { stamped = 0; return cudaSuccess; }
static cudaError_t fake_record(cudaEvent_t, cudaStream_t) {
  stamps[stamped++ & 1] = singles * single_ms + triples * triple_ms + captures * 30.0f;
  return cudaSuccess;
}
static cudaError_t fake_elapsed(float* ms, cudaEvent_t, cudaEvent_t) { *ms = stamps[1] - stamps[0]; return cudaSuccess; }
#define cudaLaunchKernel fake_launch
#define cudaStreamBeginCapture fake_begin
#define cudaStreamEndCapture fake_end
#define cudaGraphInstantiate fake_instantiate
#define cudaGraphLaunch fake_replay
#define cudaGraphExecDestroy fake_exec_destroy
#define cudaGraphDestroy fake_destroy
#define cudaMalloc fake_malloc
#define cudaFree fake_free
#define cudaDeviceGetAttribute fake_attr
#define cudaFuncSetAttribute fake_func_attr
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor fake_occupancy
#define cudaStreamIsCapturing fake_capturing
#define cudaMemcpyAsync fake_copy
#define cudaMemcpy fake_copy
#define cudaMemsetAsync fine
#define cudaStreamSynchronize fine
#define cudaGetLastError fine
#define cudaEventCreate fake_event
#define cudaEventRecord fake_record
#define cudaEventSynchronize fine
#define cudaEventElapsedTime fake_elapsed
#define cudaEventDestroy fine
#include "lbm_batch.cu"
namespace lbm_internal { void set_last_error(const char*) {} }

static void set_up(lbm_batch& b, int storage, uint64_t cells) {
  b.storage = storage;
  b.cells = cells;
  b.materialised = false;
  fake_malloc(&b.d_flag, 4);
  ensure_counters(&b);
  b.cfg.multi = cells >= 400000;  // as lbm_batch_create leaves it
}
// steps per launch of a call, as the launches of ten steps say
static int per_launch(lbm_batch& b) {
  singles = triples = 0;
  lbm_batch_step(&b, 10);
  return triples == 3 && singles == 1 ? 3 : triples == 0 && singles == 10 ? 1 : -1;
}
int main(int argc, char** argv) {
  if (!strcmp(argv[1], "cut"))
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
  if (!strcmp(argv[1], "rounding")) {  // cells, then a letter per call
    lbm_batch b;
    set_up(b, STORE_F16, strtoull(argv[2], nullptr, 10));
    printf("%d", per_launch(b));
    for (int i = 3; i < argc; i++) {
      const char c = argv[i][0];
      if (c == 's') lbm_batch_set_rounding(&b, LBM_ROUND_STOCHASTIC, (uint32_t)i);
      if (c == 'n') lbm_batch_set_rounding(&b, LBM_ROUND_NEAREST, 0);
      if (c == 'h') lbm_batch_set_schedule(&b, 1, 0, nullptr);
      if (c == 'f') triple_ms = 1.5f, lbm_batch_autotune(&b, 40, nullptr, 0);  // three steps at once are faster
      if (c == 'w') triple_ms = 4.0f, lbm_batch_autotune(&b, 40, nullptr, 0);  // slower
      printf(" %d", per_launch(b));
    }
    printf("\n");
  }
  if (!strcmp(argv[1], "tune"))  // steps per trial: the form chosen where it is the faster one by a tenth
    for (int form = 1; form <= 3; form += 2) {
      lbm_batch b;
      set_up(b, STORE_F32, 500000);
      triple_ms = form == 3 ? 2.7f : 3.3f;
      char report[16384];
      lbm_batch_autotune(&b, (uint32_t)atoi(argv[2]), report, sizeof report);
      const char* chosen = strstr(report, "chosen");
      float ms = 0.0f;
      sscanf(strstr(chosen, "ms_per_step"), "ms_per_step\": %f", &ms);
      printf("%d %d\n", per_launch(b), (int)(ms * 1000 + 0.5f));
    }
  fflush(stdout);
  _Exit(0);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    from lbm_gb300 import build
    tmp = tmp_path_factory.mktemp("batch_host")
    src, exe = tmp / "harness.cu", tmp / "harness"
    src.write_text(HARNESS)
    csrc = os.path.join(ROOT, "lbm_gb300", "csrc")
    # host code only matters: PTX, not machine code, for the kernels
    r = subprocess.run([build.nvcc(), "-gencode", "arch=compute_103a,code=compute_103a", "-G", "-O0", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", csrc, "-o", str(exe), str(src)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail(r.stderr[-3000:])

    def run(*args):
        out = subprocess.run([str(exe)] + [str(a) for a in args], capture_output=True, text=True, timeout=60)
        return [[int(v) for v in line.split()] for line in out.stdout.splitlines()]

    return run


def test_a_recording_cut_short_leaves_the_rest_planes(harness):
    rows = harness("cut")
    assert len(rows) == 14
    for left, failed, same_rest, cur, pending, steps, launches, destroyed in rows:
        assert failed == (left < 6)  # a run is six launches
        assert same_rest and cur == 1 and pending == 0 and steps == 7 and launches == 0
        assert destroyed == 1


@pytest.mark.parametrize("cells,calls,want", [
    (450000, "s n", [3, 1, 3]),        # the default of each mode
    (1600000, "s n", [3, 3, 3]),
    (399999, "s n", [1, 1, 1]),
    (450000, "s f s n s", [3, 1, 3, 3, 3, 3]),   # found with stochastic rounding: stays there, also for another seed
    (450000, "w n s n", [3, 1, 1, 1, 1]),        # found without: stays there
    (1600000, "w s n", [3, 1, 3, 1]),            # and leaves the other mode its default
    (2000000, "h s n", [3, 1, 1, 1]),            # fixed by hand: both modes
])
def test_steps_per_launch_follow_the_rounding_mode(harness, cells, calls, want):
    assert harness("rounding", cells, *calls.split()) == [want]


@pytest.mark.parametrize("steps", [1, 2, 3, 8, 18, 19, 20, 21, 40, 100])
def test_the_autotuner_finds_the_faster_form_at_any_trial_length(harness, steps):
    """A three-step launch that costs a tenth less (more) than three single ones:
    short trials, in which few or no steps share a launch, and trials during which
    a run would have to be recorded choose it (not) like long ones."""
    assert harness("tune", steps) == [[1, 1000], [3, 900]]
