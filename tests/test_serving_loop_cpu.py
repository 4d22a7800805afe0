"""The serving loop's bookkeeping under every failure it can meet (CPU only).

The loop is compiled here against stand-ins for the world: builds commit in the order they
are queued, a failed one poisons those behind it, as on the device.  Scripts let the k-th
build, the build alone that follows, the set-up after it or the queueing of a step fail, and
one host allocation after the other.  Whatever happens: an edit is reported as applied
exactly if it was committed, in commit order; the committed allocator state is what the world is
left with; nothing stays queued, in flight or running; the entry returns.
"""
import os
import subprocess

from pixels_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pixels_gb300", "csrc")

MAIN = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

static std::atomic<long> left{-1};  // allocations until one fails (-1: none does)
static void* take(size_t n) {
  if (left.load() >= 0 && left.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void* operator new(size_t n) { return take(n); }
void* operator new[](size_t n) { return take(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }

#include "px_serve.cu"

// ---- the world's stand-in
static struct Script {
  int fail_build, fail_alone, fail_resume, fail_enqueue;  // which one fails (-1: none)
} script;

constexpr int MAX = 64;
static struct Device {
  bool poisoned, parity;      // parity: the holes buffer the next committing build must read
  int log[MAX], n_log;        // committed edits, in order
  uint32_t pool_used;
  int builds, alones, resumes, enqueues, in_flight;
} dev;
static const char* wrong = nullptr;
static void expect(bool ok, const char* what) {
  if (!ok && !wrong) wrong = what;
}

struct px_world {
  int queued[MAX], n_queued;
  bool in_flight, failed, apply, parity;
  uint32_t pool_used, committed_pool;
  uint64_t ops_applied;
};
static px_world W0, W1;
static bool twin_alive, ended;

static void commit(px_world* w) {
  expect(w->parity == dev.parity, "a build read the wrong holes buffer");
  for (int i = 0; i < w->n_queued; i++) dev.log[dev.n_log++] = w->queued[i];
  dev.pool_used += w->n_queued;
  dev.parity = !dev.parity;
  w->committed_pool = dev.pool_used;
  w->failed = false;
}

extern "C" {
int px_world_info(px_world*, int dims[3], double* vpm) {
  for (int k = 0; k < 3; k++) dims[k] = 4096;
  *vpm = 1;
  return PX_OK;
}
int px_get_stats(px_world* w, px_stats* out) {
  std::memset(out, 0, sizeof *out);
  out->pool_used = w->pool_used;
  out->pool_capacity = 1u << 30;
  return PX_OK;
}
int px_reserve_pool(px_world*, uint64_t) { return PX_OK; }
int px_submit_ops(px_world* w, const void* ir, size_t) {
  expect(!w->in_flight, "ops submitted to a busy world");
  expect(w->n_queued == 0, "ops queued behind a failed step's");
  const uint32_t* h = (const uint32_t*)ir;
  const IrOp* ops = (const IrOp*)((const char*)ir + 32);
  for (uint32_t i = 0; i < h[2]; i++) w->queued[w->n_queued++] = (int)((ops[i].mn[0] + ops[i].mx[0]) / 2 / 16 + 0.5);
  return PX_OK;
}
int px_build_enqueue(px_world* w, int, void*) {
  if (dev.enqueues++ == script.fail_enqueue) return PX_E_OOM;
  expect(w->apply, "a step was not pipelined");
  const int k = dev.builds++;
  w->in_flight = true;
  dev.in_flight++;
  if (dev.poisoned || k == script.fail_build) dev.poisoned = w->failed = true;
  else commit(w);
  return PX_OK;
}
int px_build_finish(px_world* w) {
  expect(w->in_flight, "an idle world was finished");
  w->in_flight = false;
  dev.in_flight--;
  if (w->failed) return PX_E_QUEUE_OVERFLOW;
  w->n_queued = 0;
  w->pool_used = w->committed_pool;
  return PX_OK;
}
int px_build(px_world* w, int, void*) {
  expect(!w->apply && w == &W0 && !dev.in_flight && !dev.poisoned, "a build alone among others");
  if (dev.alones++ == script.fail_alone) return PX_E_QUEUE_OVERFLOW;
  commit(w);
  w->n_queued = 0;
  w->pool_used = w->committed_pool;
  return PX_OK;
}
}
namespace px {
int reserve_build_scratch(px_world*, uint64_t, uint32_t) { return PX_OK; }
uint64_t build_stage_slots(const px_world*, uint64_t P) { return P; }
px_world* twin_create(px_world*, uint64_t, uint32_t, int* rc) {
  *rc = PX_OK;
  twin_alive = true;
  return &W1;
}
void twin_destroy(px_world*) {
  expect(!dev.in_flight, "the twin was destroyed in flight");
  twin_alive = false;
}
void pipeline_set(px_world* w, cudaStream_t apply, bool holes_in_a, uint32_t used, uint32_t) {
  expect(!w->in_flight, "settings of a busy world");
  w->apply = apply != nullptr;
  w->parity = holes_in_a;
  w->pool_used = used;
}
PipelineState pipeline_begin(px_world* w) {
  PipelineState s;
  std::memset(&s, 0, sizeof s);
  s.pool_used = dev.pool_used;
  s.holes_in_a = dev.parity;
  return s;
}
void pipeline_end(px_world* w, const PipelineState& st, uint64_t ops, cudaStream_t) {
  expect(!dev.in_flight, "the run ended with a build in flight");
  expect(st.pool_used == dev.pool_used && st.holes_in_a == dev.parity, "the world is left with another state than the committed one");
  expect(ops == (uint64_t)dev.n_log, "another count of ops applied");
  expect(w->n_queued == 0, "ops stay queued");
  dev.poisoned = false;
  ended = true;
}
int pipeline_clear(px_world* w, px_world* twin, cudaStream_t) {
  expect(!dev.in_flight, "cleared with a build in flight");
  w->n_queued = twin->n_queued = 0;
  dev.poisoned = false;
  return PX_OK;
}
int pipeline_resume(px_world*, px_world*, uint64_t, uint32_t) {
  return dev.resumes++ == script.fail_resume ? PX_E_OOM : PX_OK;
}
bool build_done(px_world*) { return true; }
void build_times(px_world*, cudaEvent_t, double* a, double* b) { *a = 0; *b = 1; }
}

static int run(Script s, long fail_alloc, int n, uint32_t max_batch) {
  script = s;
  std::memset(&dev, 0, sizeof dev);
  std::memset(&W0, 0, sizeof W0);
  std::memset(&W1, 0, sizeof W1);
  dev.pool_used = 5;
  wrong = nullptr;
  twin_alive = ended = false;
  px_edit edits[MAX];
  double at[MAX];
  px_edit_result res[MAX];
  uint64_t order[MAX];
  std::memset(edits, 0, sizeof edits);
  std::memset(res, 0xff, sizeof res);
  for (int i = 0; i < n; i++) {
    edits[i].a[0] = 16.0 * i;
    edits[i].a[1] = edits[i].a[2] = 64;
    edits[i].r = 1;
    at[i] = 0;
  }
  size_t applied = 0;
  left = fail_alloc;
  const int rc = px_serve_run(&W0, edits, at, (size_t)n, max_batch, 1ull << 40, 1, (void*)0, res, order, &applied);
  const bool alloc_failed = left.exchange(-1) < 0 && fail_alloc >= 0;
  const bool started = ended;
  expect(!twin_alive && !dev.in_flight, "the run left something behind");
  if (rc == PX_OK || started) {
    expect(applied == (size_t)dev.n_log, "applied edits");
    bool done[MAX] = {false};
    for (int i = 0; i < dev.n_log; i++) {
      expect((int)order[i] == dev.log[i] && dev.log[i] == i, "order applied");
      done[dev.log[i]] = true;
    }
    for (int i = 0; i < n; i++) expect((res[i].status == PX_OK) == done[i], "an edit's status");
  } else {
    expect(dev.n_log == 0, "edits applied before the run began");
  }
  expect((rc == PX_OK) == (dev.n_log == n) || n == 0, "the run's status");
  const bool all = s.fail_enqueue < 0 && s.fail_alone < 0 && s.fail_resume < 0 && !alloc_failed;
  if (all) expect(rc == PX_OK, "a run that had to succeed");
  if (wrong) {
    std::printf("%s: build %d alone %d resume %d enqueue %d alloc %ld, %d edits by %u: rc %d, %d committed\n", wrong, s.fail_build,
                s.fail_alone, s.fail_resume, s.fail_enqueue, fail_alloc, n, max_batch, rc, dev.n_log);
    std::exit(1);
  }
  return alloc_failed;
}

int main() {
  int n_runs = 0, n_alloc = 0;
  for (int n : {0, 1, 7, 24})
    for (uint32_t mb : {1u, 4u, 64u})
      for (int fb = -1; fb < 6; fb++)
        for (int fe = -1; fe < 6; fe++)
          for (int fa = -1; fa < 2; fa++)
            for (int fr = -1; fr < 2; fr++, n_runs++) run({fb, fa, fr, fe}, -1, n, mb);
  for (int fb = -1; fb < 4; fb++)
    for (long a = 0; run({fb, -1, -1, -1}, a, 24, 4); a++) n_alloc++;
  std::printf("ok %d %d\n", n_runs, n_alloc);
  return n_alloc < 20;
}
"""

RUNTIME = r"""
#include <cuda_runtime.h>
extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)8; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
void* __cudaRegisterFatBinary(void*) { static void* h; return &h; }  // (no kernels here)
void __cudaRegisterFatBinaryEnd() {}
void __cudaUnregisterFatBinary() {}
void __cudaInitModule() {}
}
"""


def test_every_failure_is_accounted_for(tmp_path):
    main, runtime = tmp_path / "main.cu", tmp_path / "runtime.cpp"
    main.write_text(MAIN)
    runtime.write_text(RUNTIME)
    exe = tmp_path / "serve"
    r = subprocess.run([build._nvcc(), *build.ARCH, "-O1", "-std=c++17", "-cudart", "none", "-I", CSRC, str(main),
                        str(runtime), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), (r.returncode, r.stdout, r.stderr)
