"""Failed host allocations while an op list is queued (CPU only).

Every host exception becomes PX_E_OOM at the C entry, also one thrown on a thread of the
conversion pool, and the queue stays as it was: the host runtime is compiled here with an
operator new that fails on demand, at one allocation after the other, and a list is queued on
an empty world and behind another list.  After each failure the list is queued again and has
to equal the one of a world that never failed.
"""
import os
import subprocess

import numpy as np

from pixels_gb300 import build, config
from pixels_gb300.ir import Program
from pixels_gb300.paints import tufted
from pixels_gb300.shapes import box, lathe, rotateY, sphere, subtract

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

#include "px_api.cu"

static px_world* world() {  // what px_submit_ops reads of a world; no device
  px_world* w = new px_world();
  w->dx = 640; w->dy = 176; w->dz = 480;
  w->BX = 80; w->BY = 22; w->BZ = 60; w->TX = 20; w->TY = 6; w->TZ = 15;
  w->ncells = 80 * 22 * 60; w->ntiles = 20 * 6 * 15;
  w->vpm = 40; w->vs = 1 / 40.0;
  return w;
}

template <class V>
static bool same(const V& a, const V& b) {
  return a.size() == b.size() && (a.empty() || !std::memcmp(a.data(), b.data(), a.size() * sizeof(a[0])));
}
static bool same_queue(const px_world* a, const px_world* b) {
  if (a->ops.size() != b->ops.size() || a->lite.size() != b->ops.size()) return false;
  for (size_t i = 0; i < a->ops.size(); i++) {
    const OpDev &x = a->ops[i], &y = b->ops[i];
    if (x.pair_base != y.pair_base || x.code_off != y.code_off || x.base_off != y.base_off || x.vq_class != y.vq_class ||
        x.paint32_off != y.paint32_off || std::memcmp(x.lw, y.lw, sizeof x.lw) || std::memcmp(x.lip, y.lip, sizeof x.lip) ||
        a->lite[i].n_pairs != b->lite[i].n_pairs)
      return false;
  }
  return same(a->boxes, b->boxes) && same(a->code, b->code) && same(a->code32, b->code32) && same(a->p32, b->p32) &&
         same(a->bases, b->bases) && same(a->params, b->params) && same(a->q.painted64, b->q.painted64) &&
         same(a->q.painted32, b->q.painted32) && a->q.pairs == b->q.pairs && a->q.tile_pairs == b->q.tile_pairs;
}

static int run(const std::vector<char>& ir, const std::vector<char>* before) {
  px_world* good = world();
  if (before && px_submit_ops(good, before->data(), before->size()) != PX_OK) return 1;
  px_world* none = world();
  if (before && px_submit_ops(none, before->data(), before->size()) != PX_OK) return 1;
  if (px_submit_ops(good, ir.data(), ir.size()) != PX_OK) return 1;
  int failures = 0;
  for (long n = 0;; n += 1 + n / 40) {
    px_world* w = world();
    if (before && px_submit_ops(w, before->data(), before->size()) != PX_OK) return 1;
    left = n;
    const int rc = px_submit_ops(w, ir.data(), ir.size());
    const bool failed = left.exchange(-1) < 0;
    if (!failed && rc != PX_OK) { std::printf("%ld: refused with %d\n", n, rc); return 1; }
    if (rc != PX_OK) {
      if (rc != PX_E_OOM || !same_queue(w, none)) { std::printf("%ld: status %d, queue of %zu ops\n", n, rc, w->ops.size()); return 1; }
      failures++;
      if (px_submit_ops(w, ir.data(), ir.size()) != PX_OK) return 1;
    }
    if (!same_queue(w, good)) { std::printf("%ld: another queue\n", n); return 1; }
    delete w;
    if (!failed) break;
  }
  delete good;
  delete none;
  std::printf("%d failures\n", failures);
  return failures == 0;
}

static std::vector<char> file(const char* path) {
  std::vector<char> v;
  FILE* f = std::fopen(path, "rb");
  for (int c; (c = std::fgetc(f)) != EOF;) v.push_back((char)c);
  std::fclose(f);
  return v;
}

int main(int, char** argv) {
  const std::vector<char> many = file(argv[1]), few = file(argv[2]);
  return run(many, nullptr) || run(many, &few) || run(few, nullptr) || run(few, &many);
}
"""


def op_list(n, seed):
    rng = np.random.default_rng(seed)
    prog = Program()
    with config.using(40.0):
        for k in range(n):
            c = tuple(float(v) for v in rng.uniform(0.5, 4.0, 3))
            r = float(rng.uniform(0.05, 0.4))
            s = (sphere(c, r), rotateY(box(c, (r, r, 2 * r)), 0.3, c), subtract(sphere(c, r), box(c, (r, r / 2, r))),
                 lathe(c, [r, -r, r / 2, 0.0, r, r], 0))[k % 4]
            prog.add_op(k % 3, s, tufted(0.1, 0.1, 5) if k % 5 == 2 else k % 50 + 1)
    return prog.to_bytes()


def test_every_failed_allocation_is_reported_and_undone(built_lib, tmp_path):
    main = tmp_path / "main.cu"
    main.write_text(MAIN)
    exe = tmp_path / "submit"
    objs = [os.path.join(build.BUILD_DIR, "kernels.o")]
    r = subprocess.run([build._nvcc(), *build.ARCH, "-O1", "-std=c++17", "-fmad=false", "-Xcompiler", "-ffp-contract=off",
                        "-I", CSRC, str(main), *objs, "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    paths = []
    for n in (700, 20):  # converted by the pool, and by the calling thread
        paths.append(tmp_path / f"{n}.ir")
        paths[-1].write_bytes(op_list(n, n))
    r = subprocess.run([str(exe), *map(str, paths)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
