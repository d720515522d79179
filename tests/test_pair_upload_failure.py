"""Double-float pair records when device memory runs out between their two
arrays: the call fails and the next one uploads both again, so that no build
ever reads primitive records that were never there.  Runs on the host: a small
program takes the pair list of the library's own header and brings its own
cudaMalloc, cudaMemcpy and cudaFree, the first of which fails on demand."""
import os
import subprocess

import pytest

from openlowdin_gb300 import build as B

# the fake runtime, in a unit of its own: the CUDA headers define some of these names inline
RUNTIME = r"""
#include <cstdlib>
#include <cstring>
int mallocs = 0, malloc_fails = -1, copies = 0, copy_fails = -1, live = 0;
extern "C" int cudaMalloc(void **p, size_t n) {
  if (++mallocs == malloc_fails) return 2;
  *p = malloc(n);
  ++live;
  return 0;
}
extern "C" int cudaFree(void *p) {
  if (p) --live;
  free(p);
  return 0;
}
extern "C" int cudaMemcpy(void *d, const void *s, size_t n, int) {
  if (++copies == copy_fails) return 1;
  memcpy(d, s, n);
  return 0;
}
"""

SOURCE = r"""
#include "lint_host.cuh"
extern int mallocs, malloc_fails, copies, copy_fails, live;
namespace lgb {
void set_error(const char *, ...) {}
}
int main(int, char **argv) {
  int &fails = argv[1][0] == 'c' ? copy_fails : malloc_fails;
  lgb::PairList L;
  lgb::PairRec r{};
  r.nprim = 1;
  r.Q = 0.5;
  lgb::PrimRec q{};
  q.p = 1.5;
  for (int k = 0; k < 3; ++k) {
    r.prim0 = k;
    L.h.push_back(r);
    L.hp.push_back(q);
  }
  fails = atoi(argv[2]);
  if (L.upload_dd()) return 10;                      // the failure is reported
  fails = -1;
  if (!L.upload_dd()) return 11;                     // and the next call starts again
  if (!L.dd || !L.ddp) return 12;
  if (L.dd[2].prim0 != 2 || L.ddp[2].p.hi != 1.5f) return 13;
  const int n = mallocs;
  if (!L.upload_dd() || mallocs != n) return 14;     // uploaded once
  L.release();
  return live == 0 ? 0 : 15;                         // nothing is left behind
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    src, run, exe = d / "pairs.cu", d / "runtime.cpp", d / "pairs"
    src.write_text(SOURCE)
    run.write_text(RUNTIME)
    cmd = [B.nvcc(), *B._flags(), "-cudart", "shared", "-I", B.SRC, "-o", str(exe), str(src), str(run)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(exe)


@pytest.mark.parametrize("what", ["malloc", "copy"])
@pytest.mark.parametrize("at", [1, 2])
def test_second_upload_after_a_failed_one(program, what, at):
    env = dict(os.environ, LD_LIBRARY_PATH=os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "lib64"))
    assert subprocess.run([program, what[0], str(at)], env=env).returncode == 0
