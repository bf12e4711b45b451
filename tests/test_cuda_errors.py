"""Failed CUDA calls while a context and its tables are set up, made on the host: a child process runs the library
over a fake of the CUDA runtime calls it makes (memory is host memory, kernels are counted and not run), which fails
the chosen call and keeps the error for cudaGetLastError as the runtime does.  A call that could not set up what it
needs has to say so before it launches anything, and the next call has to start over."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

FAKE = r"""
#include <cuda_runtime_api.h>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
static std::map<std::string, long> calls, fail_at;
static cudaError_t last = cudaSuccess;
static long live = 0, blocks = 0;
static cudaError_t call(const char *name) {
  const long n = ++calls[name];
  const auto f = fail_at.find(name);
  if (f == fail_at.end() || f->second != n) return cudaSuccess;
  return last = std::strcmp(name, "cudaMalloc") ? cudaErrorUnknown : cudaErrorMemoryAllocation;
}
extern "C" {
void fake_reset() { calls.clear(), fail_at.clear(); }
void fake_fail(const char *name, long nth) { fail_at[name] = nth; }
long fake_calls(const char *name) { return calls[name]; }
long fake_live() { return live; }
long fake_blocks() { return blocks; }  // of the latest launch
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  const cudaError_t e = call("cudaMalloc");
  if (e) return e;
  *p = std::calloc(n ? n : 1, 1), ++live;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (p) std::free(p), --live;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  const cudaError_t e = call("cudaMemcpy");
  if (!e) std::memcpy(d, s, n);
  return e;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static char scratch[16];
  *p = scratch;
  return call("cudaGetSymbolAddress");
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)16; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *, dim3 g, dim3, void **, size_t, cudaStream_t) {
  blocks = (long)g.x * g.y * g.z;
  return call("cudaLaunchKernel");
}
}
"""

CHILD = r"""
import ctypes as C, json, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from icoatmosbenchmark_v1_b200 import api
from icoatmosbenchmark_v1_b200.grid import Grid
fake = C.CDLL(None)
for f in (fake.fake_calls, fake.fake_live, fake.fake_blocks):
    f.restype = C.c_long
calls = lambda name: fake.fake_calls(name.encode())
fail = lambda name, nth: fake.fake_fail(name.encode(), C.c_long(nth))
assert "torch" not in sys.modules
"""


@pytest.fixture(scope="module")
def child(built, tmp_path_factory):
    from icoatmosbenchmark_v1_b200 import build
    d = tmp_path_factory.mktemp("fake_cuda")
    (d / "fake.cpp").write_text(FAKE)
    inc = Path(build.nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-I{inc}", str(d / "fake.cpp"), "-o", str(d / "fake.so")],
                   check=True)

    def run(body, *args):
        r = subprocess.run([sys.executable, "-c", CHILD + body, str(ROOT), *map(str, args)], capture_output=True, text=True,
                           env=dict(os.environ, LD_PRELOAD=str(d / "fake.so")), timeout=120)
        assert r.returncode == 0, r.stderr
        return json.loads(r.stdout)

    return run


INIT = r"""
kind, out = sys.argv[2], []

def init():
    try:
        api.IcoAdv(2, 0, 4).close()
        return True
    except api.IcoAdvError:
        return False

n = 1
while True:
    fake.fake_reset()
    fail(kind, n)
    fail("cudaGetSymbolAddress", 1)  # handled inside ica_init, with the error it leaves behind
    first = init()
    if calls(kind) < n:  # past the last such call: nothing failed
        break
    fake.fake_reset()
    out.append([first, fake.fake_live(), init()])
    n += 1
print(json.dumps(out))
"""


@pytest.mark.parametrize("kind", ["cudaMalloc", "cudaMemcpy"])
def test_init_reports_a_failed_call_and_can_be_repeated(child, kind):
    out = child(INIT, kind)
    assert len(out) >= 6  # the halo map, two plans of two lists, the singular-point flags
    for n, (first, live, again) in enumerate(out, 1):
        assert not first and live == 0 and again, (n, first, live, again)


STEP = r"""
kind, out = sys.argv[2], []
n, shapes = 1, lambda ctx: ((ctx.sizes.lall, ctx.sizes.kall, ctx.sizes.gall), (2, ctx.sizes.kall, 6))
while True:
    ctx = api.IcoAdv(2, 0, 4)
    ctx.set_grid(Grid(2, 0, 6))
    reg, pol = shapes(ctx)
    arrs = [np.ones(reg), np.ones(pol), np.ones((2,) + reg), np.ones((2,) + pol)]
    arrs += [np.ones(s) for _ in range(4) for s in (reg, pol)]

    def step():
        try:
            ctx.advect_step(1.0, *arrs)
            return True
        except api.IcoAdvError:
            return False

    fake.fake_reset()
    fail(kind, n)
    first = step()
    if calls(kind) < n:
        break
    launched = calls("cudaLaunchKernel")
    fake.fake_reset()
    again = step()
    copies = calls("cudaMemcpy")
    ctx.close()
    out.append([first, launched, again, copies, fake.fake_live()])
    n += 1
print(json.dumps(out))
"""


@pytest.mark.parametrize("kind", ["cudaMalloc", "cudaMemcpy"])
def test_plain_step_whose_tables_failed_can_be_repeated(child, kind):
    """The plain step builds the boundary tables on its first call.  Whatever fails there, nothing is launched on
    the state, and the next call builds what is missing and succeeds; closing the context frees all of it."""
    out = child(STEP, kind)
    assert len(out) >= 6
    for n, (first, launched, again, copies, live) in enumerate(out, 1):
        assert not first and launched == 0 and again and live == 0, (n, first, launched, again, live)
        if kind == "cudaMemcpy":
            assert copies == 6, (n, copies)
