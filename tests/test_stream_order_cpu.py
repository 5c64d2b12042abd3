"""What the library leaves queued on the legacy stream while it works on
streams that do not wait for it (a case's own, a caller's non-blocking one).

The library runs here on a stand-in for the CUDA runtime: memory is the
host's, kernels do nothing, and the stand-in keeps the operations that the
legacy stream may not have finished -- memsets, small copies from pageable
memory, whatever is asynchronous -- until something waits for them.  Work
given to another stream while there are any is a hazard: it may run first, or
the late operation may overwrite its results."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

from volcanor_gb300 import build as vbuild

ROOT = Path(__file__).resolve().parents[1]

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>
namespace {
struct Config { dim3 g, b; size_t sm; cudaStream_t st; };
std::vector<std::string> pending;
std::string hazards;
std::vector<Config> configs;
std::map<const void*, std::string> names;
std::map<const char*, size_t> pinned;
int handles = 16;
bool legacy(cudaStream_t s) { return !s || s == cudaStreamLegacy; }
void op(cudaStream_t s, const std::string& what) {
  if (legacy(s)) pending.push_back(what);
  else if (!pending.empty()) hazards += pending.back() + " may run after " + what + "\n";
}
bool is_pinned(const void* p) {
  auto it = pinned.upper_bound((const char*)p);
  return it != pinned.begin() && (const char*)p < (--it)->first + it->second;
}
template <class T> cudaError_t make(T* t) { *t = (T)(size_t)(handles += 16); return cudaSuccess; }
std::string name(const void* f) { return names.count(f) ? names[f] : "a kernel"; }
}
extern "C" {
const char* fake_hazards() { return hazards.c_str(); }
void fake_reset() { hazards.clear(); }
cudaStream_t fake_stream() { cudaStream_t s; make(&s); return s; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); memset(*p, 0, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(n, 1); pinned[(char*)*p] = n; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { pinned.erase((char*)p); free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { op(0, "cudaMemset"); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { op(s, "cudaMemsetAsync"); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* a, size_t n, cudaMemcpyKind k) {
  memcpy(d, a, n);
  // a small copy from pageable memory returns when it is staged; the others wait
  if (k == cudaMemcpyHostToDevice && n <= (64u << 10) && !is_pinned(a)) pending.push_back("cudaMemcpy from pageable memory");
  else pending.clear();
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* a, size_t n, cudaMemcpyKind, cudaStream_t s) {
  op(s, "cudaMemcpyAsync"); memcpy(d, a, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (legacy(s)) pending.clear(); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return make(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return make(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { return make(g); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { op(s, "a graph"); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return make(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { *a = 0; *b = -5; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { memset(p, 0, sizeof *p); p->multiProcessorCount = 152; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static void* q = calloc(32u << 20, 1); *p = q; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { op(c->stream, name(f)); return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t s) { configs.push_back({g, b, sm, s}); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* s) {
  Config c = configs.back(); configs.pop_back();
  *g = c.g; *b = c.b; *sm = c.sm; *(cudaStream_t*)s = c.st; return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t s) { op(s, name((const void*)k)); return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* n, int, uint3*, uint3*, dim3*, dim3*, int*) { names[f] = n; }
}
"""

PRELUDE = """
import ctypes
import numpy as np
from volcanor_gb300 import lib
rt = ctypes.CDLL(None)
rt.fake_stream.restype = ctypes.c_void_p
rt.fake_hazards.restype = ctypes.c_char_p
rng = np.random.default_rng(0)
L = lib.load()
"""

# a program per entry that has work on streams of its own or of the caller
PROGRAMS = {
    # device buffers on a caller's non-blocking stream, the scratch grown by the second call
    "ring sums": """
st = rt.fake_stream()
for n, m in ((100, 50), (300, 5000)):
    a = [rng.normal(size=k) for k in (12 * n, 4 * n, n, 3 * m, 3 * m)]
    p = [x.ctypes.data for x in a]
    lib.biot_savart_rings_device(p[0], p[1], p[2], n, p[3], m, p[4], lib.PREC_FP32_NEAR64, st)
""",
    # the network of a case's surrogate, trained on the case's stream (what the case itself
    # left behind is waited for first)
    "surrogate": """
from volcanor_gb300 import cases as C
c = C.rotor_2blade_hover(nt=40, n_nwake=10, truncate_nt=30)
k = lib.Case(c.config, c.geom, precision=lib.PREC_FP32_NEAR64)
rt.cudaStreamSynchronize(None)
rt.fake_reset()
k.set_surrogate(collect_steps=2, sample_stride=2, train_iters=4, batch=64, hidden=16, layers=3, min_far=4, young_far=2)
k.start()
k.step(40)
assert k.surrogate_stats()["trainings"] > 0
""",
    # a case's tables: created, steady (graph and incremental plan), asked for velocities, resumed
    "case": """
from volcanor_gb300 import cases as C
c = C.rotor_2blade_hover(nt=60, n_nwake=10, truncate_nt=16)
for precision in (lib.PREC_FP64, lib.PREC_FP32, lib.PREC_FP32_NEAR64):
    k = lib.Case(c.config, c.geom, precision=precision)
    k.start()
    k.step(30)
    k.vind_points(rng.normal(size=(5, 3)))
    k.step(2)
    k.checkpoint_save("case.ckpt")
    k.checkpoint_load("case.ckpt")
    k.step(2)
k.checkpoint_load("case.ckpt")
f = lib.Case(c.config, c.geom, precision=lib.PREC_FP64)
f.start()
f.checkpoint_save("case.ckpt")
k.checkpoint_load("case.ckpt")  # without FP32 factors: made from the restored AIC
""",
    "batch": """
from volcanor_gb300 import cases as C
c = C.rotor_2blade_hover(nt=40, n_nwake=10, truncate_nt=16)
b = lib.Batch([(c.config, c.geom, "")] * 3, precision=lib.PREC_FP32_NEAR64)
b.start()
b.step(30)
""",
    "system": """
from volcanor_gb300 import cases as C
sc = C.rotor_pair(nt=20, n_nwake=8, truncate_nt=12)
for precision in (lib.PREC_FP64, lib.PREC_FP32_NEAR64):
    y = lib.System(sc.config, sc.geoms, precision=precision)
    y.start()
    y.step(20)
""",
}


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    vbuild.build()
    d = tmp_path_factory.mktemp("runtime")
    (d / "rt.cpp").write_text(RUNTIME)
    (d / "rt.map").write_text("libcudart.so.13 { global: *; };\n")
    so = d / "libcudart.so.13"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{vbuild._cuda_home() / 'include'}",
                           str(d / "rt.cpp"), "-Wl,-soname,libcudart.so.13", f"-Wl,--version-script={d / 'rt.map'}",
                           "-o", str(so)])
    return so


@pytest.mark.parametrize("program", sorted(PROGRAMS))
def test_nothing_left_on_the_legacy_stream(runtime, program, tmp_path):
    code = PRELUDE + PROGRAMS[program] + "\nprint(rt.fake_hazards().decode())"
    env = {**os.environ, "LD_PRELOAD": str(runtime), "PYTHONPATH": str(ROOT)}
    r = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "", sorted(set(r.stdout.strip().splitlines()))
