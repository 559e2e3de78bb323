"""A stand-in for the CUDA runtime, preloaded into a child process: it runs nothing and records every
kernel launch and every shared-memory limit that the library sets, by kernel name and device. Host-side
launch rules are checked with it, without a GPU."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <cuda_runtime_api.h>
#include <map>
#include <mutex>
#include <string>
namespace {
std::mutex mu;
std::map<const void*, std::string> names;
std::string text;
thread_local int device = 0;
char symbol[64];
int encode(...) { return 0; }
void note(const char* what, const void* f, long long bytes, int overlap) {
  std::lock_guard<std::mutex> lock(mu);
  text += std::string(what) + " " + (names.count(f) ? names[f] : "?") + " " + std::to_string(device) + " " +
          std::to_string(bytes) + " " + std::to_string(overlap) + "\n";
}
}  // namespace
extern "C" {
const char* recorder_text() { return text.c_str(); }
void recorder_clear() { text.clear(); }
void recorder_device(int d) { device = d; }
void** __cudaRegisterFatBinary(void*) { return (void**)symbol; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  std::lock_guard<std::mutex> lock(mu);
  names[host] = name;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  int overlap = 0;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      overlap = c->attrs[i].val.programmaticStreamSerializationAllowed;
  note("launch", f, (long long)c->dynamicSmemBytes, overlap);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) {
  note("launch", f, (long long)smem, 0);
  return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) {
  note("launch", f, (long long)smem, 0);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) note("limit", f, v, 0);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = (void*)0x40000; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *p = (void*)&encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
"""

# what the child defines for the code under test: L (the library), P (a device address of its own, never
# read), recorded() (the records since the last call) and on_device(d)
PRELUDE = r"""
import ctypes, itertools, json, sys
import numpy as np
from loadpath_b200._lib import lib
L = lib()
_rec = ctypes.CDLL(None)
_rec.recorder_text.restype = ctypes.c_char_p
_next = itertools.count(1)
def P():
    return next(_next) << 24
def recorded():
    lines = [r.split() for r in _rec.recorder_text().decode().splitlines()]
    _rec.recorder_clear()
    return [dict(what=w, kernel=k, device=int(d), bytes=int(b), overlap=int(o)) for w, k, d, b, o in lines]
on_device = _rec.recorder_device
_rec.recorder_clear()
"""


def record(tmp_path, body):
    """Runs body (which leaves its result in `out`) in a child process under the recorder; returns out."""
    from loadpath_b200 import build

    build.build()
    src, so = os.path.join(tmp_path, "recorder.cpp"), os.path.join(tmp_path, "recorder.so")
    with open(src, "w") as f:
        f.write(SHIM)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I", include, src, "-o", so], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", PRELUDE + body + "\nprint('OUT' + json.dumps(out))"], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.split("OUT")[-1])
