"""The library's host side on a CUDA runtime that runs nothing: the objects of
some translation units linked against stand-ins for the runtime's functions,
which write down every copy, synchronisation, allocation, attribute and launch in
order.  Device memory is host memory and copies are done, kernels are not run.
For what the launches of a call are and how they are ordered; needs no GPU."""
import ctypes as C
import os
import subprocess

from rc_gb300 import build as B

_SRC = r"""
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <mutex>
#include <string>
#include <vector>

struct dim3_ { unsigned x, y, z; };
static std::mutex mu;
static std::vector<std::string> ops;
static std::map<const void*, std::string> names;
static unsigned coop_limit = 1u << 30;
static uintptr_t next_stream = 0x5000;
static int last_error = 0;
static struct { dim3_ g, b; size_t smem; void* s; } cfg;

static void op(const char* fmt, const std::string& name, unsigned long long a = 0,
               unsigned long long b = 0, unsigned long long c = 0, unsigned long long d = 0) {
  char line[512];
  snprintf(line, sizeof line, fmt, name.c_str(), a, b, c, d);
  std::lock_guard<std::mutex> lk(mu);
  ops.push_back(line);
}
typedef unsigned long long u64;
#define U(x) ((u64)(uintptr_t)(x))

extern "C" {
int fake_ops() { return (int)ops.size(); }
const char* fake_op(int i) { return ops[i].c_str(); }
void fake_clear() { ops.clear(); }
void fake_coop_limit(unsigned n) { coop_limit = n; }
void* fake_args = nullptr;  // of the last cooperative launch: its first argument
size_t fake_args_bytes = 0;

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, void*, void*,
                            void*, void*, int*) { names[fn] = name; }
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t smem, void* s) {
  cfg = {g, b, smem, s};
  return 0;
}
int __cudaPopCallConfiguration(dim3_* g, dim3_* b, size_t* smem, void** s) {
  *g = cfg.g;
  *b = cfg.b;
  *smem = cfg.smem;
  *s = cfg.s;
  return 0;
}
int __cudaGetKernel(void** k, const void* fn) { *k = (void*)fn; return 0; }
int __cudaLaunchKernel(void* k, dim3_ g, dim3_ b, void**, size_t smem, void* s) {
  op("launch %s grid=%llu block=%llu smem=%llu stream=%llx", names[k], u64(g.x) * g.y * g.z, b.x, smem, U(s));
  return 0;
}
int cudaLaunchCooperativeKernel(const void* k, dim3_ g, dim3_ b, void** args, size_t smem, void* s) {
  if (g.x > coop_limit) {
    op("refuse %s grid=%llu", names[k], g.x);
    return last_error = 720;  // cudaErrorCooperativeLaunchTooLarge
  }
  if (fake_args) memcpy(fake_args, args[0], fake_args_bytes);
  op("coop %s grid=%llu block=%llu smem=%llu stream=%llx", names[k], g.x, b.x, smem, U(s));
  return 0;
}
int cudaFuncSetAttribute(const void* k, int, int v) { op("attr %s %llu", names[k], (u64)v); return 0; }
int cudaGetLastError() { const int e = last_error; last_error = 0; return e; }
const char* cudaGetErrorString(int) { return "fake"; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int, int) { *v = 152; return 0; }
int cudaMalloc(void** p, size_t n) { op("malloc%s %llu", "", n); *p = malloc(n); return 0; }
int cudaFree(void* p) { free(p); return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int) {
  op("memcpy%s %llu", "", n);
  memcpy(d, s, n);
  return 0;
}
int cudaMemcpyAsync(void* d, const void* s, size_t n, int, void* st) {
  op("memcpyAsync%s %llu stream=%llx", "", n, U(st));
  memcpy(d, s, n);
  return 0;
}
int cudaMemsetAsync(void* d, int v, size_t n, void* st) {
  op("memset%s %llu stream=%llx", "", n, U(st));
  memset(d, v, n);
  return 0;
}
int cudaStreamCreateWithFlags(void** s, unsigned) { *s = (void*)(next_stream += 16); return 0; }
int cudaStreamSynchronize(void* s) { op("sync%s stream=%llx", "", U(s)); return 0; }
int cudaDeviceSynchronize() { op("sync%s device", ""); return 0; }
"""


class Fake:
    """lib: the linked library; ops(): what happened since the last clear()."""

    def __init__(self, lib):
        self.lib = lib
        lib.fake_op.restype = C.c_char_p

    def clear(self):
        self.lib.fake_clear()

    def ops(self):
        return [self.lib.fake_op(i).decode() for i in range(self.lib.fake_ops())]


def load(out_dir, units) -> Fake:
    """The units (such as ["gb_fft"]) and gb_runtime on the stand-ins."""
    B.build()
    objs = [os.path.join(B.BUILD, u + ".o") for u in [*units, "gb_runtime"]]
    if not all(os.path.exists(o) for o in objs):
        B.build(force=True)
    und = subprocess.run(["nm", "-u", *objs], capture_output=True, text=True, check=True).stdout
    rest = {w for w in und.split() if w.startswith(("cuda", "__cuda", "cufft"))
            and f" {w}(" not in _SRC and f" {w} (" not in _SRC and f"* {w}(" not in _SRC}
    src = _SRC + "".join(f"int {w}() {{ return 0; }}\n" for w in sorted(rest)) + "}\n"
    cpp, so = os.path.join(out_dir, "fake.cpp"), os.path.join(out_dir, "fake.so")
    with open(cpp, "w") as f:
        f.write(src)
    r = subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-w", "-Wl,-Bsymbolic", cpp, *objs, "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return Fake(C.CDLL(so))
