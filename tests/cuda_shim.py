"""A library put in front of the CUDA runtime (LD_PRELOAD) in a child process.  It counts device memory, refuses
allocations past a limit as a full device does, counts cooperative launches or refuses them as a device whose SMs are not
all available does, and notes a kernel's shared-memory limit being lowered.  Nothing reaches the GPU that would not otherwise."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <pthread.h>
#include <stddef.h>

static pthread_mutex_t lock = PTHREAD_MUTEX_INITIALIZER;
static struct { void *p; size_t bytes; } block[1 << 16];
static int blocks, mallocs, lowered, refused, refuse_coop, attempts, fail_from = 1 << 30;
static __thread int coop;   // this thread's
static size_t held, cap = (size_t)-1;
static struct { const void *f; int bytes; } limit[4096];
static int limits;

static void *real(const char *name) {
  static void *rt;
  if (!rt) rt = dlopen("libcudart.so.13", RTLD_NOLOAD | RTLD_LAZY);
  return dlsym(rt, name);
}

size_t shim_held(void) { return held; }
int shim_mallocs(void) { return mallocs; }
int shim_lowered(void) { return lowered; }
int shim_coop(void) { return coop; }
int shim_refused(void) { return refused; }
void shim_cap(size_t bytes) { cap = bytes; }
void shim_fail_from(int n) { attempts = 0, fail_from = n; }   // the n-th allocation from now and all after it
void shim_refuse_coop(int on) { refuse_coop = on; }

cudaError_t cudaMalloc(void **p, size_t bytes) {
  cudaError_t (*f)(void **, size_t) = real("cudaMalloc");
  pthread_mutex_lock(&lock);
  cudaError_t e = cudaErrorMemoryAllocation;
  if (held + bytes <= cap && attempts++ < fail_from) e = f(p, bytes);
  if (e == cudaSuccess) {
    int i = 0;
    while (i < blocks && block[i].p) ++i;
    if (i == blocks) ++blocks;
    block[i].p = *p;
    block[i].bytes = bytes;
    held += bytes;
    ++mallocs;
  }
  pthread_mutex_unlock(&lock);
  return e;
}
cudaError_t cudaFree(void *p) {
  cudaError_t (*f)(void *) = real("cudaFree");
  pthread_mutex_lock(&lock);
  for (int i = 0; p && i < blocks; ++i)
    if (block[i].p == p) {
      held -= block[i].bytes;
      block[i].p = 0;
    }
  pthread_mutex_unlock(&lock);
  return f(p);
}
cudaError_t cudaFuncSetAttribute(const void *func, enum cudaFuncAttribute attr, int value) {
  cudaError_t (*f)(const void *, enum cudaFuncAttribute, int) = real("cudaFuncSetAttribute");
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    pthread_mutex_lock(&lock);
    int i = 0;
    while (i < limits && limit[i].f != func) ++i;
    if (i == limits) limit[limits++].f = func;
    else if (value < limit[i].bytes) ++lowered;
    limit[i].bytes = value;
    pthread_mutex_unlock(&lock);
  }
  return f(func, attr, value);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *func, void **args) {
  cudaError_t (*f)(const cudaLaunchConfig_t *, const void *, void **) = real("cudaLaunchKernelExC");
  for (unsigned i = 0; i < cfg->numAttrs; ++i)
    if (cfg->attrs[i].id == cudaLaunchAttributeCooperative && cfg->attrs[i].val.cooperative) {
      ++coop;
      if (refuse_coop) {
        ++refused;
        return cudaErrorCooperativeLaunchTooLarge;
      }
    }
  return f(cfg, func, args);
}
"""

PRELUDE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, {root!r})
import __graft_entry__
pkg = __graft_entry__.load_package()
shim = ctypes.CDLL(None)
shim.shim_held.restype = ctypes.c_size_t
shim.shim_cap.argtypes = [ctypes.c_size_t]
"""


def run(tmp_path, script, timeout=300, **env):
    """Run `script` (after PRELUDE: numpy as np, pkg, shim) behind the shim; fails when it does."""
    lib = str(tmp_path / "shim.so")
    if not os.path.exists(lib):
        src = str(tmp_path / "shim.c")
        with open(src, "w") as f:
            f.write(SOURCE)
        subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", src, "-o", lib, "-ldl", "-lpthread"],
                       check=True)
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT) + script], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=lib, **env), timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
