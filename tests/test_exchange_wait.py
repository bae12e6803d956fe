"""The waits of the persistent solves run out: partial sums that no block publishes, or a stamped word that no row writes,
end the wait with the error flag set, and the next exchange on the same context works."""
import ctypes
import os
import subprocess

import pytest

import cuda_shim

SOURCE = r"""
#include "ufe_krylov.cuh"

// One block waits for the partial sums of `blocks` blocks (its own are there, the others' as `stamped` says).
__global__ void k_wait(ExSlot *slots, GridSync *gs, int np, int others, int *out) {
  __shared__ double sp[kPersistSlots * kHaloMaxBlocks];
  if (threadIdx.x < np * kReplicas)
    slot_publish(slots + slot_index(threadIdx.x / kReplicas, 0, threadIdx.x % kReplicas), 1.0, 7u);
  if (others && threadIdx.x < np * kReplicas)
    slot_publish(slots + slot_index(threadIdx.x / kReplicas, 1, threadIdx.x % kReplicas), 2.0, 7u);
  bool ok = exchange_wait<false>(np, slots, sp, nullptr, nullptr, 0, nullptr, 7u, gs);
  ok = __syncthreads_and(ok);
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    out[0] = ok;
    out[1] = ok ? (int)(sp[0] + sp[1]) : 0;
  }
}

// One row of two entries, whose second column's word is or is not there.
__global__ void k_row(CsrMat mat, ExSlot *words, GridSync *gs, int both, int *out) {
  if (threadIdx.x == 0) slot_publish(words, 3.0, 9u);
  if (threadIdx.x == 0 && both) slot_publish(words + 1, 4.0, 9u);
  bool ok = true;
  const double y = threadIdx.x == 0 ? csr_row(mat, 0, words, 9u, gs, ok) : 0.0;
  if (threadIdx.x == 0) {
    out[0] = ok;
    out[1] = ok ? (int)y : 0;
  }
}

// what: 0 sums, 1 row; complete: whether everything that is waited for arrives.  out: ok, value, error flag.
extern "C" int run(int what, int complete, int *out) {
  ExSlot *slots;
  GridSync *gs;
  int *res, *idx;
  double *val;
  const int ptr_ind[] = {0, 2, 0, 1};
  const double v[] = {10.0, 100.0};
  if (cudaMalloc(&slots, sizeof(ExSlot) * kExSlots) || cudaMalloc(&gs, sizeof(GridSync)) || cudaMalloc(&res, 64) ||
      cudaMalloc(&idx, sizeof(ptr_ind)) || cudaMalloc(&val, sizeof(v)))
    return -1;
  cudaMemset(slots, 0, sizeof(ExSlot) * kExSlots);
  cudaMemset(gs, 0, sizeof(GridSync));
  cudaMemcpy(idx, ptr_ind, sizeof(ptr_ind), cudaMemcpyHostToDevice);
  cudaMemcpy(val, v, sizeof(v), cudaMemcpyHostToDevice);
  // a grid of two, of which the second block publishes nothing of its own
  if (what == 0) k_wait<<<2, 256>>>(slots, gs, 1, complete, res);
  else k_row<<<1, 32>>>(CsrMat{1, idx, idx + 2, val}, slots, gs, complete, res);
  if (cudaDeviceSynchronize() != cudaSuccess) return -2;
  cudaMemcpy(out, res, 8, cudaMemcpyDeviceToHost);
  GridSync h;
  cudaMemcpy(&h, gs, sizeof(h), cudaMemcpyDeviceToHost);
  out[2] = h.err;
  cudaFree(slots), cudaFree(gs), cudaFree(res), cudaFree(idx), cudaFree(val);
  return 0;
}
"""


@pytest.fixture(scope="module")
def probe(pkg, gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    src, lib = str(d / "wait.cu"), str(d / "wait.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    build = pkg.build.__globals__
    csrc = os.path.join(cuda_shim.ROOT, "ufemism2.0_gb300", "csrc")
    subprocess.run([build["nvcc_path"](), *build["_flags"](False), "-I" + csrc, "-shared", src, "-o", lib], check=True)
    return ctypes.CDLL(lib)


@pytest.mark.gpu
@pytest.mark.parametrize("what,value", [(0, 3), (1, 430)])
def test_waits_run_out_and_the_next_one_works(probe, what, value):
    out = (ctypes.c_int * 3)()
    for complete in (1, 0, 1):
        assert probe.run(what, complete, out) == 0
        assert list(out) == ([1, value, 0] if complete else [0, 0, 1])
