"""What the last warp of a chain does when a warp in front of it gave up on a wait: the sums lack that warp's part and must not be
stored. csrc/pipeline.cuh in a small program of its own, because no wait of a kernel runs out when nothing is wrong: one warp
waits a few polls for a phase that nobody completes, in the first or the second round of a chain over eight warps."""
import os
import shutil
import subprocess

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nntrainer_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include "common.cuh"
#include "pipeline.cuh"
using namespace nntr;
constexpr int WARPS = 8, ROUNDS = 2, TILES = 2;
__global__ void kernel(int who, int round, int *status, int *out) {
  __shared__ alignas(8) unsigned long long done, never;
  __shared__ int flag_word, chain[WARPS][TILES][32];
  volatile int *flag = &flag_word;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    flag_word = 0;
    mbar_init(smem_u32(&done), 1);
    mbar_init(smem_u32(&never), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_arrive(smem_u32(&done));
  }
  __syncthreads();
  bool ok = true;
  for (int rd = 0; rd < ROUNDS; ++rd) {
    ok = mbar_wait_bounded(smem_u32(warp == who && rd == round ? &never : &done), 0, flag, status, 64, 2048) && ok;
    __syncwarp();
    for (int i = 0; i < TILES; ++i) {
      int sum = 0;
      if (rd || warp) {
        pair_sync(warp * TILES + i);
        sum = chain[warp][i][lane];
      }
      sum += 1;
      const int to = warp + 1 < WARPS ? warp + 1 : 0;
      if (rd + 1 < ROUNDS || warp + 1 < WARPS) {
        chain[to][i][lane] = sum;
        pair_arrive(to * TILES + i);
      } else if (nobody_gave_up(ok, flag)) {
        out[i * 32 + lane] = sum;
      }
    }
  }
}
int main() {
  int *mem;
  if (cudaMallocManaged(&mem, (1 + TILES * 32) * sizeof(int)) != cudaSuccess)
    return 2;
  for (int k = -1; k < WARPS * ROUNDS; ++k) {
    for (int i = 0; i < 1 + TILES * 32; ++i)
      mem[i] = i ? -1 : 0;
    kernel<<<1, WARPS * 32>>>(k < 0 ? -1 : k % WARPS, k / WARPS, mem, mem + 1);
    if (cudaDeviceSynchronize() != cudaSuccess)
      return 3;
    for (int i = 0; i < TILES * 32; ++i)
      if (mem[1 + i] != (k < 0 ? WARPS * ROUNDS : -1) || mem[0] != (k < 0 ? 0 : NNTR_CUDA_ERR_TIMEOUT)) {
        printf("unit %d gave up: output %d is %d, status %d\n", k, i, mem[1 + i], mem[0]);
        return 1;
      }
  }
  puts("ok");
  return 0;
}
"""


def test_the_last_warp_of_a_chain_stores_nothing_when_a_warp_in_front_gave_up(tmp_path):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    from nntrainer_b200 import build
    src, exe = tmp_path / "handover_abort.cu", tmp_path / "handover_abort"
    src.write_text(SOURCE)
    ccbin = ["-ccbin", build.HOST_CXX] if os.path.exists(build.HOST_CXX) else []
    subprocess.run([nvcc, *ccbin, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-cudart", "static", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
