"""Waits in front of instructions that take a whole warp: the lanes have to go on or leave together, also when some of them see a
phase completed and the others give up."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nntrainer_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include "common.cuh"
#include "pipeline.cuh"
using namespace nntr;
__global__ void kernel(int patient, int *status, int *out) { // lanes below `patient` poll the completed phase, the others not once
  __shared__ alignas(8) unsigned long long done;
  __shared__ int flag_word;
  const int lane = threadIdx.x;
  if (lane == 0) {
    flag_word = 0;
    mbar_init(smem_u32(&done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_arrive(smem_u32(&done));
  }
  __syncthreads();
  out[lane] = mbar_wait_warp(smem_u32(&done), 0, &flag_word, status, lane < patient ? 4096 : 0, 8192);
}
int main() {
  int *mem;
  if (cudaMallocManaged(&mem, 33 * sizeof(int)) != cudaSuccess)
    return 2;
  for (int patient = 0; patient <= 32; ++patient) {
    mem[32] = 0;
    kernel<<<1, 32>>>(patient, mem + 32, mem);
    if (cudaDeviceSynchronize() != cudaSuccess)
      return 3;
    for (int i = 0; i < 32; ++i)
      if (mem[i] != (patient == 32) || mem[32] != (patient == 32 ? 0 : NNTR_CUDA_ERR_TIMEOUT)) {
        printf("%d lanes polled: lane %d has %d, status %d\n", patient, i, mem[i], mem[32]);
        return 1;
      }
  }
  puts("ok");
  return 0;
}
"""


@pytest.mark.gpu
def test_a_warps_wait_ends_alike_in_every_lane(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    from nntrainer_b200 import build
    src, exe = tmp_path / "warp_wait.cu", tmp_path / "warp_wait"
    src.write_text(SOURCE)
    ccbin = ["-ccbin", build.HOST_CXX] if os.path.exists(build.HOST_CXX) else []
    subprocess.run([nvcc, *ccbin, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-cudart", "static", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def _block(text, start):
    """The text of the braces that open behind position start."""
    i, depth = text.index("{", start) + 1, 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[start:i]


def test_the_warps_that_turn_value_tiles_wait_as_warps():
    """The turners' loads (ldmatrix) and barriers (__syncwarp) take all lanes: neither their share of a tile nor the loop around it
    may be entered or left by a part of a warp. By reading, because no wait of the kernel runs out when nothing is wrong."""
    with open(os.path.join(CSRC, "attention.cu")) as f:
        text = f.read()
    turn = _block(text, text.index("auto turn = [&]"))
    loop = _block(text, text.index("else if (turner)"))
    assert "ldmatrix.sync.aligned" in turn and "turn(turned++)" in loop
    for part in (turn, loop):
        assert re.findall(r"mbar_\w*wait\w*", part) == ["mbar_wait_warp"]
