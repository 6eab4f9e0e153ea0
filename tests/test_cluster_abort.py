"""What the CTAs of a cluster do when one of them gave up on a wait: all of them have to know before they use its part of a
result. csrc/cluster.cuh in a small program of its own, because no wait of a kernel runs out when nothing is wrong: one CTA
raises its flag, and behind the barrier the flags of its cluster are up and those of every other cluster are not."""
import os
import shutil
import subprocess

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nntrainer_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "cluster.cuh"
#include "pipeline.cuh"
using namespace nntr;
__global__ void kernel(int who, int thread, int push, int *out) {
  __shared__ int flag_word;
  volatile int *flag = &flag_word;
  if (threadIdx.x == 0)
    *flag = 0;
  __syncthreads();
  cluster_arrive();
  if ((int)blockIdx.x == who && (int)threadIdx.x == thread)
    *flag = 1;
  __syncwarp();
  cluster_wait();
  if (push && *flag)
    raise_in_cluster(smem_u32(&flag_word));
  __syncwarp();
  cluster_sync();
  out[blockIdx.x * blockDim.x + threadIdx.x] =
    push ? *flag : __any_sync(0xffffffffu, neighbour_raised(smem_u32(&flag_word), threadIdx.x & 31));
  cluster_sync();
}
int main(int, char **argv) {
  const int parts = atoi(argv[1]), clusters = 3, threads = 96, n = parts * clusters * threads;
  int *out;
  if (cudaMallocManaged(&out, n * sizeof(int)) != cudaSuccess)
    return 2;
  for (int k = -2; k < 2 * parts * clusters; ++k) {
    const int who = k / 2 - (k < 0), push = k & 1;
    if (launch_in_clusters(kernel, dim3(clusters), parts, threads, 0, cudaStream_t(0), who, (31 * who) % threads, push, out) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess)
      return 3;
    for (int i = 0; i < n; ++i)
      if (out[i] != (who >= 0 && i / threads / parts == who / parts)) {
        printf("parts %d, push %d, CTA %d gave up: CTA %d, thread %d sees %d\n", parts, push, who, i / threads, i % threads, out[i]);
        return 1;
      }
  }
  puts("ok");
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    from nntrainer_b200 import build
    d = tmp_path_factory.mktemp("cluster")
    src, exe = d / "cluster_abort.cu", d / "cluster_abort"
    src.write_text(SOURCE)
    ccbin = ["-ccbin", build.HOST_CXX] if os.path.exists(build.HOST_CXX) else []
    subprocess.run([nvcc, *ccbin, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-cudart", "static", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("parts", [2, 4, 8])
def test_a_cta_that_gave_up_is_known_to_its_cluster_and_to_no_other(program, parts):
    r = subprocess.run([program, str(parts)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
