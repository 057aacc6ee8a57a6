"""The bounded waits of the tensor-core kernels (csrc/tcgen05.cuh) when they give up: a small kernel built
around them, because no input makes a wait of the prefill kernel run out."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inquant-open-source_b200", "csrc")
SOURCE = r"""
#include "tcgen05.cuh"
using namespace inq;
// Lanes below `cut` wait for a phase that is complete (the one before a new barrier's first), the others for
// one that nobody completes.
__global__ void wait_kernel(int cut, int tries, int* result, int* flag_out, long long* nanoseconds) {
  __shared__ __align__(8) unsigned long long barrier;
  __shared__ int flag;
  if (threadIdx.x == 0) {
    tc_bar_init(tc_smem(&barrier), 1);
    flag = 0;
  }
  __syncthreads();
  long long times[3];
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(times[0]));
  result[threadIdx.x] = tc_wait(tc_smem(&barrier), threadIdx.x < cut ? 1u : 0u, &flag, tries);
  // what the kernels do next needs the whole warp
  const unsigned chosen = tc_elect();
  result[32 + threadIdx.x] = __popc(__ballot_sync(0xffffffffu, chosen != 0u));
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(times[1]));
  if (flag) tc_wait(tc_smem(&barrier), 0u, &flag);   // the flag is raised: this does not wait for a second
  __syncwarp();
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(times[2]));
  if (threadIdx.x == 0) {
    *flag_out = flag;
    nanoseconds[0] = times[1] - times[0];
    nanoseconds[1] = times[2] - times[1];
  }
}
extern "C" int run_wait(int cut, int tries, int* result, int* flag, long long* nanoseconds) {
  wait_kernel<<<1, 32>>>(cut, tries, result, flag, nanoseconds);
  return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    folder = tmp_path_factory.mktemp("waits")
    source, target = folder / "waits.cu", folder / "waits.so"
    source.write_text(SOURCE)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-I", CSRC, "-shared",
                    "-Xcompiler", "-fPIC", "-o", str(target), str(source)], check=True)
    return ctypes.CDLL(str(target))


@pytest.mark.parametrize("cut", [0, 1, 16, 31, 32])
def test_lanes_whose_wait_gives_up_go_on_with_the_others(library, cut):
    result = torch.full((64,), -1, dtype=torch.int32, device="cuda")
    flag, times = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert library.run_wait(cut, 4096, *(ctypes.c_void_p(t.data_ptr()) for t in (result, flag, times))) == 0
    assert result[:32].tolist() == [1] * cut + [0] * (32 - cut)
    assert result[32:].tolist() == [1] * 32            # one lane is elected, by all of them
    assert flag.item() == int(cut < 32)                # a wait that gave up says so to the other roles
    first, second = times.tolist()
    assert first < 4096 * 20e3                         # 4 us per try were measured: 2^18 tries are about a second
    assert second < 1e6                                # with the flag raised a wait ends after 16 tries
