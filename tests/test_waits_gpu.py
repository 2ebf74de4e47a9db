"""The bounded wait of a whole warp (garnet_b200/csrc/common.cuh): one answer for all lanes, whatever each of them saw."""
import ctypes
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "garnet_b200", "csrc")
KERNEL = """
#include "common.cuh"
using namespace gb200;
// Lane i waits for barrier i; the lanes of `complete` find theirs done, the others run into a limit of a millisecond.
__global__ void wait_kernel(unsigned complete, int* out)
{
    __shared__ uint64_t bars[32];
    __shared__ int flag;
    const int lane = threadIdx.x;
    mbar_init(&bars[lane], 1);
    if (lane == 0) flag = 0;
    __syncwarp();
    if ((complete >> lane) & 1) mbar_arrive(&bars[lane]);
    __syncwarp();
    const bool there = mbar_wait_warp(&bars[lane], 0, &flag, 1000000ull);
    out[lane] = __shfl_sync(0xffffffffu, int(there), lane);
    __syncwarp();
    if (lane == 0) out[32] = flag;
}
extern "C" int run_wait(unsigned complete, int* out)
{
    wait_kernel<<<1, 32>>>(complete, out);
    return int(cudaDeviceSynchronize());
}
"""


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    path = tmp_path_factory.mktemp("waits")
    (path / "wait.cu").write_text(KERNEL)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-Xcompiler", "-fPIC", "--shared", "-I", CSRC,
                           str(path / "wait.cu"), "-o", str(path / "wait.so")], env=env)
    return ctypes.CDLL(str(path / "wait.so"))


@pytest.mark.parametrize("complete,there", [(0xffffffff, 1), (0x0000ffff, 0), (0x7fffffff, 0), (0xfffffffe, 0), (1, 0), (0, 0)])
def test_a_warp_gives_up_together(waits, complete, there):
    out = torch.full((33,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert waits.run_wait(ctypes.c_uint(complete), ctypes.c_void_p(out.data_ptr())) == 0
    assert out[:32].tolist() == [there] * 32
    assert int(out[32]) == 1 - there
