"""The bounded wait of the prompt kernels (csrc/prompt_f16.cuh, wait_warp), on a barrier that nothing completes: it gives up within the second or two that the
kernels state, and within milliseconds once another role of the CTA has."""
import ctypes
import os
import subprocess

import pytest
import torch

from candle_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "prompt_f16.cuh"
__device__ unsigned long long now_ns() { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }
__global__ void wait_kernel(int *out, int abort_after_2ms) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) { cq_mbar_init(&bar, 1); abort_flag = 0; cq_fence_mbar_init(); }
    __syncthreads();
    const unsigned long long t0 = now_ns();
    if (threadIdx.x < 32) {
        const bool done = cq_prompt::wait_warp(&bar, 0, &abort_flag);
        if (threadIdx.x == 0) { out[0] = done; out[1] = *(volatile int *)&abort_flag; out[2] = (int)((now_ns() - t0) / 1000000); }
    } else if (abort_after_2ms) {
        for (int i = 0; i < 10000000 && now_ns() - t0 < 2000000; ++i) {}
        *(volatile int *)&abort_flag = 1;
    }
}
extern "C" int run(int *out, int abort_after_2ms) {
    wait_kernel<<<1, 64>>>(out, abort_after_2ms);
    return (int)cudaDeviceSynchronize();
}
"""


def test_a_wait_that_nothing_ends_gives_up_in_time(cuda_dev, tmp_path):
    src, so = tmp_path / "wait.cu", tmp_path / "libwait.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include"), "-shared", str(src), "-o", str(so)], check=True)
    run = ctypes.CDLL(str(so)).run
    out = torch.full((3,), -1, dtype=torch.int32, device=cuda_dev)
    assert run(ctypes.c_void_p(out.data_ptr()), 0) == 0
    done, aborted, ms = out.tolist()
    assert (done, aborted) == (0, 1) and 500 <= ms <= 4000       # 2e9 clocks at 0.5 - 2 GHz, and the tries between two looks at the clock
    assert run(ctypes.c_void_p(out.data_ptr()), 1) == 0
    done, aborted, ms = out.tolist()
    assert (done, aborted) == (0, 1) and ms <= 100
