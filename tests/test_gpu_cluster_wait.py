"""The bounded wait of the cluster kernels (csrc/cluster.cuh): elements that never come end it with a
status within its limit, and the context stays usable."""
from __future__ import annotations

import ctypes
import subprocess

import pytest

import __graft_entry__ as graft

pytestmark = pytest.mark.gpu

# one CTA waits for 8 bytes that nothing sends, then for 8 that it sends itself
SOURCE = r"""
#include "cluster.cuh"
using namespace b2p;
__global__ void __cluster_dims__(1, 1, 1) k(unsigned long long* out) {
    __shared__ uint64_t bar[2];
    __shared__ double v;
    if (threadIdx.x == 0) {
        tx_init(bar);
        tx_init(bar + 1);
        tx_expect(bar, 8);
        tx_expect(bar + 1, 8);
    }
    __syncthreads();
    const unsigned long long t0 = global_ns();
    const bool never = tx_wait(bar, 0);
    const unsigned long long t1 = global_ns();
    if (threadIdx.x == 0) st_async(peer_addr(smem_addr(&v), 0), 3.0, peer_addr(smem_addr(bar + 1), 0));
    const bool sent = tx_wait(bar + 1, 0);
    if (threadIdx.x == 0) {
        out[0] = never;
        out[1] = t1 - t0;
        out[2] = sent && v == 3.0;
        out[3] = kTxWaitNs;
    }
}
extern "C" int run(unsigned long long* out) {
    unsigned long long* d;
    if (cudaMalloc(&d, 32) != cudaSuccess) return 1;
    k<<<1, 64>>>(d);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(out, d, 32, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


def test_a_wait_for_what_never_comes_ends_in_time(b2p, ctx, tmp_path):
    src, so = tmp_path / "wait.cu", tmp_path / "libwait.so"
    src.write_text(SOURCE)
    subprocess.run([graft.NVCC, *graft.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", str(graft.CSRC),
                    "-o", str(so), str(src)], check=True)
    out = (ctypes.c_ulonglong * 4)()
    assert ctypes.CDLL(str(so)).run(out) == 0
    never, ns, sent, limit = out
    assert never == 0 and sent == 1
    # the limit, and at most one suspended try_wait and one sleep more
    assert limit <= ns <= limit + 500_000_000
    assert ctx.norm2([3.0, 4.0]) == 5.0  # the device goes on
