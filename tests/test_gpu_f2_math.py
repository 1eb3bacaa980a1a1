"""The packed arithmetic of the growth normals (csrc/to_f2.cuh) on the GPU, a
kernel of this test over every 24-bit uniform: the square root of -2 log(u)
against CUDA's sqrtf, and the Box-Muller pairs of two paths against the scalar
ones, bit for bit in both halves of the pair."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
CSRC = Path(__file__).resolve().parents[1] / "transportoptimiser_gb300" / "csrc"

SOURCE = r"""
#include "to_f2.cuh"
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__global__ void k(unsigned* bad) {
    __shared__ to_bm_tables tab;
    to_bm_load(tab);
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, j = 0xFFFFFFu - i;   // 2^24 threads
    const uint32_t ai = i << 8, aj = j << 8, bi = i * 2654435761u, bj = ~bi * 0x9E3779B9u;
    const float xi = -2.0f * to_log_u01(ai), xj = -2.0f * to_log_u01(aj);
    float ri, rj;
    unpack2(to_sqrt2(pack2(xi, xj)), ri, rj);
    if (!same(ri, sqrtf(xi)) || !same(rj, sqrtf(xj))) atomicAdd(bad, 1u);
    f2 c, s;
    to_box_muller2(ai, bi, aj, bj, tab, c, s);
    float ci, cj, si, sj, wc, ws;
    unpack2(c, ci, cj);
    unpack2(s, si, sj);
    to_box_muller(ai, bi, &wc, &ws);
    bool ok = same(ci, wc) && same(si, ws);
    to_box_muller(aj, bj, &wc, &ws);
    ok = ok && same(cj, wc) && same(sj, ws);
    if (!ok) atomicAdd(bad + 1, 1u);
}
extern "C" int run(unsigned* out) {
    unsigned* d = nullptr;
    if (cudaMalloc(&d, 8) != cudaSuccess) return 1;
    cudaMemset(d, 0, 8);
    k<<<(1 << 24) / 256, 256>>>(d);
    const cudaError_t e = cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 1;
}
"""


def test_packed_normals_equal_scalar_for_every_uniform(ctx, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, lib = tmp_path / "t.cu", tmp_path / "t.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode=arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-I", str(CSRC), str(src),
                    "-o", str(lib)], check=True, capture_output=True, text=True)
    bad = (ctypes.c_uint * 2)(7, 7)
    assert ctypes.CDLL(str(lib)).run(bad) == 0
    assert list(bad) == [0, 0]
