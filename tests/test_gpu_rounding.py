"""recip, root and quot of csrc/gfsph_device.cuh against CUDA's IEEE operators,
bit for bit: the first two over every mantissa at several exponents of their
range, the quotient over seeded random operands and over dividends next to
the midpoints between two floats."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "deslizamientos-y-flujos_b200", "csrc")

SOURCE = r"""
#include "gfsph_device.cuh"
using namespace gfsph;
__global__ void k_check(unsigned long long* bad) {
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const int ex[6] = {-60, -31, -1, 0, 28, 59};
    unsigned long long b0 = 0, b1 = 0, b2 = 0;
    for (unsigned m = tid; m < (1u << 23); m += nt)
        for (int e = 0; e < 6; e++) {
            const float b = __uint_as_float(((unsigned)(127 + ex[e]) << 23) | m);
            if (recip(b) != __fdiv_rn(1.f, b)) b0++;
            if (root(b) != __fsqrt_rn(b)) b1++;
        }
    unsigned long long s = 88172645463325252ULL + tid * 7919000003ULL;
    for (int i = 0; i < 4000; i++) {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;
        const float b = __uint_as_float(0x3f800000u | (unsigned)((s >> 23) & 0x7fffffu));
        float a = __uint_as_float(0x3f800000u | (unsigned)(s & 0x7fffffu));
        if (i & 1) a = (float)(((double)a + ldexp(1.0, -24)) * (double)b);  // a/b next to a midpoint
        if (quot(a, b, recip(b)) != __fdiv_rn(a, b)) b2++;
    }
    if (b0) atomicAdd(bad, b0);
    if (b1) atomicAdd(bad + 1, b1);
    if (b2) atomicAdd(bad + 2, b2);
}
extern "C" int check(unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc((void**)&d, 24) != cudaSuccess || cudaMemset(d, 0, 24) != cudaSuccess) return 1;
    k_check<<<148 * 8, 256>>>(d);
    const int st = cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return st;
}
"""


def test_recip_root_quot_round_correctly(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "check.cu", tmp_path / "check.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(so)], check=True, capture_output=True)
    out = (C.c_ulonglong * 3)()
    assert C.CDLL(str(so)).check(out) == 0
    assert list(out) == [0, 0, 0]


POW = r"""
#include "gfsph_device.cuh"
using namespace gfsph;
__global__ void k_check(unsigned long long* bad) {
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const int ex[7] = {-60, -24, -7, -1, 0, 3, 14};
    unsigned long long b0 = 0;
    for (unsigned m = tid; m < (1u << 23); m += nt)
        for (int e = 0; e < 7; e++) {
            const float x = __uint_as_float(((unsigned)(127 + ex[e]) << 23) | m);
            if (pow73(x) != powr(x, 7.f / 3.f)) b0++;
        }
    if (b0) atomicAdd(bad, b0);
}
extern "C" int check(unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc((void**)&d, 24) != cudaSuccess || cudaMemset(d, 0, 24) != cudaSuccess) return 1;
    k_check<<<148 * 8, 256>>>(d);
    const int st = cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return st;
}
"""


PAIR = r"""
#include "gfsph_device.cuh"
using namespace gfsph;
__device__ float rnd(unsigned long long& s) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    return __uint_as_float(0x3f800000u | (unsigned)(s & 0x7fffffu)) - 1.f;
}
__global__ void k_check(unsigned long long* bad) {
    unsigned long long s = 88172645463325252ULL + (blockIdx.x * blockDim.x + threadIdx.x) * 7919000003ULL;
    for (int i = 0; i < 20; i++) rnd(s);
    unsigned long long b0 = 0, b1 = 0, b2 = 0;
    for (int it = 0; it < 1000; it++) {
        // separations from 0 to the support and beyond the spline's inner edge, smoothing lengths over 13 decades
        float w[2], t[2], dr[2], h[2];
        for (int k = 0; k < 2; k++) {
            h[k] = exp10f(-5.5f + 13.f * rnd(s));
            const float a = 6.2831853f * rnd(s), q = (it % 50 == 0) ? (it % 100 ? 1.f : 0.f) : 2.f * rnd(s);
            const float dx = q * h[k] * cosf(a), dy = q * h[k] * sinf(a);
            dr[k] = dx * dx + dy * dy;
            if (!(sqrtf(dr[k]) < 2.f * h[k])) dr[k] = 0.f;
            float wr, g0, g1, wi, ti, d0, d1, e0, e1;
            sph_kernel<1>(sqrtf(dr[k]), dx, dy, h[k], wr, g0, g1);
            spline_pair(dr[k], h[k], true, w[k], t[k]);
            spline_pair(dr[k], h[k], false, wi, ti);
            if (w[k] != wr || wi != wr || t[k] != ti) b0++;
            if (dr[k] != dx * dx + dy * dy) continue;
            spline_grad(t[k], dx, dy, true, d0, d1);
            spline_grad(t[k], dx, dy, false, e0, e1);
            if (d0 != g0 || d1 != g1 || e0 != g0 || e1 != g1) b1++;
        }
        F2 w2, t2;
        spline_pair2(f2(dr[0], dr[1]), f2(h[0], h[1]), w2, t2);
        float x, y;
        split(w2, x, y);
        if (x != w[0] || y != w[1]) b2++;
        split(t2, x, y);
        if (x != t[0] || y != t[1]) b2++;
    }
    if (b0) atomicAdd(bad, b0);
    if (b1) atomicAdd(bad + 1, b1);
    if (b2) atomicAdd(bad + 2, b2);
}
extern "C" int check(unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc((void**)&d, 24) != cudaSuccess || cudaMemset(d, 0, 24) != cudaSuccess) return 1;
    k_check<<<148 * 8, 256>>>(d);
    const int st = cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return st;
}
"""


def test_pair_kernels_agree_bit_for_bit(tmp_path):
    """spline_pair and spline_grad, with shared reciprocals and without, and the
    two-pairs-at-once spline_pair2 against the plain kernel function."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "pair.cu", tmp_path / "pair.so"
    src.write_text(PAIR)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(so)], check=True, capture_output=True)
    out = (C.c_ulonglong * 3)()
    assert C.CDLL(str(so)).check(out) == 0
    assert list(out) == [0, 0, 0]


def test_manning_power_equals_the_fp64_power(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "pow.cu", tmp_path / "pow.so"
    src.write_text(POW)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(so)], check=True, capture_output=True)
    out = (C.c_ulonglong * 3)()
    assert C.CDLL(str(so)).check(out) == 0
    assert out[0] == 0
