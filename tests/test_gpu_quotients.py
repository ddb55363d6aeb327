"""recip_any, root_any and quot2 of csrc/gfsph_device.cuh against CUDA's IEEE operators for operands of every
size: zeros, subnormals, the edges of the ranges they hand to the shared-reciprocal forms, infinities and NaN.  Equal
values (either zero, any NaN).  And the pair kernels' shared-reciprocal form at the ends of its range of smoothing lengths,
where its quotients are smallest (next to the edge of the support) and largest, against the plain one."""
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
__device__ bool same(float a, float b) { return a == b || (a != a && b != b); }
__device__ float operand(unsigned long long& s, int i) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    const unsigned bits = (unsigned)(s >> 16);
    switch (i % 8) {
        case 0: return __uint_as_float(bits & 0x80000000u);                     // a zero
        case 1: return __uint_as_float(bits & 0x807fffffu);                     // subnormal
        case 2: return __uint_as_float((bits & 0x80000000u) | 0x7f800000u);     // infinity
        case 3: return (bits & 64) ? __uint_as_float(0x7fc00000u) : __uint_as_float(bits);
        case 4: return __uint_as_float(0x21800000u + (bits & 0x1ffffu) - 0x10000u);  // about 2^-60
        case 5: return -__uint_as_float(0x5e000000u + (bits & 0x1ffffu) - 0x10000u);  // about 2^61
        default: return __uint_as_float(bits);                                  // any exponent
    }
}
__global__ void k_check(unsigned long long* bad) {
    unsigned long long s = 88172645463325252ULL + (blockIdx.x * blockDim.x + threadIdx.x) * 7919000003ULL;
    unsigned long long n[3] = {0, 0, 0};
    for (int i = 0; i < 6400; i++) {
        const float a = operand(s, i / 8), c = operand(s, i / 64);
        const float b = fabsf((i & 1) ? operand(s, i / 512) : exp10f(-20.f + 40.f * (float)((s >> 40) & 0xffff) / 65536.f));
        if (b != b) continue;
        float qa, qc;
        quot2(a, c, b, qa, qc);
        if (b > 0.f && (!same(qa, __fdiv_rn(a, b)) || !same(qc, __fdiv_rn(c, b)))) n[0]++;
        if (b > 0.f && !same(recip_any(b), __fdiv_rn(1.f, b))) n[1]++;
        if (!same(root_any(a), __fsqrt_rn(a))) n[2]++;
    }
    for (int k = 0; k < 3; k++)
        if (n[k]) atomicAdd(bad + k, n[k]);
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


EDGES = r"""
#include "gfsph_device.cuh"
using namespace gfsph;
__global__ void k_check(unsigned long long* bad) {
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
    const float hs[4] = {kQuotMin, 1.37f * kQuotMin, 0.61f * kQuotMax, kQuotMax};
    for (int m = 0; m < 4; m++) {
        const float h = hs[m], edge = 4.f * h * h;
        // squares of distances: the floats below the edge of the support, and from 0 on
        const float dr[2] = {__uint_as_float(__float_as_uint(edge) - 1u - tid), edge * exp10f(-30.f * (float)tid / 303104.f)};
        float w[2], t[2], wr, tr;
        for (int k = 0; k < 2; k++) {
            if (!(sqrtf(dr[k]) < 2.f * h)) continue;
            spline_pair(dr[k], h, true, w[k], t[k]);
            spline_pair(dr[k], h, false, wr, tr);
            if (w[k] != wr || t[k] != tr) atomicAdd(bad + k, 1ULL);
            F2 w2, t2;
            spline_pair2(f2(dr[k], dr[k]), f2(h), w2, t2);
            float a, b, c, d;
            split(w2, a, b);
            split(t2, c, d);
            if (a != wr || b != wr || c != tr || d != tr) atomicAdd(bad + 2, 1ULL);
        }
    }
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


@pytest.mark.parametrize("source", ["SOURCE", "EDGES"])
def test_equal_to_the_operators(tmp_path, source):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, so = tmp_path / "check.cu", tmp_path / "check.so"
    src.write_text(globals()[source])
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(so)], check=True, capture_output=True)
    out = (C.c_ulonglong * 3)()
    assert C.CDLL(str(so)).check(out) == 0
    assert list(out) == [0, 0, 0]
