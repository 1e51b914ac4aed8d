"""pt_fp64.cuh: products, sums, differences and quotients in fused form round like the plain operations."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "pt_fp64.cuh"
__global__ void k(const double* a, const double* b, double* o, int* in, int n, pt::FmaForms F) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = F.mul(a[i], b[i]);
    o[n + i] = F.add(a[i], b[i]);
    o[2 * n + i] = F.sub(a[i], b[i]);
    in[i] = pt::in_range(a[i], 800) && pt::in_range(b[i], 100);
    o[3 * n + i] = in[i] ? pt::quotient(a[i], b[i], 1.0 / b[i]) : 0.0;
}
extern "C" int forms(const double* a, const double* b, double* o, int* in, int n) {
    double *da, *db, *dout;
    int* di;
    const size_t s = sizeof(double) * (size_t)n;
    if (cudaMalloc(&da, s) || cudaMalloc(&db, s) || cudaMalloc(&dout, 4 * s) || cudaMalloc(&di, sizeof(int) * (size_t)n)) return 1;
    cudaMemcpy(da, a, s, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, s, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(da, db, dout, di, n, pt::FmaForms());
    cudaMemcpy(o, dout, 4 * s, cudaMemcpyDeviceToHost);
    cudaMemcpy(in, di, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(da), cudaFree(db), cudaFree(dout), cudaFree(di);
    return (int)cudaGetLastError();
}
"""


def test_fused_forms_round_like_the_plain_operations(tmp_path):
    from projectracer_gb300 import build

    src, lib = tmp_path / "forms.cu", tmp_path / "libforms.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.CSRC, "-shared",
                                                  str(src), "-o", str(lib)], check=True)
    L = ctypes.CDLL(os.fspath(lib))
    rng = np.random.default_rng(11)
    # mantissas at random and at the edges of a binade, exponents over the accepted ranges and past them
    edge = np.array([1.0, 1 + 2.0**-52, 1 + 2.0**-51, 1.25, 1.5 - 2.0**-52, 1.5, 1.5 + 2.0**-52, 2 - 2.0**-51, 2 - 2.0**-52])
    x, y = (m.ravel() for m in np.meshgrid(edge, edge))
    n = 1 << 21
    a = np.concatenate([1 + rng.random(n), np.repeat(x, 500), 1 + rng.random(n // 4), np.repeat(edge, n // 32)])
    b = np.concatenate([1 + rng.random(n), np.repeat(y, 500), np.resize(edge, n // 4), 1 + rng.random(n // 32 * edge.size)])
    a = np.ldexp(a, rng.integers(-802, 803, a.size)) * rng.choice([-1.0, 1.0], a.size)
    b = np.ldexp(b, rng.integers(-102, 103, b.size)) * rng.choice([-1.0, 1.0], b.size)
    # zeros of both signs, infinities, NaN, subnormals, the ends of the ranges
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.0**-1060, 1.0, -1.0, 2.0**-800, 2.0**800, 2.0**-100,
                    -2.0**100, np.nextafter(2.0**-800, 0), np.nextafter(2.0**800, 0), np.nextafter(2.0**100, 0), 1e308])
    u, v = (m.ravel() for m in np.meshgrid(odd, odd))
    a, b = np.concatenate([a, u]), np.concatenate([b, v])
    out, ok = np.empty((4, a.size)), np.empty(a.size, dtype=np.int32)
    vp = ctypes.c_void_p
    assert L.forms(vp(a.ctypes.data), vp(b.ctypes.data), vp(out.ctypes.data), vp(ok.ctypes.data), a.size) == 0

    def same(got, ref):
        nan = np.isnan(ref)
        return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.int64), ref[~nan].view(np.int64))

    with np.errstate(all="ignore"):
        assert same(out[0], a * b)
        assert same(out[1], a + b)
        assert same(out[2], a - b)
        inside = lambda w, bits: (np.abs(w) >= 2.0**-bits) & (np.abs(w) < 2.0**bits)  # noqa: E731
        assert np.array_equal(ok == 1, inside(a, 800) & inside(b, 100))
        q = ok == 1
        assert q.sum() > 0.9 * n and same(out[3][q], a[q] / b[q])
