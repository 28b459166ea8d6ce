"""The rounded quotients and square roots of gray_b200/csrc/round64.cuh against
the operators, on the device and with its seeds: equal for every operand that
all_ones() does not mark, and the marked ones are the exception."""
import ctypes
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gray_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SRC = r"""
#include "round64.cuh"
using namespace round64;
__global__ void check(const double *x, const double *a, long long n, unsigned long long *bad)
{
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= n)
		return;
	const double b = x[i];
	if(all_ones(b)) {
		atomicAdd(bad + 4, 1ull);
		return;
	}
	double y;
	const double r = 1.0 / b;
	atomicAdd(bad + 0, (unsigned long long)(sqrt_rn(b, y) != sqrt(b)));
	atomicAdd(bad + 1, (unsigned long long)(rcp_rn(b) != r));
	/* as the kernels start it: from the root's own 1/sqrt, twice from a few ulp */
	const double s = sqrt_rn(b, y);
	atomicAdd(bad + 2, (unsigned long long)(rcp_near(s, y) != 1.0 / s && !all_ones(s)));
	for(int k = -4; k <= 4; ++k)
		atomicAdd(bad + 2, (unsigned long long)(rcp_near(b, rcp_near(b, fma(r, k * 0x1p-52, r))) != r));
	atomicAdd(bad + 3, (unsigned long long)(div_rn(a[i], b, r) != a[i] / b));
}
__global__ void powers(const double *x, double *y, long long n)
{
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n)
		y[i] = pow_m07(x[i]);
}
extern "C" int pow_run(const double *x, double *y, long long n)
{
	double *d = 0;
	if(cudaMalloc(&d, 2 * n * sizeof(double)))
		return 1;
	cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
	powers<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, n);
	cudaError_t e = cudaMemcpy(y, d + n, n * sizeof(double), cudaMemcpyDeviceToHost);
	cudaFree(d);
	return e != cudaSuccess;
}
extern "C" int run(const double *x, const double *a, long long n, unsigned long long *out)
{
	double *d = 0;
	unsigned long long *c = 0;
	if(cudaMalloc(&d, 2 * n * sizeof(double)) || cudaMalloc(&c, 5 * sizeof(*c)))
		return 1;
	cudaMemset(c, 0, 5 * sizeof(*c));
	cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
	cudaMemcpy(d + n, a, n * sizeof(double), cudaMemcpyHostToDevice);
	check<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, n, c);
	cudaError_t e = cudaMemcpy(out, c, 5 * sizeof(*c), cudaMemcpyDeviceToHost);
	cudaFree(d);
	cudaFree(c);
	return e != cudaSuccess;
}
"""


def near_middles():
    """Radicands whose roots lie next to the middle of two numbers: x with
    4 x 2^k' = (2m + 1)^2 - s for small s, from the square roots of s mod 2^k."""
    out = []
    for k in (54, 55):
        for s in range(-255, 256):
            if s % 8 != 1:
                continue
            r = 1
            for b in range(3, k):
                if ((r * r - s) >> b) & 1:
                    r += 1 << (b - 1)
            for t in (r, -r, r + (1 << (k - 1)), (1 << (k - 1)) - r):
                t %= 1 << k
                while t < 1 << 54:
                    x, rest = divmod(t * t - s, 1 << k)
                    if t >= 1 << 53 and rest == 0 and 1 << 52 <= x < 1 << 53:
                        out.append(np.ldexp(float(x), k - 2 - 104))
                    t += 1 << k
    return np.array(out)


def operands():
    rng = np.random.default_rng(5)
    grid = np.ldexp((1.0 + np.arange(64) / 64.0)[:, None], np.arange(2)[None, :]).ravel()
    near = (grid.view(np.int64)[:, None] + np.arange(-3000, 3001)[None, :]).ravel().view(np.float64)
    # 2^106 + 1 = 9007199120523265 x 9007199388958721: a reciprocal 2^-53 ulp below a middle
    odd = np.array([9007199120523265.0, 4503599694479360.0]) * 2.0**-52
    x = np.concatenate([near_middles(), near, near * near, odd, rng.uniform(1.0, 4.0, 1 << 22),
                        np.exp(rng.uniform(np.log(1e-6), np.log(1e60), 1 << 21))])
    a = np.concatenate([rng.uniform(0.5, 8.0, x.size - near.size), rng.permutation(near)])
    return x, a


def test_the_hard_radicands_are_hard():
    """In integers: 4 x 4^j is an odd square less a small number, so the root is
    half an odd integer but for less than 2^-46."""
    xs = near_middles()
    assert xs.size > 50
    for x in xs:
        n, d = float(x).as_integer_ratio()
        v = 4 * n * (1 << 106) // d
        v = v if v < 1 << 108 else v >> 2
        t = math.isqrt(v) | 1
        assert min(abs(v - q * q) for q in (t - 2, t, t + 2)) < 256


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("round64")
    (d / "r.cu").write_text(SRC)
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                           "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, "-o", str(d / "libr.so"), str(d / "r.cu")])
    return ctypes.CDLL(str(d / "libr.so"))


@pytest.mark.gpu
def test_equal_to_the_operators(lib):
    x, a = operands()
    out = (ctypes.c_ulonglong * 5)()
    f = lib.run
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p]
    assert f(x.ctypes.data, a.ctypes.data, x.size, ctypes.byref(out)) == 0
    assert list(out)[:4] == [0, 0, 0, 0]      # roots, reciprocals, refined ones, quotients
    assert 0 < out[4] < 1000                  # the exception is met and is rare


@pytest.mark.gpu
@pytest.mark.parametrize("span", [0.01, 1.5, np.log(1e9)])
def test_power(lib, span):
    """Each rounding is at most 2^-53 of its value: u carries two and enters
    five times, its powers and x^2 carry seven with their weights (6 in sum), a
    tenth of which reaches the result, and one more: 1 + (10 + 6) / 10."""
    x = np.exp(np.random.default_rng(3).uniform(-span, span, 1 << 21))
    y = np.empty_like(x)
    f = lib.pow_run
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong]
    assert f(x.ctypes.data, y.ctypes.data, x.size) == 0
    want = x.astype(np.longdouble) ** np.longdouble(-0.7)
    err = np.abs((y.astype(np.longdouble) - want) / want) * 2.0**53
    print("x^-0.7: mean %.3f, max %.3f x 2^-53" % (err.mean(), err.max()))
    assert err.max() <= 2.6
