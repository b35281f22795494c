"""Bits of the packed grid reductions (krylov_dev.cuh), by a kernel of their own: sums that change from one reduction to
the next, compared with exact ones."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from drops_gb300 import build

pytestmark = pytest.mark.gpu

NT = 512
SOURCE = r"""
#include "krylov_dev.cuh"
using namespace tf;
template <class T>
__global__ void __launch_bounds__(512, 1) k_sums(const T* v, T* out, long long* slow, int rounds, PackedAR pa, GridAR g) {
    PkState st;
    unsigned long long epoch = 0;
    for (int r = 0; r < rounds; ++r) {
        T a[1] = {v[((size_t)r * gridDim.x + blockIdx.x) * 512 + threadIdx.x]}, o[1];
        if (!packed_allreduce<1>(pa, st, g, epoch, a, o, (r & 1) != 0)) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            out[r] = o[0];
            slow[r] = (long long)epoch;
        }
    }
}
template <class T>
static int run(int nb, int rounds, const T* v, T* out, long long* slow) {
    const size_t n = (size_t)rounds * nb * 512, words = 2 * kPkWords;
    T *dv = nullptr, *dout = nullptr;
    unsigned long long* dw = nullptr;  // packed words, then the counter and the status
    double* dp = nullptr;
    long long* ds = nullptr;
    cudaMalloc(&dv, n * sizeof(T));
    cudaMalloc(&dout, rounds * sizeof(T));
    cudaMalloc(&dw, (words + 2) * 8);
    cudaMalloc(&dp, (size_t)4 * nb * kArMax * 8);
    cudaMalloc(&ds, rounds * 8);
    cudaMemcpy(dv, v, n * sizeof(T), cudaMemcpyHostToDevice);
    cudaMemset(dw, 0, (words + 2) * 8);
    PackedAR pa{dw, (int*)(dw + words + 1)};
    GridAR g{dw + words, (float*)(dp + (size_t)2 * nb * kArMax), dp, (int*)(dw + words + 1)};
    void* args[] = {&dv, &dout, &ds, &rounds, &pa, &g};
    cudaLaunchCooperativeKernel((const void*)k_sums<T>, nb, 512, args, 0, 0);
    cudaMemcpy(out, dout, rounds * sizeof(T), cudaMemcpyDeviceToHost);
    cudaMemcpy(slow, ds, rounds * 8, cudaMemcpyDeviceToHost);
    cudaFree(dv);
    cudaFree(dout);
    cudaFree(dw);
    cudaFree(dp);
    cudaFree(ds);
    return (int)cudaGetLastError();
}
extern "C" int sums_f32(int nb, int rounds, const float* v, float* out, long long* slow) { return run(nb, rounds, v, out, slow); }
extern "C" int sums_f64(int nb, int rounds, const double* v, double* out, long long* slow) { return run(nb, rounds, v, out, slow); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("packed")
    src, so = str(d / "sums.cu"), str(d / "sums.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    csrc = os.path.join(os.path.dirname(build.__file__), "csrc")
    subprocess.run([build.nvcc(), "-std=c++17", "-O3", *build.ARCH, "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-I", csrc,
                    "-shared", "-o", so, src], check=True)
    return C.CDLL(so)


def device_sums(lib, v):
    """v[rounds, blocks, NT]: the sums, and how many of the reductions up to each took the floating-point form."""
    rounds, nb, _ = v.shape
    out, slow = np.empty(rounds, v.dtype), np.empty(rounds, np.int64)
    fn = lib.sums_f32 if v.dtype == np.float32 else lib.sums_f64
    p = [a.ctypes.data_as(C.c_void_p) for a in (np.ascontiguousarray(v), out, slow)]
    assert fn(C.c_int(nb), C.c_int(rounds), *p) == 0
    return out, slow


def ulps(out, v, unit):
    """error of each sum in units of `unit` times the sum"""
    err = []
    for o, x in zip(out, v):
        vals, counts = np.unique(x, return_counts=True)
        exact = sum(Fraction(float(a)) * int(c) for a, c in zip(vals, counts))
        err.append(float(abs(Fraction(float(o)) - exact) / (abs(exact) * Fraction(unit))) if exact else abs(float(o)))
    return np.array(err)


@pytest.mark.parametrize("nb", [1, 16, 152])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["alike", "random"])
def test_falling_sums_keep_their_bits(lib, nb, dtype, kind):
    """Sums that fall by 2^0 to 2^16 from one reduction to the next: whatever form the reduction takes, the terms'
    rounding adds up to at most half of the type's own rounding (2^-24, 2^-53), so a sum is off by at most 1.5 of it.
    "alike": every term is cut at the same place of its mantissa, so that errors add up.  FP32 terms come from one
    thread of each block: the blocks' own sums are exact, and the packed ones are what is tested.  A sum repeated by
    grid_allreduce is rounded at most 10 times in FP32 (a tree over 32 blocks, then five warps), in FP64 once for the
    warp, the block and the grid, and its terms to a quarter of their sum's last place each time."""
    f32 = dtype == np.float32
    bits = 23 if f32 else 52
    rng = np.random.default_rng(3)
    rounds = []
    for drop in range(17):
        for k in (0, drop):  # back up, then down
            if kind == "random":
                x = (1.0 + rng.random((nb, NT))) * 2.0**-k
            else:
                x = np.full((nb, NT), (1.0 + rng.integers(1, 2**bits) * 2.0**-bits) * 2.0**-k)
            if f32:
                x[:, 1:] = 0.0
            rounds.append(x.astype(dtype))
            rounds.append(rounds[-1])  # the second in units of the same sum
    v = np.stack(rounds)
    out, slow = device_sums(lib, v)
    err = ulps(out, v, 2.0**-24 if f32 else 2.0**-53)
    repeated = np.diff(np.concatenate([[0], slow])) > 0
    assert err[~repeated].max() <= 1.5, err.round(2)
    assert err[repeated].max() <= (10.0 if f32 else 5.0), err.round(2)
    assert not repeated[1::2].any()  # an unchanged sum is never repeated


@pytest.mark.parametrize("nb", [1, 152])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_jumps_zeros_and_no_numbers(lib, nb, dtype):
    """Growth past the words' range, a sum held by one block, zero, infinity and NaN, and back."""
    one = np.zeros((nb, NT), dtype)
    one[:, 0] = 1.0
    corner = np.zeros((nb, NT), dtype)
    corner[nb - 1, 0] = 3.0 * nb
    inf, nan = one.copy(), one.copy()
    inf[0, 0], nan[nb - 1, 0] = np.inf, np.nan
    rounds = [one, one, one * 1024, one * 2.0**40, one, corner, corner, one, one * 0, one, one, inf, one, one, nan, one, one]
    v = np.stack(rounds).astype(dtype)
    out, _ = device_sums(lib, v)
    want = v.astype(np.float64).sum(axis=(1, 2))
    assert np.array_equal(out, want.astype(dtype), equal_nan=True)
