"""The exponential and the quotient of the double-float line solve (fh_hline_df.cuh)
over their ranges (kHdfExp; quotients that a pair holds), against 64-bit and longer host arithmetic.  The kernel is built
from the header by the test.

Bounds: the exponential ends in T + T t with a table value T rounded to 2^-49 and
|t| < 0.022, one double-float multiply-add (2^-46 with the renormalisation); the
argument's parts of ln 2 / 16 add n 2^-64, the series' next term 2^-51: 2^-45
relative.  The quotient corrects twice by its remainder: 2^-46."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

SRC = r"""
#include "fhist.h"
#include "fh_hline_df.cuh"
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <vector>
// the pair of a value that is one (fh_df_bits itself rounds to 2^-48)
__device__ fh_df pair_of(double x) {
  const float h = (float)x;
  return fh_df{h, (float)(x - (double)h)};
}
__global__ void k_exp(const double *x, float2 *y, int n) {
  __shared__ float2 tab[16];
  if (threadIdx.x < 16) tab[threadIdx.x] = kHdfTab[threadIdx.x];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fh_df_pair(fh_df_exp(pair_of(x[i]), tab));
}
__global__ void k_quot(const double *a, const double *b, float2 *y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fh_df_pair(fh_df_quot(pair_of(a[i]), pair_of(b[i])));
}
static uint64_t st = 88172645463325252ull;
static double rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return (double)(st >> 11) * 0x1p-53; }
static double pair48(double x) { const float h = (float)x; return (double)h + (double)(float)(x - (double)h); }  // as a pair
int main(int argc, char **argv) {
  const bool want_exp = argc > 1 && argv[1][0] == 'e';
  const int n = 1 << 20;
  std::vector<double> x(n), a(n), b(n);
  for (int i = 0; i < n; ++i) {
    x[i] = pair48(2.0 * kHdfExp * rnd() - kHdfExp);
    if (i % 4 == 1) x[i] = pair48(x[i] * ldexp(1.0, -(int)(40 * rnd())));
    if (i % 4 == 2) x[i] = pair48(log(2.0) / 32 * (int)(113 * rnd() - 56) * (1 + 1e-7 * rnd()));  // ends of the table's intervals
    a[i] = pair48((1 + rnd()) * ldexp(i & 1 ? 1 : -1, (int)(120 * rnd() - 60)));
    b[i] = pair48((1 + rnd()) * ldexp(i & 2 ? 1 : -1, (int)(120 * rnd() - 60)));
  }
  x[0] = 0; x[1] = kHdfExp; x[2] = -kHdfExp;
  double *dx, *da, *db;
  float2 *dy;
  cudaMalloc(&dx, 8 * n); cudaMalloc(&da, 8 * n); cudaMalloc(&db, 8 * n); cudaMalloc(&dy, 8 * n);
  cudaMemcpy(dx, x.data(), 8 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(da, a.data(), 8 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b.data(), 8 * n, cudaMemcpyHostToDevice);
  std::vector<float2> y(n);
  long double we = 0, wq = 0;
  k_exp<<<n / 256, 256>>>(dx, dy, n);
  cudaMemcpy(y.data(), dy, 8 * n, cudaMemcpyDeviceToHost);
  for (int i = 0; i < n; ++i) {
    const long double e = expl((long double)x[i]);
    we = fmaxl(we, fabsl(((long double)y[i].x + y[i].y - e) / e));
  }
  k_quot<<<n / 256, 256>>>(da, db, dy, n);
  const cudaError_t err = cudaMemcpy(y.data(), dy, 8 * n, cudaMemcpyDeviceToHost);
  for (int i = 0; i < n; ++i) {
    const long double q = (long double)a[i] / (long double)b[i];
    if (fabsl(q) >= 0x1p-78L) wq = fmaxl(wq, fabsl(((long double)y[i].x + y[i].y - q) / q));  // a pair holds it
  }
  printf("%s exp 2^%.2f quotient 2^%.2f\n", cudaGetErrorString(err), (double)log2l(we), (double)log2l(wq));
  return err != cudaSuccess || !(want_exp ? we <= 0x1p-45L : wq <= 0x1p-46L);
}
"""


@pytest.mark.parametrize("what", ["quotient", "exp"])
def test_accuracy(what, tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "dff.cu", tmp_path / "dff"
    src.write_text(SRC)
    csrc = os.path.join(REPO, "theses_code_gb300", "csrc")
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                        "arch=compute_103a,code=sm_103a", "-I", csrc, "-I", os.path.join(REPO, "include"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), what], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
