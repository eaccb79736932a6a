"""The 3x3 solve of the walls' first-order systems by itself (pinv3_solve, csrc/sph_math.cuh), against
numpy's float64 pseudo-inverse of the same float32 matrix with the same cut-off: conditions
from 1 to 1e7 on both sides of the bound between the adjugate and the singular value sweeps
(2.5e6) and of the cut-off at 3 FLT_EPSILON (2.8e6), rank 2, and entries scaled from 1e-12 to 1e12.

Tolerance, relative to |b| / (smallest singular value kept): the adjugate's determinant is good to
1e-5 (its bound on |det|), the sweeps work on A^T A, whose smallest eigenvalue carries a few
roundings of the largest, 16 x 1.1e-16 c^2 at a kept condition of c.  Matrices within 1 % of
the cut-off are left out: there the sweeps' rounding may decide either way."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SOURCE = """
#include "sph_math.cuh"
__global__ void k(int n, const float* A, const float* b, double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float a[3][3], r[3];
  for (int q = 0; q < 9; ++q) a[q / 3][q % 3] = A[9 * i + q];
  for (int q = 0; q < 3; ++q) r[q] = b[3 * i + q];
  double s[3];
  sph::pinv3_solve(a, r, s);
  for (int q = 0; q < 3; ++q) x[3 * i + q] = s[q];
}
extern "C" int solve(int n, const void* A, const void* b, void* x) {
  k<<<(n + 127) / 128, 128>>>(n, (const float*)A, (const float*)b, (double*)x);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def solve(cuda, tmp_path_factory):
    from pytorchsph_gb300 import build
    d = tmp_path_factory.mktemp("pinv3")
    (d / "pinv3.cu").write_text(SOURCE)
    out = str(d / "pinv3.so")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-shared",
                    *build.ARCH, "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include"), str(d / "pinv3.cu"),
                    os.path.join(build.OUT_DIR, "scan_sort.o"), "-o", out], check=True)
    lib = ctypes.CDLL(out)

    def run(A, b):
        dA, db = torch.from_numpy(A).to(cuda).contiguous(), torch.from_numpy(b).to(cuda).contiguous()
        x = torch.empty((len(A), 3), dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        assert lib.solve(len(A), p(dA), p(db), p(x)) == 0
        return x.cpu().numpy()
    return run


def matrices(n, scale, seed):
    """Random float32 matrices scale x U diag(1, s2, s3) V^T, s3 from 1 to 1e-7, s2 = 1, sqrt(s3) or s3."""
    rng = np.random.default_rng(seed)
    U, V = (np.linalg.qr(rng.normal(size=(n, 3, 3)))[0] for _ in range(2))
    s3 = 10.0 ** -rng.uniform(0, 7, n)
    s2 = np.choose(np.arange(n) % 3, [np.ones(n), np.sqrt(s3), s3])
    A = (U * np.stack([np.ones(n), s2, s3], 1)[:, None]) @ np.swapaxes(V, 1, 2) * scale
    return A.astype(np.float32), rng.normal(size=(n, 3)).astype(np.float32)


def check(A, b, x):
    cut = 3 * np.finfo(np.float32).eps
    A64 = A.astype(np.float64)
    s = np.linalg.svd(A64, compute_uv=False)
    ratio = s / s[:, :1]
    clear = (np.abs(ratio / cut - 1) > 0.01).all(1)
    want = np.stack([np.linalg.pinv(m, rcond=cut) @ r for m, r in zip(A64, b.astype(np.float64))])
    kept = np.where(ratio > cut, s, np.inf).min(1)
    c = s[:, 0] / kept
    err = np.linalg.norm(x - want, axis=1) / (np.linalg.norm(b, axis=1) / kept)
    assert (err <= 1e-5 + 16 * 1.1e-16 * c * c)[clear].all(), (err[clear].max(), c[clear][err[clear].argmax()])
    return s[clear, 0] / np.maximum(s[clear, 2], 1e-300)


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e12])
def test_conditions(solve, scale):
    A, b = matrices(12000, scale, 1)
    cond = check(A, b, solve(A, b))
    for lo, hi in ((1, 1e3), (1e3, 1e5), (1e5, 2.5e6), (2.5e6, 2.79e6), (2.9e6, 1e9)):
        assert ((cond > lo) & (cond < hi)).sum() >= 20, (lo, hi)


def test_singular(solve):
    """Rank 2, rank 1 and zero: exact in small integers."""
    rng = np.random.default_rng(2)
    u, v = rng.integers(-8, 9, (2, 300, 3, 2))
    A = (u @ np.swapaxes(v, 1, 2)).astype(np.float32)
    A[::5] = (u[::5, :, :1] @ np.swapaxes(v[::5, :, :1], 1, 2)).astype(np.float32)
    A[0] = 0
    b = rng.normal(size=(300, 3)).astype(np.float32)
    live = np.linalg.norm(A, axis=(1, 2)) > 0
    x = solve(A, b)
    assert np.isfinite(x).all() and not x[~live].any()
    check(A[live], b[live], x[live])
