"""The reciprocal and the root of the stabilization's panel kernels
(csrc/z2_blocked.cuh rcp_newton, sqrt_rcp), and the panel QR on columns whose
squares leave the range of a double.

Error bounds, u = 2^-53 (the hardware's approximations are good to 2^-20):
  rcp_newton  one rounding of r (1 + e), r's own error squared twice: 1.01 u
  sqrt_rcp    nb: t = q y is rounded once, which the step halves (u / 2), the
              last fma once (u), the series stops at 5 e^3 / 16 with |e| < 2^-19
              (0.02 u): 1.55 u
              g: al nb <= q, so nb's error counts half (0.78 u), d = q + al nb
              once (u), the last fma once (u), the series stops at f^3 with
              |f| < 1.5 2^-19 (0.22 u): 3 u
QR: columns are backward stable one by one, 32 N u of a column's norm, and the
orthogonal factor is orthogonal to 32 N u."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from z2_gauge_zfy_b200 import Chain, Z2Batch

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "z2_gauge_zfy_b200", "csrc")
SRC = """
#include "z2_blocked.cuh"
__global__ void probe(int n, const double *x, const double *q, const double *al, double *r, double *nb,
                      double *g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = rcp_newton(x[i]);
  sqrt_rcp(q[i], al[i], nb[i], g[i]);
}
extern "C" int run(int n, const double *x, const double *q, const double *al, double *r, double *nb,
                   double *g) {
  probe<<<(n + 255) / 256, 256>>>(n, x, q, al, r, nb, g);
  return (int)cudaDeviceSynchronize();
}
"""


def test_reciprocal_and_root_to_rounding(tmp_path):
    torch = pytest.importorskip("torch")
    from z2_gauge_zfy_b200.build import ARCH, nvcc
    src, so = tmp_path / "p.cu", tmp_path / "p.so"
    src.write_text(SRC)
    subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-diag-suppress", "177", "-I", CSRC, "-o", str(so), str(src)], check=True)
    rng = np.random.default_rng(1)
    n = 1 << 20
    m = rng.uniform(1.0, 2.0, n)
    m[:4096] = 1.0 + np.arange(4096) * 2.0 ** -52        # and both ends of a binade
    m[4096:8192] = 2.0 - (1 + np.arange(4096)) * 2.0 ** -52
    x = np.ldexp(m, rng.integers(-1022, 1022, n)) * rng.choice([-1.0, 1.0], n)
    # q = al^2 + ss over the range of exponents the kernels use it in
    ss = np.ldexp(m, rng.integers(-959, 959, n))
    al = np.sqrt(ss) * np.choose(rng.integers(0, 4, n), [np.zeros(n), np.ldexp(1.0, rng.integers(-40, 1, n)),
                                                         rng.uniform(0, 1, n), np.full(n, 1e-160)])
    q = ss + al * al
    dev = [torch.tensor(a, device="cuda") for a in (x, q, al)]
    out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    lib = ctypes.CDLL(str(so))
    assert lib.run(n, *[ctypes.c_void_p(t.data_ptr()) for t in dev + out]) == 0
    r, nb, g = (t.cpu().numpy().astype(np.longdouble) for t in out)
    xl, ql, al_ = (a.astype(np.longdouble) for a in (x, q, al))
    err = lambda v, ref: float(np.max(np.abs(v - ref) / np.abs(ref)))
    root = np.sqrt(ql)
    assert err(r, 1 / xl) <= 1.01 * U
    assert err(nb, root) <= 1.55 * U
    assert err(g, 1 / (ql + al_ * root)) <= 3.0 * U


@pytest.mark.parametrize("Lx,Ly", [(4, 4), (6, 10), (10, 10), (12, 12), (16, 16)])
@pytest.mark.parametrize("powers", [(0,), (-515,), (-530, -300), (511,), (-600,), (600, 520, 300)])
def test_panel_qr_of_columns_beyond_the_squares_range(Lx, Ly, powers):
    N = Lx * Ly
    rng = np.random.default_rng(N)
    A = rng.standard_normal((N, N))
    A /= np.linalg.norm(A, axis=0)
    k = np.array([powers[j % len(powers)] for j in range(N)])
    with Z2Batch([Chain(Nlx=Lx, Nly=Ly, Ltrot=4, beta=0.4, Nwrap=1, seed=3)]) as b:
        b.set_prop(0, UR=np.ldexp(A, k), DR=np.ones(N), VR=np.eye(N))
        b.wrap_pre(0, 1)
        p = b.get_prop(0)
    assert np.max(np.abs(p["UR"].T @ p["UR"] - np.eye(N))) <= 32 * N * U
    # U D V against the columns, both divided by the columns' powers of two
    s = int(k.max())
    got = p["UR"] @ (np.ldexp(p["DR"], -s)[:, None] * np.ldexp(p["VR"], s - k))
    assert np.max(np.linalg.norm(got - A, axis=0)) <= 32 * N * U
