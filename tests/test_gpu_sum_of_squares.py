"""The two-float sum of squares behind the L2 norm of a particle spectrum (common.cuh), compiled on its own, against the
exact sum. With t = RN(s + x^2) and b = RN(t - s), the rounding of b is found exactly (s - (t - b), at most 2^-24 of t) and
x^2 - b, at most 2^-23 of t, is rounded by 2^-24 of itself; adding the two rounds by 1.5 2^-47 of t, and the running sum of
these small parts, at most 1.5 k 2^-23 of the whole after k squares, by 2^-24 of itself each time. Together
n (n + 3) 2^-47 of the sum after n squares. A sum that loses the rounding of b is off by up to 2^-24. Adding the two
halves' small parts, 3 n 2^-24 of the whole at most, rounds by 2^-24 of that twice: 8 n 2^-47 covers it."""
import ctypes as C
import math
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.build_native import ARCH, SRC, cuda_home  # noqa: E402

SOURCE = r"""
#include "common.cuh"
__global__ void sums(const float2* x, float4* out, double* total, int lanes, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= lanes) return;
  float2 s = make_float2(0.f, 0.f), c = s;
  for (int k = 0; k < n; ++k) add_squares(x[(size_t)k * lanes + i], s, c);
  out[i] = make_float4(s.x, s.y, c.x, c.y);
  total[i] = squares_total(s, c);
}
extern "C" int run(const void* x, void* out, void* total, int lanes, int n, void* st) {
  sums<<<(lanes + 127) / 128, 128, 0, (cudaStream_t)st>>>((const float2*)x, (float4*)out, (double*)total, lanes, n);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("sums")
    (d / "sums.cu").write_text(SOURCE)
    r = subprocess.run([str(cuda_home() / "bin" / "nvcc"), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        "-cudart", "shared", "-I", str(SRC), "-o", str(d / "libsums.so"), str(d / "sums.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = C.CDLL(str(d / "libsums.so")).run
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    return fn


def _terms(kind, rng, n, lanes):
    x = rng.standard_normal((n, lanes, 2))
    k = np.arange(n)[:, None, None]
    if kind == "growing":  # every square exceeds the sum before it
        x = np.exp2(0.75 * (k - n / 2)) * (1.0 + 0.2 * np.abs(x))
    elif kind == "shrinking":
        x *= np.exp2(-0.75 * k)
    elif kind == "late":  # a zero frequency that comes last
        x[-1] *= 3e4
    elif kind == "early":
        x[0] *= 3e4
    elif kind == "ties":
        x = np.exp2(rng.integers(-6, 7, x.shape))
    return x.astype(np.float32)


@pytest.mark.parametrize("kind", ["plain", "growing", "shrinking", "late", "early", "ties"])
@pytest.mark.parametrize("n", [1, 2, 33, 65])
def test_sum_is_held_in_two_floats(run, kind, n):
    lanes = 96
    x = _terms(kind, np.random.default_rng(n), n, lanes)
    dev = torch.from_numpy(x).to("cuda:0")
    out = torch.empty(lanes, 4, device="cuda:0")
    total = torch.empty(lanes, dtype=torch.float64, device="cuda:0")
    assert run(dev.data_ptr(), out.data_ptr(), total.data_ptr(), lanes, n, torch.cuda.current_stream().cuda_stream) == 0
    got, total = out.cpu().numpy().astype(np.float64), total.cpu().numpy()
    for i in range(lanes):
        both = [float(v) ** 2 for v in x[:, i].ravel()]
        assert abs(total[i] - math.fsum(both)) <= (n * (n + 3) + 8 * n) * 2.0 ** -47 * math.fsum(both)
        for h in range(2):
            terms = [float(v) ** 2 for v in x[:, i, h]]  # exact: 48 bits
            assert abs(math.fsum([got[i, h], got[i, 2 + h]] + [-t for t in terms])) <= n * (n + 3) * 2.0 ** -47 * math.fsum(terms)
