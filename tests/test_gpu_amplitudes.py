"""The amplitude of a spectrum entry in the particle preparation (sqrt_fp64 of a fused sum of squares, common.cuh),
compiled on its own. The square root is within 2^-52 of the value, so at most one unit from the correctly rounded one.
With u = 2^-53 the sum of squares is within 2 u (two roundings), its root within u of that, the root's own error 2 u:
3 u together, where CUDA states 2 ulp, 4 u at the worst, for hypot."""
import ctypes as C
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.build_native import ARCH, SRC, cuda_home  # noqa: E402

SOURCE = r"""
#include "common.cuh"
__global__ void roots(const double* x, const double* y, double* root, double* amplitude, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  root[i] = sqrt_fp64(x[i] * x[i]);
  amplitude[i] = sqrt_fp64(fma(x[i], x[i], y[i] * y[i]));
}
__global__ void plain(const double* e, double* root, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) root[i] = sqrt_fp64(e[i]);
}
extern "C" int run(const void* x, const void* y, void* root, void* amplitude, int n, void* st) {
  roots<<<(n + 255) / 256, 256, 0, (cudaStream_t)st>>>((const double*)x, (const double*)y, (double*)root,
                                                       (double*)amplitude, n);
  return (int)cudaGetLastError();
}
extern "C" int run_plain(const void* e, void* root, int n, void* st) {
  plain<<<(n + 255) / 256, 256, 0, (cudaStream_t)st>>>((const double*)e, (double*)root, n);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("roots")
    (d / "roots.cu").write_text(SOURCE)
    r = subprocess.run([str(cuda_home() / "bin" / "nvcc"), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        "-cudart", "shared", "-I", str(SRC), "-o", str(d / "libroots.so"), str(d / "roots.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    so = C.CDLL(str(d / "libroots.so"))
    so.run.argtypes = [C.c_void_p] * 4 + [C.c_int, C.c_void_p]
    so.run_plain.argtypes = [C.c_void_p] * 2 + [C.c_int, C.c_void_p]
    return so


def _stream():
    return torch.cuda.current_stream().cuda_stream


def test_square_root_is_within_one_unit(lib):
    rng = np.random.default_rng(1)
    n = 1 << 20
    e = np.concatenate([np.exp2(rng.uniform(-1021, 1023, n)), rng.uniform(1, 4, n),  # normal values
                        (np.arange(1, 4097) / 64.0) ** 2, np.nextafter((np.arange(1, 4097) / 64.0) ** 2, 0),
                        [1.0, 2.0, np.nextafter(1.0, 2), np.nextafter(4.0, 0), np.finfo(np.float64).tiny]])
    dev = torch.from_numpy(e).to("cuda:0")
    out = torch.empty_like(dev)
    assert lib.run_plain(dev.data_ptr(), out.data_ptr(), len(e), _stream()) == 0
    want = np.sqrt(e)
    assert (np.abs(out.cpu().numpy() - want) <= np.spacing(want)).all()
    for special in (0.0, -0.0, np.nan):
        dev = torch.full((1,), special, dtype=torch.float64, device="cuda:0")
        out = torch.ones_like(dev)
        assert lib.run_plain(dev.data_ptr(), out.data_ptr(), 1, _stream()) == 0
        assert np.array_equal(out.cpu().numpy(), [special], equal_nan=True)


def test_amplitudes(lib):
    """Over the values of float32 images' spectra: amplitudes from 1e-40 to 1e43, either part the larger or zero."""
    rng = np.random.default_rng(2)
    n = 1 << 18
    size = np.exp2(rng.uniform(-130, 140, n))
    angle = rng.uniform(0, 2 * np.pi, n)
    x, y = size * np.cos(angle), size * np.sin(angle) * np.exp2(-rng.integers(0, 40, n) * (rng.random(n) < 0.3))
    y[::97] = 0.0
    dev = [torch.from_numpy(v).to("cuda:0") for v in (x, y)]
    root, amplitude = torch.empty_like(dev[0]), torch.empty_like(dev[0])
    assert lib.run(dev[0].data_ptr(), dev[1].data_ptr(), root.data_ptr(), amplitude.data_ptr(), n, _stream()) == 0
    wide = np.longdouble
    want = np.sqrt(x.astype(wide) ** 2 + y.astype(wide) ** 2)
    # the comparison's own rounding is 2^-63 at the most (80 or 128 bits)
    assert float(np.max(np.abs(amplitude.cpu().numpy().astype(wide) - want) / want)) <= 3 * 2.0 ** -53 + 2.0 ** -62
    assert float(np.max(np.abs(root.cpu().numpy() - np.abs(x)) / np.abs(x))) <= 3 * 2.0 ** -53
