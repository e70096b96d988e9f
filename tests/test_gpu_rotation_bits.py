"""The particle preparation's packed rotation (rotate.cuh), compiled on its own, against the same coordinate chain and
bilinear sum in scalar operations that round one by one: the same bits at every pixel, staged with its border and not,
for angles over the whole circle and offsets that move the image partly and wholly out of its frame."""
import ctypes as C
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from gisapr_gb300.build_native import ARCH, SRC, cuda_home  # noqa: E402

SOURCE = r"""
#include "rotate.cuh"
__device__ float scalar_pixel(const float* img, int N, float4 ps, int i, int j) {
  const float yy = (float)i, xx = (float)j, nm1 = (float)(N - 1), half = __fdiv_rn(nm1, 2.0f);
  const float sy = __fadd_rn(__fmaf_rn(-ps.y, xx, __fmul_rn(ps.x, yy)), ps.z);
  const float sx = __fadd_rn(__fmaf_rn(ps.x, xx, __fmul_rn(ps.y, yy)), ps.w);
  const float yn = __fsub_rn(__fdiv_rn(__fmul_rn(2.0f, sy), nm1), 1.0f);
  const float xn = __fsub_rn(__fdiv_rn(__fmul_rn(2.0f, sx), nm1), 1.0f);
  const float iy = __fmul_rn(__fadd_rn(yn, 1.0f), half), ix = __fmul_rn(__fadd_rn(xn, 1.0f), half);
  const float fy = floorf(iy), fx = floorf(ix);
  const float w = __fsub_rn(ix, fx), e = __fsub_rn(1.0f, w), n = __fsub_rn(iy, fy), s = __fsub_rn(1.0f, n);
  auto at = [&](float y, float x) {
    return y >= 0.f && y < (float)N && x >= 0.f && x < (float)N ? img[(int)y * N + (int)x] : 0.f;
  };
  float v = __fmul_rn(at(fy, fx), __fmul_rn(s, e));
  v = __fadd_rn(v, __fmul_rn(at(fy, fx + 1.f), __fmul_rn(s, w)));
  v = __fadd_rn(v, __fmul_rn(at(fy + 1.f, fx), __fmul_rn(n, e)));
  return __fadd_rn(v, __fmul_rn(at(fy + 1.f, fx + 1.f), __fmul_rn(n, w)));
}
template <int N>
__global__ void rotate(const float* img, const float* staged, const float4* table, float* out) {
  const float4 ps = table[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x, q = t / N, j = t % N;
  if (q >= N / 2) return;
  float* o = out + (size_t)blockIdx.y * 3 * N * N;
  const float2 a = rotated_pair<N, true>(staged, ps, q, j), b = rotated_pair<N, false>(img, ps, q, j);
  for (int r = 0; r < 2; ++r) {
    const int at = (2 * q + r) * N + j;
    o[at] = r ? a.y : a.x;
    o[N * N + at] = r ? b.y : b.x;
    o[2 * N * N + at] = scalar_pixel(img, N, ps, 2 * q + r, j);
  }
}
extern "C" int image_stride(int N) { return N == 32 ? image_ld<32>() : (N == 64 ? image_ld<64>() : (N == 96 ? image_ld<96>() : image_ld<128>())); }
extern "C" int border() { return kBorder; }
extern "C" int run(int N, const void* img, const void* staged, const void* table, int n, void* out, void* st) {
  const dim3 grid(N * N / 2 / 128, n);
  auto go = [&](auto kernel) {
    kernel<<<grid, 128, 0, (cudaStream_t)st>>>((const float*)img, (const float*)staged, (const float4*)table, (float*)out);
  };
  if (N == 32) go(rotate<32>);
  else if (N == 64) go(rotate<64>);
  else if (N == 96) go(rotate<96>);
  else go(rotate<128>);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("rotation")
    (d / "rotation.cu").write_text(SOURCE)
    r = subprocess.run([str(cuda_home() / "bin" / "nvcc"), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        "-cudart", "shared", "-I", str(SRC), "-o", str(d / "librotation.so"), str(d / "rotation.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    so = C.CDLL(str(d / "librotation.so"))
    so.run.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    return so


@pytest.mark.parametrize("N", [32, 64, 96, 128])
def test_bits_of_the_scalar_chain(lib, N):
    rng = np.random.default_rng(N)
    angles = np.concatenate([np.arange(0.0, 360.0, 7.5), rng.uniform(0, 360, 48)])
    c, s = np.cos(np.deg2rad(angles)), np.sin(np.deg2rad(angles))
    centre = (N - 1) / 2 + rng.choice([0.0, 0.5, 0.3 * N, 2.0 * N], len(angles))
    table = np.stack([c, s, centre - c * centre + s * centre, centre - s * centre - c * centre], 1).astype(np.float32)
    image = rng.standard_normal((N, N)).astype(np.float32)
    ld, b = lib.image_stride(N), lib.border()
    staged = np.zeros((N + 2 * b, ld), np.float32)
    staged[b:b + N, b:b + N] = image
    dev = [torch.from_numpy(v).to("cuda:0") for v in (image, staged, table)]
    out = torch.empty(len(angles), 3, N, N, device="cuda:0")
    assert lib.run(N, *(v.data_ptr() for v in dev), len(angles), out.data_ptr(),
                   torch.cuda.current_stream().cuda_stream) == 0
    assert bool((out[:, 2] != 0).any()) and bool((out[:, 2] == 0).any())
    assert torch.equal(out[:, 1], out[:, 2])
    assert torch.equal(out[:, 0], out[:, 2])
