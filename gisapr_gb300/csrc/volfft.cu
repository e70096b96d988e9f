// Volume spectrum for the projector at power-of-two boxes, sm_103a: the
// reference's pad / sinc^2 / fftshift / rfftn / fftshift (v606:1063-1073)
// computed from the box^3 density without materialising the (2N)^3 padded
// volume, written straight into the blocked copy the slice gather reads.
//
// The padded, fftshifted volume holds the density at signed positions
// j = i - N/2 in [-N/2, N/2) along each axis (mod 2N) and zeros elsewhere.
// A length-2N DFT of such a line splits by output parity k = 2m + e into two
// N-point DFTs of the line's N samples, the odd one premultiplied by
// w^j = exp(-i pi j / N):
//     Y(2m + e) = sum_j [u_j w^{e j}] exp(-2 pi i m j / N).
// Three passes, each a batch of four-step warp FFTs (pairplane.cuh) that read
// their lines from global memory into the first codelet and leave their results
// in an output tile:
//   x: the density rows (sinc^2-weighted on load, as the reference filters
//      the padded volume in float32) -> kx in [0, N], written [z][kx][y];
//   y: lines along y -> ky in [0, 2N), written [ky][kx][z];
//   z: lines along z -> kz in [0, 2N), written in the blocked layout:
//      centred (z, y) order, blocks of 2 (z) x 4 (y) x 2 (x) voxels of 128
//      bytes, x padded to N + 2 (the pad column repeats column N).
// The intermediate arrays (N (N+1) N and 2N (N+1) N complex) stay in L2 at
// box 128, where the passes take 20, 17 and 30 us (45 us of memory traffic at
// the copy rate if none of it stayed in L2); at box 256 117, 118 and 234 us
// against 30, 60 and 119. With the lines staged first and every result carried
// through registers into a second staging they took 25, 26 and 41, and 159, 233
// and 331: shared-memory round trips between barriers, not traffic. The x pass is
// bound by the weights (a square root, a sine and a division), so the two voxels
// at N/2 - j and N/2 + j share one (24 -> 20 us, 156 -> 117).
#include "common.cuh"
#include "pairplane.cuh"

namespace {

// A pass with ``W`` warps: every warp transforms fft_lines<N>() lines, the two
// output parities of half as many data lines.
template <int N, int W>
struct Pass {
  static constexpr int G = fft_lines<N>(), lines = W * G / 2, threads = W * 32;
  // Results of parity e, m of data line l in the output tile: lanes that store (16 consecutive m) or that read
  // (8 lines of an even and an odd k) fall on different banks.
  static constexpr int pitch = lines + 1;
  __host__ __device__ static constexpr int parity(int rows) { return (rows * pitch + 7) / 16 * 16 + 8; }
  static constexpr int stage = stage_elems(N, G);
  // complex elements of shared memory: both twiddle tables, the warps' lines, a tile of 2 ``rows``
  __host__ __device__ static constexpr int elems(int rows) { return 2 * N + W * stage + 2 * parity(rows); }
};

// The twiddles of the N-point transforms and, at position n = j mod N, w^j.
template <int N>
__device__ __forceinline__ void vf_tables(const float2* __restrict__ tw, float2* s_tw, float2* s_w) {
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
    s_tw[t] = tw_full<-1>(tw, twiddle_exponent<N>(t), N);
    s_w[t] = tw_full<-1>(tw, t < N / 2 ? t : t - N, 2 * N);
  }
}

// The two complex products with their roundings spelled out: the templates' zero
// frequency keeps its amplitude through the whitening, and a rounding of it that
// falls the other way shows in a whole column of a template.
__device__ __forceinline__ float2 mul_parity(float2 a, float2 w) {
  return make_float2(fmaf(a.x, w.x, -__fmul_rn(a.y, w.y)), fmaf(a.x, w.y, __fmul_rn(a.y, w.x)));
}
struct MulTwiddle {
  __device__ __forceinline__ float2 operator()(float2 a, float2 w) const {
    return make_float2(fmaf(a.x, w.x, -__fmul_rn(a.y, w.y)), fmaf(a.y, w.x, __fmul_rn(a.x, w.y)));
  }
};

// One warp's lines: ``load(q, i)`` is sample i of its data line q, results m of
// parity e of line q go to ``out(e, m, q, value)``.
template <int N, class Load, class Out>
__device__ __forceinline__ void vf_lines(float2* stage, const float2* s_tw, const float2* s_w, const Load& load,
                                         const Out& out) {
  line_fft_warp<N, -1>(
      StagedLines<N>{stage}, s_tw,
      [&](int g, int n) {
        const float2 u = load(g >> 1, (n + N / 2) & (N - 1)), v = mul_parity(u, s_w[n]);
        return g & 1 ? v : u;
      },
      [&](int g, int m, float2 v) { out(g & 1, m, g >> 1, v); }, MulTwiddle());
}

// x and y passes
template <int N>
using PassXY = Pass<N, N == 256 ? 8 : 4>;

// x pass: CTA = one z plane and a band of rows. Output A1[z][kx][y], kx in [0, N].
template <int N>
__global__ void __launch_bounds__(PassXY<N>::threads) vfft_x(const float* __restrict__ vol, float2* __restrict__ a1,
                                                              const float2* __restrict__ tw_g) {
  using V = PassXY<N>;
  constexpr int m = 2 * N, W = N + 1, R = V::lines, D = V::G / 2, E = V::parity(N / 2 + 1);
  extern __shared__ float2 s_vf[];
  __shared__ float s_row[R][N];
  float2 *s_tw = s_vf, *s_w = s_tw + N, *s_line = s_w + N, *s_out = s_line + (V::threads / 32) * V::stage;
  constexpr int half = N / 2;
  const int warp = threadIdx.x >> 5;
  const int z = blockIdx.y, y0 = blockIdx.x * R;
  const float fz = fftfreq_shifted_f32(z + half, m);
  // the weight at x = N/2 - j and N/2 + j is the same
  for (int idx = threadIdx.x; idx < R * (half + 1); idx += blockDim.x) {
    const int q = idx / (half + 1), j = idx % (half + 1), y = y0 + q;
    const float fy = fftfreq_shifted_f32(y + half, m), fx = fftfreq_shifted_f32(N - j, m);
    const float w = sinc2_f32(__fmul_rn(fz, fz), __fmul_rn(fy, fy), __fmul_rn(fx, fx));
    const float* row = vol + ((size_t)z * N + y) * N;
    s_row[q][half - j] = __fmul_rn(__ldg(row + half - j), w);
    if (j > 0 && j < half) s_row[q][half + j] = __fmul_rn(__ldg(row + half + j), w);
  }
  vf_tables<N>(tw_g, s_tw, s_w);
  __syncthreads();
  vf_lines<N>(
      s_line + warp * V::stage, s_tw, s_w, [&](int q, int i) { return make_float2(s_row[warp * D + q][i], 0.f); },
      [&](int e, int k, int q, float2 v) {
        if (2 * k + e <= N) s_out[e * E + k * V::pitch + warp * D + q] = v;
      });
  __syncthreads();
  for (int idx = threadIdx.x; idx < W * R; idx += blockDim.x) {
    const int k = idx / R, r = idx - k * R;
    a1[((size_t)z * W + k) * N + y0 + r] = s_out[(k & 1) * E + (k >> 1) * V::pitch + r];
  }
}

// y pass: CTA = one kx and a band of z; lines along y. Output
// A2[ky][kx][z], ky in [0, 2N) (unshifted).
template <int N>
__global__ void __launch_bounds__(PassXY<N>::threads) vfft_y(const float2* __restrict__ a1, float2* __restrict__ a2,
                                                              const float2* __restrict__ tw_g) {
  using V = PassXY<N>;
  constexpr int m = 2 * N, W = N + 1, R = V::lines, D = V::G / 2, E = V::parity(N);
  extern __shared__ float2 s_vf[];
  float2 *s_tw = s_vf, *s_w = s_tw + N, *s_line = s_w + N, *s_out = s_line + (V::threads / 32) * V::stage;
  const int warp = threadIdx.x >> 5;
  const int kx = blockIdx.x, z0 = blockIdx.y * R;
  vf_tables<N>(tw_g, s_tw, s_w);
  __syncthreads();
  vf_lines<N>(
      s_line + warp * V::stage, s_tw, s_w,
      [&](int q, int i) { return __ldg(a1 + ((size_t)(z0 + warp * D + q) * W + kx) * N + i); },
      [&](int e, int k, int q, float2 v) { s_out[e * E + k * V::pitch + warp * D + q] = v; });
  __syncthreads();
  for (int idx = threadIdx.x; idx < m * R; idx += blockDim.x) {
    const int k = idx / R, r = idx - k * R;
    a2[((size_t)k * W + kx) * N + z0 + r] = s_out[(k & 1) * E + (k >> 1) * V::pitch + r];
  }
}

// Blocked layout of the slice gather (project.cu): 2 (z) x 4 (y) x 2 (x)
// voxels per 128-byte block, centred (z, y) order, x padded to N + 2.
constexpr int kBZ = 2, kBY = 4, kBX = 2, kBE = kBZ * kBY * kBX;

// z pass: eight data lines
template <int N>
using PassZ = Pass<N, 16 / fft_lines<N>()>;

// z pass: CTA = 4 centred y (one block row) x 2 kx. Writes whole 128-byte
// blocks of the blocked copy.
template <int N>
__global__ void __launch_bounds__(PassZ<N>::threads) vfft_z(const float2* __restrict__ a2, float2* __restrict__ blocked,
                                                             const float2* __restrict__ tw_g) {
  using V = PassZ<N>;
  constexpr int m = 2 * N, W = N + 1, XB = (N + 2) / 2, YB = m / kBY, D = V::G / 2, E = V::parity(N);
  static_assert(V::lines == 8, "eight (y, x) lines per CTA");
  extern __shared__ float2 s_vf[];
  float2 *s_tw = s_vf, *s_w = s_tw + N, *s_line = s_w + N, *s_out = s_line + (V::threads / 32) * V::stage;
  const int warp = threadIdx.x >> 5;
  const int yb = blockIdx.y, xb = blockIdx.x;
  vf_tables<N>(tw_g, s_tw, s_w);
  __syncthreads();
  // line l = 2 * (yc - 4 yb) + (x - 2 xb)
  vf_lines<N>(
      s_line + warp * V::stage, s_tw, s_w,
      [&](int q, int i) {
        const int l = warp * D + q;
        const int yc = kBY * yb + (l >> 1), kx = min(kBX * xb + (l & 1), W - 1);  // the pad column repeats N
        const int ky = yc < N ? yc + N : yc - N;                                  // centred -> unshifted
        return __ldg(a2 + ((size_t)ky * W + kx) * N + i);
      },
      [&](int e, int k, int q, float2 v) { s_out[e * E + k * V::pitch + warp * D + q] = v; });
  __syncthreads();
  // block (zb, yb, xb) element ((zc % 2) * 4 + yc % 4) * 2 + x % 2
  for (int idx = threadIdx.x; idx < m * 8; idx += blockDim.x) {
    const int zc = idx >> 3, l = idx & 7, k = zc < N ? zc + N : zc - N;  // centred -> unshifted kz
    blocked[(((size_t)(zc / kBZ) * YB + yb) * XB + xb) * kBE + (zc % kBZ) * 8 + l] =
        s_out[(k & 1) * E + (k >> 1) * V::pitch + l];
  }
}

template <class Kernel, class... Args>
cudaError_t launch_pass(Kernel kernel, SmemLimit& limit, dim3 grid, int threads, int elems, cudaStream_t st,
                        Args... args) {
  const size_t smem = elems * sizeof(float2);
  const cudaError_t e = allow_smem(kernel, smem, limit);
  if (e != cudaSuccess) return e;
  kernel<<<grid, threads, smem, st>>>(args...);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_vfft(cudaStream_t st, const float* vol, float2* a1, float2* a2, float2* blocked,
                        const float2* tw) {
  using V = PassXY<N>;
  using Z = PassZ<N>;
  static_assert(N % V::lines == 0, "row bands tile the box");
  static SmemLimit lx, ly, lz;
  cudaError_t e = launch_pass(vfft_x<N>, lx, dim3(N / V::lines, N), V::threads, V::elems(N / 2 + 1), st, vol, a1, tw);
  if (e != cudaSuccess) return e;
  e = launch_pass(vfft_y<N>, ly, dim3(N + 1, N / V::lines), V::threads, V::elems(N), st, a1, a2, tw);
  if (e != cudaSuccess) return e;
  return launch_pass(vfft_z<N>, lz, dim3((N + 2) / 2, 2 * N / 4), Z::threads, Z::elems(N), st, a2, blocked, tw);
}

}  // namespace

// complex elements of the two intermediate arrays (x pass, y pass)
size_t vfft_scratch_elems(int N) { return (size_t)N * (N + 1) * N + (size_t)2 * N * (N + 1) * N; }

cudaError_t launch_volume_spectrum_blocked(cudaStream_t st, const float* vol, int N, float2* scratch,
                                           float2* blocked, const float2* tw) {
  float2* a1 = scratch;
  float2* a2 = scratch + (size_t)N * (N + 1) * N;
  switch (N) {
    case 32: return launch_vfft<32>(st, vol, a1, a2, blocked, tw);
    case 64: return launch_vfft<64>(st, vol, a1, a2, blocked, tw);
    case 128: return launch_vfft<128>(st, vol, a1, a2, blocked, tw);
    case 256: return launch_vfft<256>(st, vol, a1, a2, blocked, tw);
    default: return cudaErrorInvalidValue;
  }
}
