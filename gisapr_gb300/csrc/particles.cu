// Packed CTF*ISSPA table and particle spectra (v606:695-829, 1193-1374).
//
// packed_ctf: one thread per packed coefficient of one particle. The static
// frequency terms (x, y, u^4, ISSPA noise curve) are host tables built with
// the reference's float32 numpy expressions; the per-particle trigonometry
// and the phase gamma repeat the reference's float32 operation order without
// fused multiply-add, because gamma reaches hundreds of radians and a single
// rounding difference moves sin(gamma) by ~1e-5.
//
// prepare_plane (boxes up to 192): the rotated image (bilinear, zero padding,
// align_corners=True, in the weight order of torch's vectorised 2-D CPU kernel)
// is masked and transformed in one shared-memory plane; the packed half plane
// is Fourier-cropped, multiplied by the CTF table, conjugated, L2-normalised
// and written pre-shifted. prepare_particles does the same for box 256, whose
// plane does not fit an SM, through a global scratch plane.
#include "common.cuh"
#include "pairplane.cuh"
#include "rotate.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kRowBatch = 8;
constexpr int kColBatch = 16;

struct CtfConst {
  float k1, k2, k3, k5, kk;
};

__global__ void packed_ctf(const float* __restrict__ dfu, const float* __restrict__ dfv,
                           const float* __restrict__ dfa, int n, const float* __restrict__ tx,
                           const float* __restrict__ ty, const float* __restrict__ tu4,
                           const float* __restrict__ tnc, int K, CtfConst c,
                           float* __restrict__ out) {
  const int p = blockIdx.y;
  if (p >= n) return;
  // angle = deg2rad(dfa) in float32: dfa * float(pi/180)
  const float ang = __fmul_rn(dfa[p], (float)(3.14159265358979323846 / 180.0));
  const float sa = sinf(ang), ca = cosf(ang);
  const float u = dfu[p], v = dfv[p];
  const float axx = __fsub_rn(__fmul_rn(__fmul_rn(-u, ca), ca), __fmul_rn(__fmul_rn(v, sa), sa));
  const float ayy = __fsub_rn(__fmul_rn(__fmul_rn(-u, sa), sa), __fmul_rn(__fmul_rn(v, ca), ca));
  const float axy = __fadd_rn(__fmul_rn(__fmul_rn(-u, sa), ca), __fmul_rn(__fmul_rn(v, sa), ca));
  const float axy2 = __fmul_rn(2.0f, axy);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
    const float x = tx[k], y = ty[k];
    const float t1 = __fmul_rn(__fmul_rn(axx, x), x);
    const float t2 = __fmul_rn(__fmul_rn(axy2, x), y);
    const float t3 = __fmul_rn(__fmul_rn(ayy, y), y);
    const float s = __fadd_rn(__fadd_rn(t1, t2), t3);
    float g = __fmul_rn(c.k1, s);
    g = __fadd_rn(g, __fmul_rn(c.k2, tu4[k]));
    g = __fsub_rn(g, c.k5);
    g = __fsub_rn(g, c.k3);
    float val = -sinf(g);
    if (fabsf(val) < 1e-8f) val = (val > 0.f) ? 1e-8f : ((val < 0.f) ? -1e-8f : 0.f);
    const float den = __fadd_rn(tnc[k], __fmul_rn(__fmul_rn(c.kk, val), val));
    const float w = __fmul_rn(val, sqrtf(__frcp_rn(den)));
    out[(size_t)p * K + k] = w;
  }
}

struct PrepParams {
  const float* images;     // [n][N][N]
  const int* psi_index;    // [n][n_psi] index into psi table
  const float4* psi_tab;   // (cos, sin, off_row, off_col) float32 per psi angle
  const float* mask;       // [N][N] or null
  const float* ctf;        // [n][nb][H]
  float2* out;             // [n][n_psi][nb][H]
  float2* scratch;
  size_t scratch_stride;
  const float2* tw;
  const float2* tw3;       // twiddles of lengths 3 * 2^k
  int n, n_psi, N, nb;
};

__global__ void __launch_bounds__(kThreads) prepare_particles(PrepParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = P.N, nb = P.nb, H = nb / 2 + 1, HC = N / 2 + 1;
  float2* sm = reinterpret_cast<float2*>(smem_raw);
  float2* s_tw = sm + max(kRowBatch, kColBatch) * N;
  double* red = reinterpret_cast<double*>(s_tw + kMaxFftLen / 2);
  for (int t = threadIdx.x; t < kMaxFftLen / 2; t += blockDim.x) s_tw[t] = P.tw[t];
  __syncthreads();
  float2* S = P.scratch + (size_t)blockIdx.x * P.scratch_stride;
  float2* Pk = S + (size_t)N * HC;
  const float half = __fdiv_rn((float)(N - 1), 2.0f);
  const float nm1 = (float)(N - 1);
  for (int job = blockIdx.x; job < P.n * P.n_psi; job += gridDim.x) {
    const int p = job / P.n_psi, si = job - p * P.n_psi;
    const float4 ps = P.psi_tab[P.psi_index[(size_t)p * P.n_psi + si]];
    const float cth = ps.x, sth = ps.y;
    const float* img = P.images + (size_t)p * N * N;
    // rows: rotate, mask, forward FFT
    for (int i0 = 0; i0 < N; i0 += kRowBatch) {
      const int nr = min(kRowBatch, N - i0);
      for (int t = threadIdx.x; t < nr * N; t += blockDim.x) {
        const int rl = t / N, j = t - rl * N;
        const float yy = (float)(i0 + rl), xx = (float)j;
        // source = [row, col] @ M^T + offset; M = [[c, -s], [s, c]]
        const float sy = __fadd_rn(__fmaf_rn(-sth, xx, __fmul_rn(cth, yy)), ps.z);
        const float sx = __fadd_rn(__fmaf_rn(cth, xx, __fmul_rn(sth, yy)), ps.w);
        const float yn = __fsub_rn(__fdiv_rn(__fmul_rn(2.0f, sy), nm1), 1.0f);
        const float xn = __fsub_rn(__fdiv_rn(__fmul_rn(2.0f, sx), nm1), 1.0f);
        const float iy = __fmul_rn(__fadd_rn(yn, 1.0f), half);
        const float ix = __fmul_rn(__fadd_rn(xn, 1.0f), half);
        float v = sample_bilinear_zero(img, N, iy, ix);
        if (P.mask != nullptr) v = __fmul_rn(v, P.mask[(size_t)(i0 + rl) * N + j]);
        sm[rl * N + fft_in_pos(j, N)] = make_float2(v, 0.f);
      }
      __syncthreads();
      smem_fft(sm, N, nr, -1.0f, s_tw, P.tw3);
      for (int t = threadIdx.x; t < nr * HC; t += blockDim.x) {
        const int rl = t / HC, k = t - rl * HC;
        S[(size_t)(i0 + rl) * HC + k] = sm[rl * N + k];
      }
      __syncthreads();
    }
    // columns
    for (int c0 = 0; c0 < HC; c0 += kColBatch) {
      const int nc = min(kColBatch, HC - c0);
      for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
        const int r = t / nc, cl = t - r * nc;
        sm[cl * N + fft_in_pos(r, N)] = S[(size_t)r * HC + c0 + cl];
      }
      __syncthreads();
      smem_fft(sm, N, nc, -1.0f, s_tw, P.tw3);
      for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
        const int r = t / nc, cl = t - r * nc;
        S[(size_t)r * HC + c0 + cl] = sm[cl * N + r];
      }
      __syncthreads();
    }
    // crop, pack, CTF, conjugate, norm
    const float* ctf = P.ctf + (size_t)p * nb * H;
    double ss = 0.0;
    for (int t = threadIdx.x; t < nb * H; t += blockDim.x) {
      const int r = t / H, c = t - r * H;
      const int ky = r < nb / 2 ? r : r - nb;
      float2 f;
      if (c < nb / 2) f = S[(size_t)((ky + N) % N) * HC + c];
      else if (nb == N) f = S[(size_t)((ky + N) % N) * HC + N / 2];
      else f = cconj(S[(size_t)((-ky + N) % N) * HC + nb / 2]);
      const float w = ctf[t];
      f = make_float2(__fmul_rn(f.x, w), -__fmul_rn(f.y, w));
      Pk[t] = f;
      ss += (double)f.x * f.x + (double)f.y * f.y;
    }
    ss = block_sum_d(ss, red);
    const float inv = (float)(1.0 / sqrt(ss));
    float2* out = P.out + ((size_t)p * P.n_psi + si) * nb * H;
    for (int t = threadIdx.x; t < nb * H; t += blockDim.x) {
      const int r = t / H, c = t - r * H;
      const int rs = (r + nb / 2) % nb, cs = (c + H / 2) % H;
      out[(size_t)rs * H + cs] = cscale(Pk[t], inv);
    }
    __syncthreads();
  }
}


// ---------------------------------------------------------------------------
// Boxes 32 to 192: one image per CTA and pass, all of it in shared memory.
//
// The image is rotated straight into the pair plane (pairplane.cuh), so a
// spectrum costs one write and one read of the plane per FFT step and one
// write to HBM, against the block-wide radix-2 transforms through a global
// scratch plane that prepare_particles runs (box 128: each of 14 stages a pass
// over shared memory with a block barrier, and three passes over the scratch).
// Measured on GB300, 2,000 particles of box 128 at three angles: 2.51 -> 0.75 ms
// (597 MB of images, weights and spectra, 0.8 TB/s). What bounds it now is issue
// and latency at 16 warps an SM: about 35 packed instructions a pixel for the
// float32 coordinate chain and the bilinear sum, and the FFT codelets.
//
// Up to box 128 the source image is staged in shared memory, with a border of
// two zero pixels that stands for the zero padding (coordinates are clamped
// into the border), because a rotated footprint touches about ten 128-byte
// lines per warp load, which the L1 serves one a cycle; the row stride of
// N + 9 spreads the footprint over the banks. A CTA takes a contiguous run of
// (particle, psi) jobs, so an image is loaded once for its psi angles; at box
// 128, where one CTA fills the SM, the next image arrives by asynchronous
// copies meanwhile. Box 192 has no room for the image and samples it through L1.
// ---------------------------------------------------------------------------
template <int N>
__host__ __device__ constexpr int prep_threads() { return N <= 64 ? 128 : (N == 96 ? 384 : (N == 128 ? 512 : 768)); }
template <int N>
__host__ __device__ constexpr int prep_images() { return N == 128 ? 2 : (N < 128 ? 1 : 0); }
template <int N>
__host__ __device__ constexpr int image_elems() { return (N + 2 * kBorder) * image_ld<N>(); }

template <int N>
__global__ void __launch_bounds__(prep_threads<N>(), N <= 64 ? 4 : (N == 96 ? 2 : 1)) prepare_plane(PrepParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT = prep_threads<N>(), NW = NT / 32, G = fft_lines<N>(), NI = prep_images<N>();
  constexpr int ILD = image_ld<N>(), IEL = image_elems<N>();
  float2* plane = reinterpret_cast<float2*>(smem_raw);
  float2* s_tw = plane + pair_elems(N);
  float2* s_last = s_tw + N;                              // [N] the Nyquist column, then packed column nb / 2
  double* red = reinterpret_cast<double*>(s_last + N);    // [NW + 1]
  float* s_img = reinterpret_cast<float*>(red + NW + 1);  // [NI][IEL]
  const PairPlane<N> Z{plane};
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = P.nb, H = nb / 2 + 1;
  for (int t = tid; t < N; t += NT) s_tw[t] = twiddle_of<N>(P.tw, P.tw3, twiddle_exponent<N>(t));
  for (int t = tid; t < NI * IEL; t += NT) s_img[t] = 0.f;  // the border stays zero
  const long long jobs = (long long)P.n * P.n_psi;
  const int j0 = (int)(jobs * blockIdx.x / gridDim.x), j1 = (int)(jobs * (blockIdx.x + 1) / gridDim.x);
  // the images of particles p0 .. p1 go to the buffers in turn
  const int p0 = j0 / P.n_psi, p1 = j1 > j0 ? (j1 - 1) / P.n_psi : p0 - 1;
  auto load_image = [&](int p) {
    if constexpr (NI > 0) {
      float* dst = s_img + ((p - p0) % NI) * IEL + kBorder * ILD + kBorder;
      const float* src = P.images + (size_t)p * N * N;
      for (int t = tid; t < N * N; t += NT)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(dst + (t / N) * ILD + t % N)),
                     "l"(src + t)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  __syncthreads();  // the zeroed border before the copies
  if (NI > 0 && p0 <= p1) load_image(p0);
  int ready = p0 - 1;  // the last image that has been waited for
  // lanes take 8 columns x 4 row pairs of the rotated image: a compact footprint
  const int lj = tid & 7, lq = (tid >> 3) & 3;
  constexpr int JT = N / 8, QT = N / 8;  // tiles of 8 columns, of 4 row pairs
  for (int job = j0; job < j1; ++job) {
    const int p = job / P.n_psi, si = job - p * P.n_psi;
    if (NI > 0 && p != ready) {
      if (NI > 1 && p + 1 <= p1) {
        load_image(p + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        if (NI == 1 && p != p0) load_image(p);  // every reader left it at the last barrier
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      ready = p;
      __syncthreads();
    }
    const float4 ps = P.psi_tab[P.psi_index[(size_t)p * P.n_psi + si]];
    const float* img = NI > 0 ? s_img + (NI > 1 ? ((p - p0) % NI) * IEL : 0) : P.images + (size_t)p * N * N;
#pragma unroll 2
    for (int tile = warp; tile < JT * QT; tile += NW) {
      // the two rows of a pair, as the halves of packed operations
      const int q = (tile / JT) * 4 + lq, j = (tile % JT) * 8 + lj;
      float2 v = rotated_pair<N, (NI > 0)>(img, ps, q, j);
      if (P.mask != nullptr) {
        const float* mk = P.mask + 2 * q * N + j;
        v = mul2(v, make_float2(__ldg(mk), __ldg(mk + N)));
      }
      Z.at(q, j) = v;
    }
    __syncthreads();
    for (int grp = warp; grp < pair_row_groups<N>(); grp += NW) {
      const PairRows<N> R{Z, grp};
      line_fft_warp<N, -1>(R, s_tw);
      pair_split_rows<N>(R);
    }
    __syncthreads();
    for (int grp = warp; grp < pair_col_groups<N>(); grp += NW) {
      line_fft_warp<N, -1>(PairCols<N>{Z, grp * G}, s_tw);
      if (grp == 0) col0_split<N>(Z, s_last);
    }
    __syncthreads();
    // crop, pack, CTF, conjugate: every value is weighted in place (column
    // nb / 2 in s_last) and squared for the norm, then scaled and written
    const float* ctf = P.ctf + (size_t)p * nb * H;
    const int hb = nb / 2;
    float2 hi = make_float2(0.f, 0.f), lo = hi;  // the L2 norm; in FP64 it took as long as the transforms
    for (int r = warp; r < nb; r += NW) {
      const int i = r < hb ? r : r + N - nb;
#pragma unroll 2
      for (int c = lane; c < hb; c += 32) {
        float2& z = Z.half(i, c);
        const float2 f = cscale(cconj(z), __ldg(ctf + r * H + c));
        z = f;
        add_squares(f, hi, lo);
      }
    }
    for (int r = tid; r < nb; r += NT) {
      const int i = r < hb ? r : r + N - nb;
      // cropped: the packed column is the negative frequency -nb / 2, the
      // conjugate of the stored one, and is conjugated once more here
      const float2 z = nb == N ? cconj(s_last[i]) : Z.half(i == 0 ? 0 : N - i, hb);
      const float2 f = cscale(z, __ldg(ctf + r * H + hb));
      s_last[r] = f;
      add_squares(f, hi, lo);
    }
    const double ss = warp_sum_d(squares_total(hi, lo));
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    if (tid == 0) {  // one thread: FP64 division and square root
      double total = 0.0;
      for (int w = 0; w < NW; ++w) total += red[w];
      red[NW] = 1.0 / sqrt(total);
    }
    __syncthreads();
    const float inv = (float)red[NW];
    float2* out = P.out + (size_t)job * nb * H;
    for (int r = warp; r < nb; r += NW) {
      const int i = r < hb ? r : r + N - nb, rs = r < hb ? r + hb : r - hb;
#pragma unroll 2
      for (int c = lane; c <= hb; c += 32) {
        const int cs = c + H / 2 < H ? c + H / 2 : c + H / 2 - H;
        out[rs * H + cs] = cscale(c < hb ? Z.half(i, c) : s_last[r], inv);
      }
    }
    __syncthreads();  // the plane, the image and red are free
  }
}

template <int N>
cudaError_t launch_plane(const PrepParams& P, int sm_count, cudaStream_t st) {
  const size_t smem = (size_t)(pair_elems(N) + 2 * N) * sizeof(float2) + (prep_threads<N>() / 32 + 1) * sizeof(double) +
                      (size_t)prep_images<N>() * image_elems<N>() * sizeof(float);
  static SmemLimit limit;
  const cudaError_t e = allow_smem(prepare_plane<N>, smem, limit);
  if (e != cudaSuccess) return e;
  // one CTA per SM at 128 and 192 (the plane and the images fill it), two at
  // 96, five at 64 and as many at 32
  const long long jobs = (long long)P.n * P.n_psi, most = (long long)sm_count * (N >= 128 ? 1 : (N == 96 ? 2 : 5));
  prepare_plane<N><<<(int)(jobs < most ? jobs : most), prep_threads<N>(), smem, st>>>(P);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_packed_ctf(cudaStream_t st, const float* dfu, const float* dfv, const float* dfa,
                              int n, const float* tx, const float* ty, const float* tu4,
                              const float* tnc, int K, float k1, float k2, float k3, float k5,
                              float kk, float* out) {
  if (n <= 0) return cudaSuccess;
  CtfConst c{k1, k2, k3, k5, kk};
  dim3 grid((K + 255) / 256, n);
  packed_ctf<<<grid, 256, 0, st>>>(dfu, dfv, dfa, n, tx, ty, tu4, tnc, K, c, out);
  return cudaGetLastError();
}

// complex elements of one CTA's scratch plane (box 256 only)
size_t prepare_scratch_elems(int N, int nb) {
  return N == 256 ? (size_t)N * (N / 2 + 1) + (size_t)nb * (nb / 2 + 1) : 0;
}

static size_t prepare_smem_bytes(int N) {
  return (size_t)max(kRowBatch, kColBatch) * N * sizeof(float2) + (kMaxFftLen / 2) * sizeof(float2) +
         40 * sizeof(double);
}

// grid: CTAs of the box-256 kernel, one scratch plane each (4 per SM)
cudaError_t launch_prepare_particles(cudaStream_t st, const float* images, int n, int n_psi,
                                     const int* psi_index, const void* psi_tab, const float* mask,
                                     const float* ctf, float2* out, float2* scratch, int grid, int sm_count,
                                     const float2* tw, const float2* tw3, int N, int nb) {
  if (n <= 0) return cudaSuccess;
  PrepParams P;
  P.images = images; P.psi_index = psi_index; P.psi_tab = (const float4*)psi_tab; P.mask = mask;
  P.ctf = ctf; P.out = out; P.scratch = scratch; P.scratch_stride = prepare_scratch_elems(N, nb);
  P.tw = tw; P.tw3 = tw3; P.n = n; P.n_psi = n_psi; P.N = N; P.nb = nb;
  switch (N) {
    case 32: return launch_plane<32>(P, sm_count, st);
    case 64: return launch_plane<64>(P, sm_count, st);
    case 96: return launch_plane<96>(P, sm_count, st);
    case 128: return launch_plane<128>(P, sm_count, st);
    case 192: return launch_plane<192>(P, sm_count, st);
    case 256: break;
    default: return cudaErrorInvalidValue;
  }
  const size_t smem = prepare_smem_bytes(N);
  static SmemLimit limit;
  const cudaError_t e = allow_smem(prepare_particles, smem, limit);
  if (e != cudaSuccess) return e;
  prepare_particles<<<grid, kThreads, smem, st>>>(P);
  return cudaGetLastError();
}
