// Central-slice projector and template tail (v606:856-1147) for sm_103a.
//
// Boxes 32, 64 and 128 (rows_inverse, template_tail): pass A is a kernel of its
// own that writes each template's plane to global memory; a CTA then holds one
// template as a plane of paired real rows in shared memory (pairplane.cuh)
// through passes B to G. General kernel (boxes 96, 192, 256): one CTA builds one
// template at a time (grid-stride over directions). Every 2-D array of a
// template lives in a global scratch plane owned by the CTA; each pass stages a
// batch of rows or columns in shared memory, transforms it there (block-wide
// radix-2/3 FFTs at 96 and 192, four-step warp FFTs at 256) and writes the batch
// back; at box 256 pass A is rows_inverse. The passes are:
//
//   A  slice gather + inverse along rows: trilinear samples of the half
//      volume (border clamp, conjugate where the rotated x < 0) feed two
//      N-point inverse FFTs per column (even/odd rows of the 2N grid); the
//      pair combines into exactly the N centred output rows of the 2N-point
//      inverse that the crop keeps (v606:1099-1130).
//   B  C2R along columns (2N-point real output from N+1 coefficients, via an
//      N-point complex inverse), keep the N centred columns, scale 1/(2N)^2;
//      then the forward row FFT that starts the whitening.
//   C  forward column FFT; radial |F| sums per bin (deterministic warp
//      reductions over a host-built bin list).
//   D  divide by the radial mean amplitude (DC bin untouched), inverse
//      column FFT.
//   E  inverse row transform (real part) of pixels centred on the image
//      mean, float32 plane-fit sums (per thread, then a fixed tree).
//   F  plane removal (the least-squares plane in closed form), population
//      sigma normalisation, soft mask, forward row FFT.
//   G  forward column FFT, Fourier crop and packing, FSC weight, L2 norm
//      over the packed half plane, pre-shift (fftshift both dims) into the
//      template bank (v606:1132-1147, 531-537).
//
// The slice coordinates repeat the reference's float32 operations, including
// the rounding of R00*x + R01*y without fused multiply-add: points where that
// sum cancels sit on the conjugation boundary (v606:881-885), and any other
// rounding there picks the mirrored sample.
#include "common.cuh"
#include "pairplane.cuh"
#include "warpfft.cuh"

namespace {

struct ProjParams {
  const float2* spectrum;   // cuFFT R2C output [2N][2N][N+1], unshifted
  const float* rot;         // [n_dir][9] float32 rotation matrices (stored transposed)
  const int* dirs;          // directions to build (indices into rot), n_build
  int n_build;
  const float* mask;        // [N][N] or null
  const float* fsc;         // [nb][H] packed FSC
  ProjTables t;
  float2* bank;             // [n_dir_out][nb][H] output templates
  const int* out_slot;      // output row in bank for each build index (null => dirs[i])
  float2* scratch;          // per-CTA scratch
  size_t scratch_stride;    // complex elements per CTA
  int* status;              // set to 1 when a plane's bulk-copy wait runs out (or null)
  unsigned wait_limit;      // bound of that wait (attempts)
  const float2* planes;     // pass-A planes written by rows_inverse: [n_build][N][plane_out_ld(N)]
  int N;
  int nb;
};

constexpr int kThreads = 256;
constexpr int kLineCols = 8;   // columns per batch in pass A
constexpr int kRowBatch = 8;   // rows per batch in passes B/E/F
constexpr int kColBatch = 16;  // columns per batch in passes C/D/G

// Trilinear sample of the half volume at clamped voxel coordinates, in the
// corner and weight order of grid_sample's 3-D kernel.
__device__ __forceinline__ float2 sample_trilinear(const float2* __restrict__ vol, int m, int w,
                                                   float iz, float iy, float ix) {
  const float fz = floorf(iz), fy = floorf(iy), fx = floorf(ix);
  const int z0 = (int)fz, y0 = (int)fy, x0 = (int)fx;
  const float wz1 = __fsub_rn(iz, fz), wy1 = __fsub_rn(iy, fy), wx1 = __fsub_rn(ix, fx);
  const float wz0 = __fsub_rn(fz + 1.0f, iz), wy0 = __fsub_rn(fy + 1.0f, iy), wx0 = __fsub_rn(fx + 1.0f, ix);
  float2 acc = make_float2(0.f, 0.f);
  // Half-volume storage is unshifted along z and y: stored index = (i + N) mod 2N.
  const int half = m / 2;
#pragma unroll
  for (int dz = 0; dz < 2; ++dz) {
    const int zz = z0 + dz;
    if (zz >= m) continue;
    const float wz = dz ? wz1 : wz0;
    const int zs = (zz + half) % m;
#pragma unroll
    for (int dy = 0; dy < 2; ++dy) {
      const int yy = y0 + dy;
      if (yy >= m) continue;
      const float wy = dy ? wy1 : wy0;
      const int ys = (yy + half) % m;
      const float2* row = vol + ((size_t)zs * m + ys) * w;
#pragma unroll
      for (int dx = 0; dx < 2; ++dx) {
        const int xx = x0 + dx;
        if (xx >= w) continue;
        const float wx = dx ? wx1 : wx0;
        const float wt = __fmul_rn(__fmul_rn(wx, wy), wz);
        const float2 v = __ldg(row + xx);
        acc.x = __fadd_rn(acc.x, __fmul_rn(v.x, wt));
        acc.y = __fadd_rn(acc.y, __fmul_rn(v.y, wt));
      }
    }
  }
  return acc;
}

// Coordinate of a slice point along one axis, through grid_sample's
// normalise (align_corners=True) and un-normalise, clamped for border mode.
__device__ __forceinline__ float grid_pixel(float c, int size) {
  const float denom = __fsub_rn(__fmul_rn(0.5f, (float)size), 0.5f);
  const float nrm = __fsub_rn(__fdiv_rn(c, denom), 1.0f);
  float pix = __fmul_rn(__fdiv_rn(__fadd_rn(nrm, 1.0f), 2.0f), (float)(size - 1));
  pix = fminf((float)(size - 1), fmaxf(pix, 0.0f));
  return pix;
}

// Hardware square-root approximation (PTX sqrt.approx.f32, relative error
// about 2^-23). Used for the radial |F| sums, whose float32 sums already
// carry larger rounding, and for radial bin indices: rint(sqrt(d2)) of an
// integer d2 <= 2 (N/2)^2 is at least 1/(8 sqrt(d2)) away from a rounding
// boundary, far above the approximation's error, so the bins are exact.
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Deterministic float32 block sums over NW warps (xor tree inside each
// warp, warps added in index order). ``scratch`` holds NW entries; two uses
// of the same scratch must be separated by a block barrier.
template <int NW>
__device__ __forceinline__ float4 block_sum_f4(float4 v, float4* scratch) {
  v.x = warp_sum(v.x); v.y = warp_sum(v.y); v.z = warp_sum(v.z); v.w = warp_sum(v.w);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float4 t = scratch[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) {
    const float4 u = scratch[w];
    t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
  }
  return t;
}
template <int NW>
__device__ __forceinline__ float block_sum_f(float v, float* scratch) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = scratch[0];
#pragma unroll
  for (int w = 1; w < NW; ++w) t += scratch[w];
  return t;
}

// Line batches of the general kernel in shared memory. Box 256 runs its
// 1-D transforms as four-step warp FFTs on padded lines (natural order in
// and out, line stride plane_ld(N), element k at k + k/8), 16 rows per row
// batch; the other boxes use the block-wide radix-2/3 transform on unpadded
// lines, input in fft_in_pos order.
template <int N>
__host__ __device__ constexpr bool warp_lines() { return N == 256; }
template <int N>
__host__ __device__ constexpr int line_len() { return warp_lines<N>() ? plane_ld(N) : N; }
template <int N>
__host__ __device__ constexpr int row_batch() { return warp_lines<N>() ? 16 : kRowBatch; }

// complex elements of the line batches (the largest of passes A-G)
__host__ __device__ constexpr int general_line_elems(int N) {
  const int len = N == 256 ? plane_ld(256) : N;
  const int rb = N == 256 ? 16 : kRowBatch;
  int lines = 2 * kLineCols;
  if (2 * rb > lines) lines = 2 * rb;
  if (kColBatch > lines) lines = kColBatch;
  return lines * len;
}

// position of input element k of a line, and of output element k
template <int N>
__device__ __forceinline__ int lin(int line, int k) {
  return warp_lines<N>() ? line * plane_ld(N) + k + (k >> 3) : line * N + fft_in_pos(k, N);
}
template <int N>
__device__ __forceinline__ int lout(int line, int k) {
  return warp_lines<N>() ? line * plane_ld(N) + k + (k >> 3) : line * N + k;
}

// One warp's transform of one or two lines (``inv``: the unnormalised
// inverse), one out-of-line copy for both directions: inlined at every call
// site of the general kernel, the lane's twiddle factors were hoisted out of
// the pass loops and held in registers throughout (255 registers, spills).
template <int N>
__device__ __noinline__ void warp_fft_lines(float2* p, int nlines, const float2* tw, bool inv) {
  warp_fft<N, -1>(StageLines<N>{p}, nlines, tw, inv);
}

// In-place transforms of ``lines`` lines of the batch (sign -1 forward, +1
// unnormalised inverse), followed by a block barrier.
template <int N>
__device__ __forceinline__ void line_fft(float2* buf, int lines, float sign, const float2* tw,
                                         const float2* tw3) {
  if constexpr (warp_lines<N>()) {
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int g0 = 2 * warp; g0 < lines; g0 += 2 * nw) {
      warp_fft_lines<N>(buf + g0 * plane_ld(N), min(2, lines - g0), tw, sign > 0.f);
    }
    __syncthreads();
  } else {
    smem_fft(buf, N, lines, sign, tw, tw3);
  }
}

template <int N>
__device__ void build_one(const ProjParams& P, int b, int dir, int slot, float2* S, float2* Pk,
                          float2* sm, float4* red4, float* redf, float* s_mu, float* s_div) {
  constexpr int m = 2 * N, W = N + 1, RB = row_batch<N>();
  // unroll of the loops that read the scratch plane: box 256 keeps four
  // loads in flight per thread (the smaller boxes run more CTAs per SM and
  // keep their register count)
  constexpr int UNR = warp_lines<N>() ? 4 : 1;
  const int nb = P.nb, H = nb / 2 + 1;
  const int LDS = N + 1;  // scratch row stride (complex)
  const float* R = P.rot + (size_t)dir * 9;
  const float R00 = R[0], R01 = R[1], R10 = R[3], R11 = R[4], R20 = R[6], R21 = R[7];
  const float inv_m = (float)(1.0 / (double)m);

  // ---- pass A: gather + row inverse (pruned to the N centred rows), unless
  // rows_inverse already wrote this template's plane (P.planes, [N][N+1])
  const float2* A = P.planes != nullptr ? P.planes + (size_t)b * N * LDS : S;
  for (int c0 = 0; P.planes == nullptr && c0 < W; c0 += kLineCols) {
    const int nc = min(kLineCols, W - c0);
    const int total = nc * m;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const int cl = t / m, r = t - cl * m;  // r: standard-order row of the 2N grid
      const int c = c0 + cl;
      const int kys = (r + N) % m;            // row in the shifted base grid
      const float gy = __fmul_rn((float)(kys - N), inv_m);
      const float gx = __fmul_rn((float)c, inv_m);
      float rx = __fadd_rn(__fmul_rn(R00, gx), __fmul_rn(R01, gy));
      float ry = __fadd_rn(__fmul_rn(R10, gx), __fmul_rn(R11, gy));
      float rz = __fadd_rn(__fmul_rn(R20, gx), __fmul_rn(R21, gy));
      const bool conj = rx < 0.0f;
      if (conj) { rx = -rx; ry = -ry; rz = -rz; }
      const float cz = __fadd_rn(__fmul_rn(rz, (float)m), (float)(m / 2));
      const float cy = __fadd_rn(__fmul_rn(ry, (float)m), (float)(m / 2));
      const float cx = __fmul_rn(rx, (float)m);
      float2 v = sample_trilinear(P.spectrum, m, W, grid_pixel(cz, m), grid_pixel(cy, m),
                                  grid_pixel(cx, W));
      if (conj) v.y = -v.y;
      const int e = r & 1, q = r >> 1;
      sm[lin<N>(cl * 2 + e, q)] = v;
    }
    __syncthreads();
    line_fft<N>(sm, 2 * nc, +1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int cl = t / N, i = t - cl * N;
      const int u = i - N / 2;               // signed output row of the 2N-point inverse
      const int k = (u + N) % N;
      const float2 a0 = sm[lout<N>(cl * 2, k)];
      const float2 a1 = sm[lout<N>(cl * 2 + 1, k)];
      const float2 z = cadd_s(a0, cmul(tw_pos_any(P.t.tw, P.t.tw3, u, m), a1));
      S[(size_t)i * LDS + c0 + cl] = z;
    }
    __syncthreads();
  }

  // ---- pass B: C2R along columns, keep centred N, then forward row FFT
  const float scale_b = (float)(1.0 / ((double)m * (double)m));
  float2* sm2 = sm + RB * line_len<N>();
  for (int i0 = 0; i0 < N; i0 += RB) {
    const int nr = min(RB, N - i0);
#pragma unroll (UNR)
    for (int t = threadIdx.x; t < nr * N; t += blockDim.x) {
      const int rl = t / N, k = t - rl * N;
      const float2* Z = A + (size_t)(i0 + rl) * LDS;
      float2 ye, yo;
      if (k == 0) {
        const float a = Z[0].x, b = Z[N].x;
        ye = make_float2(a + b, 0.f);
        yo = make_float2(a - b, 0.f);
      } else {
        const float2 zk = Z[k], zc = cconj(Z[N - k]);
        ye = cadd_s(zk, zc);
        yo = cmul(csub_s(zk, zc), tw_pos_any(P.t.tw, P.t.tw3, k, m));
      }
      // W = Ye + i*Yo
      sm[lin<N>(rl, k)] = make_float2(ye.x - yo.y, ye.y + yo.x);
    }
    __syncthreads();
    line_fft<N>(sm, nr, +1.0f, P.t.tw, P.t.tw3);
    // p(2n) = Re z(n), p(2n+1) = Im z(n); keep v = (j - N/2) mod 2N.
    for (int t = threadIdx.x; t < nr * N; t += blockDim.x) {
      const int rl = t / N, j = t - rl * N;
      const int v = (j - N / 2 + m) % m;
      const float2 zz = sm[lout<N>(rl, v >> 1)];
      const float p = ((v & 1) ? zz.y : zz.x) * scale_b;
      sm2[lin<N>(rl, j)] = make_float2(p, 0.f);
    }
    __syncthreads();
    line_fft<N>(sm2, nr, -1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nr * (N / 2 + 1); t += blockDim.x) {
      const int rl = t / (N / 2 + 1), k = t - rl * (N / 2 + 1);
      S[(size_t)(i0 + rl) * LDS + k] = sm2[lout<N>(rl, k)];
    }
    __syncthreads();
  }

  // ---- pass C: forward column FFT (kx in [0, N/2])
  const int HC = N / 2 + 1;
  for (int c0 = 0; c0 < HC; c0 += kColBatch) {
    const int nc = min(kColBatch, HC - c0);
#pragma unroll (UNR)
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int r = t / nc, cl = t - r * nc;
      sm[lin<N>(cl, r)] = S[(size_t)r * LDS + c0 + cl];
    }
    __syncthreads();
    line_fft<N>(sm, nc, -1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int r = t / nc, cl = t - r * nc;
      S[(size_t)r * LDS + c0 + cl] = sm[lout<N>(cl, r)];
    }
    __syncthreads();
  }
  // radial sums of |F| over the full grid in float32 (columns 1..N/2-1
  // stand for two bins): per lane, then a fixed xor tree across the warp
  {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int b = warp; b < P.t.n_bins; b += nw) {
      float acc = 0.f;
#pragma unroll (UNR / 2 > 0 ? UNR / 2 : 1)
      for (int e = P.t.bin_ptr[b] + lane; e < P.t.bin_ptr[b + 1]; e += 32) {
        const int idx = P.t.bin_list[e];
        const int r = idx / HC, kx = idx - r * HC;
        const float2 f = S[(size_t)r * LDS + kx];
        const float a = sqrt_approx(fmaf(f.x, f.x, f.y * f.y));
        acc += (kx == 0 || kx == N / 2) ? a : 2.0f * a;
      }
      acc = warp_sum(acc);
      if (lane == 0) s_div[b] = (b == 0) ? 1.0f : __fdiv_rn(P.t.bin_count[b], acc);
    }
  }
  // The DC term (bin 0, left as it is) over N^2 is the image mean; it is read
  // before column 0 is transformed and taken out of every pixel in pass E,
  // so the float32 plane-fit and variance sums run on centred values.
  const float scale_e = (float)(1.0 / ((double)N * (double)N));
  if (threadIdx.x == 0) s_mu[0] = S[0].x * scale_e;
  __syncthreads();

  // ---- pass D: scale by the radial divisor, inverse column FFT
  for (int c0 = 0; c0 < HC; c0 += kColBatch) {
    const int nc = min(kColBatch, HC - c0);
#pragma unroll (UNR)
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int r = t / nc, cl = t - r * nc;
      const int kx = c0 + cl;
      const int ky = r < N / 2 ? r : r - N;
      const int bin = (int)rintf(sqrtf((float)(ky * ky + kx * kx)));
      sm[lin<N>(cl, r)] = cscale(S[(size_t)r * LDS + kx], s_div[bin]);
    }
    __syncthreads();
    line_fft<N>(sm, nc, +1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int r = t / nc, cl = t - r * nc;
      S[(size_t)r * LDS + c0 + cl] = sm[lout<N>(cl, r)];
    }
    __syncthreads();
  }

  // ---- pass E: inverse row transform (real part), centred pixels, float32
  // plane-fit sums (per thread, then a fixed tree across the block)
  const float mu = s_mu[0];
  float fz = 0.f, fxz = 0.f, fyz = 0.f, fww = 0.f;
  for (int i0 = 0; i0 < N; i0 += RB) {
    const int nr = min(RB, N - i0);
#pragma unroll (UNR)
    for (int t = threadIdx.x; t < nr * N; t += blockDim.x) {
      const int rl = t / N, k = t - rl * N;
      const float2* G = S + (size_t)(i0 + rl) * LDS;
      float2 y;
      if (k == 0 || k == N / 2) y = make_float2(G[k].x, 0.f);
      else if (k < N / 2) y = G[k];
      else y = cconj(G[N - k]);
      sm[lin<N>(rl, k)] = y;
    }
    __syncthreads();
    line_fft<N>(sm, nr, +1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nr * N; t += blockDim.x) {
      const int rl = t / N, j = t - rl * N;
      const int i = i0 + rl;
      const float w = fmaf(sm[lout<N>(rl, j)].x, scale_e, -mu);
      S[(size_t)i * LDS + j] = make_float2(w, 0.f);
      fz += w;
      fxz = fmaf((float)i, w, fxz);
      fyz = fmaf((float)j, w, fyz);
      fww = fmaf(w, w, fww);
    }
    __syncthreads();
  }
  // Least-squares plane z = c0*row + c1*col + c2 over the full N x N grid in
  // closed form: the grid is a Cartesian product, so the centred row and
  // column coordinates are orthogonal and the 3x3 normal equations decouple.
  const float4 s4 = block_sum_f4<kThreads / 32>(make_float4(fz, fxz, fyz, fww), red4);
  constexpr float kMid = 0.5f * (float)(N - 1);
  constexpr float kSii = (float)((double)N * (double)N * ((double)N * (double)N - 1.0) / 12.0);
  const float pc0 = (s4.y - kMid * s4.x) / kSii;
  const float pc1 = (s4.z - kMid * s4.x) / kSii;
  const float pcm = s4.x * scale_e - (pc0 + pc1) * kMid;
  // Residual energy sum (w - P)^2 = sum w^2 - sum P w (the residual of a
  // least-squares fit is orthogonal to the fit); where the plane holds most
  // of the energy the subtraction would cancel, and the residual is summed
  // directly instead (a block-uniform choice).
  float ssr = s4.w - fmaf(pc0, s4.y, fmaf(pc1, s4.z, pcm * s4.x));
  if (!(ssr > 0.25f * s4.w)) {
    float fsv = 0.f;
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int i = t / N, j = t - i * N;
      const float v = S[(size_t)i * LDS + j].x - fmaf(pc0, (float)i, fmaf(pc1, (float)j, pcm));
      fsv = fmaf(v, v, fsv);
    }
    ssr = block_sum_f<kThreads / 32>(fsv, redf);
  }
  const float sd = sqrtf(ssr * scale_e);
  const float inv_sd = sd > 1e-12f ? 1.0f / sd : 1.0f;

  // ---- pass F: normalise, mask, forward row FFT
  for (int i0 = 0; i0 < N; i0 += RB) {
    const int nr = min(RB, N - i0);
#pragma unroll (UNR)
    for (int t = threadIdx.x; t < nr * N; t += blockDim.x) {
      const int rl = t / N, j = t - rl * N;
      const int i = i0 + rl;
      float f = (S[(size_t)i * LDS + j].x - fmaf(pc0, (float)i, fmaf(pc1, (float)j, pcm))) * inv_sd;
      if (P.mask != nullptr) f *= P.mask[(size_t)i * N + j];
      sm[lin<N>(rl, j)] = make_float2(f, 0.f);
    }
    __syncthreads();
    line_fft<N>(sm, nr, -1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nr * HC; t += blockDim.x) {
      const int rl = t / HC, k = t - rl * HC;
      S[(size_t)(i0 + rl) * LDS + k] = sm[lout<N>(rl, k)];
    }
    __syncthreads();
  }
  // ---- pass G: forward column FFT
  for (int c0 = 0; c0 < HC; c0 += kColBatch) {
    const int nc = min(kColBatch, HC - c0);
#pragma unroll (UNR)
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int r = t / nc, cl = t - r * nc;
      sm[lin<N>(cl, r)] = S[(size_t)r * LDS + c0 + cl];
    }
    __syncthreads();
    line_fft<N>(sm, nc, -1.0f, P.t.tw, P.t.tw3);
    for (int t = threadIdx.x; t < nc * N; t += blockDim.x) {
      const int r = t / nc, cl = t - r * nc;
      S[(size_t)r * LDS + c0 + cl] = sm[lout<N>(cl, r)];
    }
    __syncthreads();
  }
  // crop + pack + FSC, L2 norm (float32 per thread, fixed tree across the block)
  float fss = 0.f;
#pragma unroll (UNR)
  for (int t = threadIdx.x; t < nb * H; t += blockDim.x) {
    const int r = t / H, c = t - r * H;
    const int ky = r < nb / 2 ? r : r - nb;
    float2 f;
    if (c < nb / 2) {
      f = S[(size_t)((ky + N) % N) * LDS + c];
    } else if (nb == N) {
      f = S[(size_t)((ky + N) % N) * LDS + N / 2];
    } else {
      f = cconj(S[(size_t)((-ky + N) % N) * LDS + nb / 2]);
    }
    f = cscale(f, P.fsc[t]);
    Pk[t] = f;
    fss = fmaf(f.x, f.x, fmaf(f.y, f.y, fss));
  }
  const float inv_norm = 1.0f / sqrtf(block_sum_f<kThreads / 32>(fss, redf));
  float2* out = P.bank + (size_t)slot * nb * H;
  for (int t = threadIdx.x; t < nb * H; t += blockDim.x) {
    const int r = t / H, c = t - r * H;
    const int rs = (r + nb / 2) % nb, cs = (c + H / 2) % H;
    out[(size_t)rs * H + cs] = cscale(Pk[t], inv_norm);
  }
  __syncthreads();
}

// Box 256 asks for two CTAs per SM (128 registers); a minimum of 0 leaves the
// other boxes to the compiler's default (40 registers; 72 with a minimum of 1).
template <int N>
__global__ void __launch_bounds__(kThreads, warp_lines<N>() ? 2 : 0) project_templates(ProjParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* sm = reinterpret_cast<float2*>(smem_raw);
  float2* s_tw = sm + general_line_elems(N);
  float4* red4 = reinterpret_cast<float4*>(s_tw + kMaxFftLen / 2);  // [kThreads / 32]
  float* redf = reinterpret_cast<float*>(red4 + kThreads / 32);      // [kThreads / 32]
  float* s_mu = redf + kThreads / 32;                                 // [4]
  float* s_div = s_mu + 4;                                            // [n_bins + 4]
  for (int t = threadIdx.x; t < kMaxFftLen / 2; t += blockDim.x) s_tw[t] = P.t.tw[t];
  __syncthreads();
  ProjParams Q = P;
  Q.t.tw = s_tw;
  float2* S = P.scratch + (size_t)blockIdx.x * P.scratch_stride;
  float2* Pk = S + (size_t)N * (N + 1);
  for (int b = blockIdx.x; b < P.n_build; b += gridDim.x) {
    const int dir = P.dirs[b];
    const int slot = P.out_slot ? P.out_slot[b] : dir;
    build_one<N>(Q, b, dir, slot, S, Pk, sm, red4, redf, s_mu, s_div);
  }
}

}  // namespace

// complex elements of the pass-A planes of n_build templates
size_t project_plane_elems(int N, int n_build) { return (size_t)n_build * N * (N > 128 ? N + 1 : N + 2); }

// complex elements of one CTA's scratch in the general kernel
size_t project_scratch_elems(int N, int nb) {
  return (size_t)N * (N + 1) + (size_t)nb * (nb / 2 + 1);
}

static size_t general_smem_bytes(int N, int n_bins) {
  return (size_t)general_line_elems(N) * sizeof(float2) + (kMaxFftLen / 2) * sizeof(float2) +
         (kThreads / 32) * (sizeof(float4) + sizeof(float)) + (size_t)(4 + n_bins + 4) * sizeof(float);
}

// ===========================================================================
// Slice gather from the blocked spectrum and pass A at high occupancy
// (rows_inverse), and the template tail on a shared-memory plane
// (template_tail). The block sums are float32 over a fixed tree.
// ===========================================================================
namespace {

// Columns a warp transforms per pass-A round: G = 32 / (N/16) lines, two
// per column (even and odd rows of the 2N grid).
template <int N>
__host__ __device__ constexpr int pass_a_cols() { return 16 / (N / 16); }

// The half-volume spectrum in the blocked layout the slice gather reads:
// centred order along z and y, cut into blocks of 2 (z) x 4 (y) x 2 (x)
// voxels, one 128-byte line each (x padded to an even count). A trilinear
// footprint then spans about two lines instead of four rows, and the 32
// samples of one warp load touch 12 lines instead of 21 (counted for
// random orientations), which is what bounds the gather's L1 throughput.
constexpr int kBZ = 2, kBY = 4, kBX = 2, kBE = kBZ * kBY * kBX;

template <int N>
__host__ __device__ constexpr int blocked_x() { return (N + 1 + kBX - 1) / kBX; }

template <int N>
__global__ void __launch_bounds__(256) spectrum_blocked(const float2* __restrict__ spectrum,
                                                        float2* __restrict__ out) {
  constexpr int m = 2 * N, W = N + 1, XB = blocked_x<N>(), YB = m / kBY;
  const int total = (m / kBZ) * YB * XB * kBE;
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < total; o += gridDim.x * blockDim.x) {
    const int e = o % kBE, blk = o / kBE;
    const int xb = blk % XB, yb = (blk / XB) % YB, zb = blk / (XB * YB);
    const int x = xb * kBX + e % kBX, y = yb * kBY + (e / kBX) % kBY, z = zb * kBZ + e / (kBX * kBY);
    // the spectrum is stored unshifted along z and y: index (i + N) mod 2N
    const int zs = z < N ? z + N : z - N, ys = y < N ? y + N : y - N;
    out[o] = __ldg(spectrum + ((size_t)zs * m + ys) * W + min(x, W - 1));
  }
}

// Offset of a voxel in the blocked copy, one axis at a time.
template <int N>
__device__ __forceinline__ int blocked_z(int z) {
  return (z >> 1) * ((2 * N / kBY) * blocked_x<N>() * kBE) + (z & 1) * (kBY * kBX);
}
template <int N>
__device__ __forceinline__ int blocked_y(int y) {
  return (y >> 2) * (blocked_x<N>() * kBE) + (y & 3) * kBX;
}
__device__ __forceinline__ int blocked_xo(int x) { return (x >> 1) * kBE + (x & 1); }

// Trilinear sample of the blocked copy by a pair of lanes (h = 0, 1), at the
// slice point's voxel coordinates (grid_sample's normalise/un-normalise pair
// with align_corners=True is the identity, so the coordinates are used directly,
// clamped for border padding). Corners past the last voxel carry weight 0 and
// are read clamped. Lane h loads the four corners of plane z0 + h: the two
// planes of a pair mostly lie in one 128-byte line, so a warp load of 16 samples
// touches about 17 lines for both, against 2 x 25 when each corner is a load of
// its own over 32 samples (host count over random directions), and the data
// pipe of the L1 bounds the gather (91% to 97% busy). The sum runs in
// grid_sample's corner order: plane z0 in lane 0, which hands it on to lane 1;
// the result is lane 1's.
template <int N>
__device__ __forceinline__ float2 sample_pair(const float2* __restrict__ vol, float cz, float cy, float cx, int h) {
  constexpr int m = 2 * N, W = N + 1;
  const float pz = fminf((float)(m - 1), fmaxf(cz, 0.0f));
  const float py = fminf((float)(m - 1), fmaxf(cy, 0.0f));
  const float px = fminf((float)(W - 1), fmaxf(cx, 0.0f));
  const float fz = floorf(pz), fy = floorf(py), fx = floorf(px);
  const int z = min((int)fz + h, m - 1), y0 = (int)fy, x0 = (int)fx;
  const float wz = h ? __fsub_rn(pz, fz) : __fsub_rn(fz + 1.0f, pz);
  const float wy1 = __fsub_rn(py, fy), wx1 = __fsub_rn(px, fx);
  const float wy0 = __fsub_rn(fy + 1.0f, py), wx0 = __fsub_rn(fx + 1.0f, px);
  const int oz = blocked_z<N>(z), oy0 = oz + blocked_y<N>(y0), oy1 = oz + blocked_y<N>(min(y0 + 1, m - 1));
  const int ox0 = blocked_xo(x0), ox1 = blocked_xo(min(x0 + 1, W - 1));
  const float2 v00 = __ldg(vol + (oy0 + ox0)), v01 = __ldg(vol + (oy0 + ox1));
  const float2 v10 = __ldg(vol + (oy1 + ox0)), v11 = __ldg(vol + (oy1 + ox1));
  const float w00 = __fmul_rn(__fmul_rn(wx0, wy0), wz), w01 = __fmul_rn(__fmul_rn(wx1, wy0), wz);
  const float w10 = __fmul_rn(__fmul_rn(wx0, wy1), wz), w11 = __fmul_rn(__fmul_rn(wx1, wy1), wz);
  float2 a = make_float2(v00.x * w00, v00.y * w00);
  a.x = fmaf(v01.x, w01, a.x); a.y = fmaf(v01.y, w01, a.y);
  a.x = fmaf(v10.x, w10, a.x); a.y = fmaf(v10.y, w10, a.y);
  a.x = fmaf(v11.x, w11, a.x); a.y = fmaf(v11.y, w11, a.y);
  a.x = __shfl_xor_sync(0xffffffffu, a.x, 1);
  a.y = __shfl_xor_sync(0xffffffffu, a.y, 1);
  a.x = fmaf(v00.x, w00, a.x); a.y = fmaf(v00.y, w00, a.y);
  a.x = fmaf(v01.x, w01, a.x); a.y = fmaf(v01.y, w01, a.y);
  a.x = fmaf(v10.x, w10, a.x); a.y = fmaf(v10.y, w10, a.y);
  a.x = fmaf(v11.x, w11, a.x); a.y = fmaf(v11.y, w11, a.y);
  return a;
}

// Pass A as its own high-occupancy kernel: slice gather and pruned inverse
// along the 2N grid rows. A CTA takes kRiWarps * CPR columns of one
// template; a warp gathers its CPR columns into G = 2 * CPR staged lines
// (even and odd rows of the 2N grid), transforms them with one warp FFT and
// combines each even/odd pair into the N centred rows of the 2N-point
// inverse (output row (k + N/2) mod N takes frequency k). The CTA then
// writes its columns row by row into the template's plane in global memory.
constexpr int kRiWarps = 4;

// row stride of a pass-A plane: N + 2 up to 128 (whole 16-byte units, for the
// bulk copies), N + 1 for the general kernel of box 256
__host__ __device__ constexpr int plane_out_ld(int N) { return N > 128 ? N + 1 : N + 2; }

template <int N>
__host__ __device__ constexpr int ri_cols() { return kRiWarps * pass_a_cols<N>(); }

// Eight CTAs per SM (64 registers, 21 KB of shared memory): the gather is
// bound by the latency of its scattered loads, and resident warps hide it
// (measured on GB300 at box 128: 7 CTAs per SM 0.615 ms for the gather and
// tail of 768 templates, 8 CTAs 0.597 ms, 9 CTAs at 56 registers the same,
// 10 CTAs at 48 registers 0.644 ms; giving the L1 more of the SM's memory at
// the cost of resident CTAs was slower still). Streaming (evict-first) stores
// of the planes, to keep the blocked spectrum in L2, measured the same.
template <int N>
__global__ void __launch_bounds__(kRiWarps * 32, 8) rows_inverse(const float2* __restrict__ spectrum,
                                                              const float* __restrict__ rot,
                                                              const int* __restrict__ dirs, ProjTables tab,
                                                              float2* __restrict__ planes) {
  constexpr int m = 2 * N, W = N + 1, CPR = pass_a_cols<N>(), CC = ri_cols<N>();
  constexpr int OUTC = CC + 1, STAGE = stage_elems(N, 2 * CPR);
  static_assert(N * OUTC <= kRiWarps * STAGE, "the output tile fits the staging lines");
  static_assert(2 * CPR == fft_lines<N>(), "a warp's lines are one transform");
  __shared__ float2 s_tw[N], s_tw2[N];
  // staging lines of the gather and the FFT; once every warp has its
  // outputs in registers, the same memory holds the CTA's N x CC output tile
  __shared__ float2 s_line[kRiWarps][STAGE];
  float2(*s_out)[OUTC] = reinterpret_cast<float2(*)[OUTC]>(&s_line[0][0]);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y, c_cta = blockIdx.x * CC, cw = c_cta + warp * CPR;
  const int nc = max(0, min(CPR, W - cw));
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
    s_tw[t] = __ldg(tab.tw_n + t);
    s_tw2[t] = __ldg(tab.tw_2n + t);
  }
  const float* R = rot + (size_t)dirs[b] * 9;
  const StagedLines<N> L{s_line[warp]};
  // A pair of lanes takes a sample, 16 samples of CL columns x 16/CL rows at
  // once (neighbouring samples share trilinear corners), rows in the centred
  // order, so that a lane's column and the step between its rows are constants.
  const int ncta = max(0, min(CC, W - c_cta));
  if (nc > 0) {
    constexpr int CL = CPR < 4 ? CPR : 4, RL = 16 / CL;
    constexpr float inv_m = (float)(1.0 / (double)m);
    const int h = lane & 1, s16 = lane >> 1, r_first = s16 / CL;
    const float R1 = R[1], R4 = R[4], R7 = R[7];
#pragma unroll
    for (int cb = 0; cb < CPR; cb += CL) {
      const int cl = cb + s16 % CL;
      const float gx = __fmul_rn((float)(cw + cl), inv_m);
      const float x0 = __fmul_rn(R[0], gx), y0 = __fmul_rn(R[3], gx), z0 = __fmul_rn(R[6], gx);
      float2* dst = L.line(2 * cl + (r_first & 1));
      static_assert(RL % 2 == 0, "a lane's rows have one parity");
#pragma unroll 4
      for (int k = 0; k < m / RL; ++k) {
        const int rc = r_first + k * RL;  // centred row; row rc - N of the grid
        const float gy = __fmul_rn((float)(rc - N), inv_m);
        float rx = __fadd_rn(x0, __fmul_rn(R1, gy));
        float ry = __fadd_rn(y0, __fmul_rn(R4, gy));
        float rz = __fadd_rn(z0, __fmul_rn(R7, gy));
        const bool conj = rx < 0.0f;
        if (conj) { rx = -rx; ry = -ry; rz = -rz; }
        float2 v = sample_pair<N>(spectrum, fmaf(rz, (float)m, (float)(m / 2)), fmaf(ry, (float)m, (float)(m / 2)),
                                  __fmul_rn(rx, (float)m), h);  // products by m are exact
        if (conj) v.y = -v.y;
        const int q = ((rc + N) & (m - 1)) >> 1;  // row (rc - N) mod 2N: position within its parity's line
        if (h) dst[L.slot(q)] = v;
      }
    }
  }
  __syncthreads();
  constexpr int RES = CPR * N / 32;  // outputs of a lane (8 at every box)
  float2 res[RES];
  if (nc > 0) {
    line_fft_warp<N, 1>(L, s_tw);
#pragma unroll
    for (int i = 0; i < RES; ++i) {
      const int idx = lane + 32 * i, cl = idx / N, k = idx - cl * N;
      const int u = k < N / 2 ? k : k - N;
      const float2 w = s_tw2[abs(u)];  // exp(+2 pi i u / 2N) is its conjugate for u > 0
      res[i] = cadd(L.at(2 * cl, k), cmul(u >= 0 ? cconj(w) : w, L.at(2 * cl + 1, k)));
    }
  }
  __syncthreads();  // every warp has read its lines
  if (nc > 0) {
#pragma unroll
    for (int i = 0; i < RES; ++i) {
      const int idx = lane + 32 * i;
      if (idx < nc * N) {
        const int cl = idx / N, k = idx - cl * N;
        s_out[(k + N / 2) & (N - 1)][warp * CPR + cl] = res[i];
      }
    }
  }
  __syncthreads();
  constexpr int OUT = plane_out_ld(N);
  float2* dst = planes + (size_t)b * N * OUT;
  for (int e = threadIdx.x; e < N * CC; e += blockDim.x) {
    const int y = e / CC, cl = e - y * CC, c = c_cta + cl;
    if (cl < ncta) dst[(size_t)y * OUT + c] = s_out[y][cl];
  }
}

// ---------------------------------------------------------------------------
// The template tail: passes B to G on the pair plane.
//
// Measured before (one CTA of 20 warps per SM on an N x (N + 1) plane of 173 KB
// at box 128): issue and latency, with every barrier of the one template in
// flight exposed. The paired rows take 75 KB, so two templates of 16 warps share
// an SM at box 128 and fill one another's barriers, and the steps between the transforms
// (radial divisor, Hermitian packing, plane removal and mask) run where a
// transform loads or stores its elements instead of in passes of their own.
// Column 0 of the plane holds two real columns, DC and Nyquist, and they are
// transformed one by one (the Nyquist column in an array of its own): packed as
// one complex line they would be cheaper, but the DC bin keeps its raw amplitude
// through the whitening, thousands of times the other bins', and its rounding
// would then depend on the other column. Measured on GB300, gather and tail of
// 768 templates at box 128: 594 -> 448 us.
// ---------------------------------------------------------------------------
template <int N>
__host__ __device__ constexpr int tail_threads() {
  return N == 32 ? 64 : (N == 64 ? 128 : 512);
}
// CTAs per SM: as the registers allow (at box 128 the shared memory would hold
// three of 8 warps, which measured 485 us where two of 16 take 471, gather
// included)
template <int N>
__host__ __device__ constexpr int tail_ctas() { return N <= 64 ? 6 : 2; }

// The even rows of a template's plane arrive by bulk async copies, each into
// the shared-memory line of its pair (one contiguous row in the line's slots,
// from the first 16-byte boundary); every wait is bounded. The odd rows are
// read from global memory when the even ones have been transformed.
constexpr unsigned kPlaneWaitLimit = 1u << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <int N>
__device__ __forceinline__ int raw_row(int q) {
  const int o = q * pair_ld(N) + (q >> 2);
  return o + (o & 1);
}

template <int N>
__device__ __forceinline__ void rows_load(float2* Zs, const float2* src, uint64_t* bar) {
  constexpr uint32_t kRow = (uint32_t)plane_out_ld(N) * sizeof(float2);
  static_assert(kRow % 16 == 0 && plane_out_ld(N) + 1 <= pair_ld(N), "a row is whole 16-byte units and fits its line");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(kRow * (N / 2)) : "memory");
  for (int q = 0; q < N / 2; ++q)
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(Zs + raw_row<N>(q))),
        "l"(src + (size_t)2 * q * plane_out_ld(N)), "r"(kRow), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool plane_wait(uint64_t* bar, uint32_t parity, unsigned limit) {
  for (unsigned i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The small shared arrays of a tail CTA, after the plane and the Nyquist column.
template <int N>
struct TailShared {
  float4 red4[tail_threads<N>() / 32];
  float red[tail_threads<N>() / 32];
  float mu;
  uint64_t bar;
  float2 tw[N], tw2[N];  // twiddles of the transforms, exp(-2 pi i t / 2N)
};

template <int N>
__device__ __forceinline__ void tail_tables(const ProjTables& t, TailShared<N>& S) {
  for (int k = threadIdx.x; k < N; k += tail_threads<N>()) {
    S.tw[k] = __ldg(t.tw_n + k);
    S.tw2[k] = __ldg(t.tw_2n + k);
  }
}

// The Nyquist column's line.
template <int N>
struct NyquistLine {
  float2* p;
  __device__ __forceinline__ float2& at(int, int k) const { return p[k]; }
};

// Passes B to G of one template. ``rows``: its pass-A plane in global memory,
// whose even rows are already in the lines' slots.
template <int N>
__device__ __forceinline__ void tail_passes(const ProjParams& P, const float2* rows, int slot, float2* Zs, float* s_div,
                                            TailShared<N>& S) {
  constexpr int NT = tail_threads<N>(), NW = NT / 32, G = fft_lines<N>(), HC = N / 2 + 1, m = 2 * N;
  constexpr int RG = pair_row_groups<N>(), CG = pair_col_groups<N>(), EPL = G * N / 64;
  const PairPlane<N> Z{Zs};
  float2* nyq = Zs + pair_elems(N);
  const float2* tw = S.tw;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = P.nb, H = nb / 2 + 1;

  // ---- pass B: C2R along rows (an N-point inverse each), the centred N
  // columns kept; the two rows of a pair become the halves of its line, and
  // the line's forward transform starts the whitening
  const float scale_b = (float)(1.0 / ((double)m * (double)m));
  for (int grp = warp; grp < RG; grp += NW) {
    const PairRows<N> R{Z, grp};
    float2 even[EPL];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      // W = Ye + i Yo. A task owns the pair (k, N - k): both outputs depend
      // on the row's elements k and N - k only.
      constexpr int TASKS = G * HC, IT = (TASKS + 31) / 32;
      float2 zk[IT], zn[IT];
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const int idx = lane + 32 * i;
        if (idx < TASKS) {
          const int g = idx / HC, k = idx - g * HC;
          if (e == 0) {
            const float2* row = Zs + raw_row<N>(R.row(g));
            zk[i] = row[k];
            zn[i] = row[N - k];
          } else {
            const float2* row = rows + (size_t)(2 * R.row(g) + e) * plane_out_ld(N);
            zk[i] = __ldcg(row + k);
            zn[i] = __ldcg(row + N - k);
          }
        }
      }
      __syncwarp();  // every lane has read its rows
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const int idx = lane + 32 * i;
        if (idx < TASKS) {
          const int g = idx / HC, k = idx - g * HC;
          if (k == 0) {
            R.at(g, 0) = make_float2(zk[i].x + zn[i].x, zk[i].x - zn[i].x);  // Ye and Yo are real
          } else {
            const float2 w = cconj(S.tw2[k]);  // exp(+2 pi i k / 2N)
            const float2 ye = cadd(zk[i], cconj(zn[i])), yo = cmul(csub(zk[i], cconj(zn[i])), w);
            R.at(g, k) = make_float2(ye.x - yo.y, ye.y + yo.x);
            if (k != N / 2) {
              const float2 ye2 = cadd(zn[i], cconj(zk[i]));
              const float2 yo2 = cmul(csub(zn[i], cconj(zk[i])), cconj(S.tw2[N - k]));
              R.at(g, N - k) = make_float2(ye2.x - yo2.y, ye2.y + yo2.x);
            }
          }
        }
      }
      __syncwarp();
      line_fft_warp<N, 1>(R, tw);
      // p(2n) = Re z(n), p(2n + 1) = Im z(n); columns j, j + 1 = v + N/2 of v = 2n
      float2 p[EPL];
#pragma unroll
      for (int t = 0; t < EPL; ++t) {
        const int idx = lane + 32 * t, g = idx / (N / 2), u = idx - g * (N / 2);
        p[t] = cscale(R.at(g, u < N / 4 ? u - N / 4 + N : u - N / 4), scale_b);
      }
      __syncwarp();
      if (e == 0) {
#pragma unroll
        for (int t = 0; t < EPL; ++t) even[t] = p[t];
      } else {
#pragma unroll
        for (int t = 0; t < EPL; ++t) {
          const int idx = lane + 32 * t, g = idx / (N / 2), u = idx - g * (N / 2);
          R.at(g, 2 * u) = make_float2(even[t].x, p[t].x);
          R.at(g, 2 * u + 1) = make_float2(even[t].y, p[t].y);
        }
      }
      __syncwarp();
    }
    line_fft_warp<N, -1>(R, tw);
    pair_split_rows<N>(R);
  }
  __syncthreads();

  // Forward transforms of all columns: column 0's line is the DC column (the
  // real parts), the Nyquist column (the imaginary parts) goes to its own array
  // before the line is overwritten, by the warp of column 0.
  const NyquistLine<N> Q{nyq};
  auto forward_columns = [&]() {
    for (int grp = warp; grp < CG; grp += NW) {
      const PairCols<N> cols{Z, grp * G};
      if (grp == 0) {
        line_fft_warp<N, -1, 1>(Q, tw, [&](int, int i) { return make_float2(Z.half(i, 0).y, 0.f); },
                                [&](int, int i, float2 v) { nyq[i] = v; });
        line_fft_warp<N, -1>(cols, tw, [&](int g, int i) {
          const float2 f = cols.at(g, i);
          return g == 0 ? make_float2(f.x, 0.f) : f;
        }, [&](int g, int i, float2 v) { cols.at(g, i) = v; });
      } else {
        line_fft_warp<N, -1>(cols, tw);
      }
    }
  };

  // ---- pass C: forward column transforms, then the radial |F| sums in float32
  // (the reference sums in float32 with scatter_add_): per lane, then a fixed
  // xor tree across the warp. The bin list holds plane offsets, the top bit
  // set for columns 0 and N/2 (weight 1; every other column stands for itself
  // and its mirror, weight 2).
  forward_columns();
  __syncthreads();
  for (int b = warp; b < P.t.n_bins; b += NW) {
    float acc = 0.f;
    const int e1 = __ldg(P.t.bin_ptr + b + 1);
#pragma unroll 4
    for (int e = __ldg(P.t.bin_ptr + b) + lane; e < e1; e += 32) {
      const unsigned v = __ldg(P.t.bin_off + e);
      const float2 f = Zs[v & 0x7fffu];
      const float a = sqrt_approx(fmaf(f.x, f.x, f.y * f.y));
      acc += (v & 0x8000u) ? a : 2.0f * a;
    }
    acc = warp_sum(acc);
    if (lane == 0) s_div[b] = (b == 0) ? 1.0f : __fdiv_rn(__ldg(P.t.bin_count + b), acc);
  }
  // The DC term (bin 0, left as it is) over N^2 is the image mean; it is
  // taken out of every pixel in pass E, so the float32 plane-fit and variance
  // sums run on centred values.
  const float scale_e = (float)(1.0 / ((double)N * (double)N));
  if (tid == 0) S.mu = Z.half(0, 0).x * scale_e;
  __syncthreads();

  // ---- pass D: radial divisor on load, inverse column transforms; the real
  // parts of the DC and the Nyquist column are column 0's two halves again (the
  // imaginary parts are dropped, as the real part of the reference's ifft2 does)
  for (int grp = warp; grp < CG; grp += NW) {
    const int c0 = grp * G;
    auto scaled = [&](float2 f, int i, int k) {
      const int ky = i < N / 2 ? i : i - N;
      return cscale(f, s_div[(int)rintf(sqrt_approx((float)(ky * ky + k * k)))]);
    };
    if (grp == 0)
      line_fft_warp<N, 1, 1>(Q, tw, [&](int, int i) { return scaled(nyq[i], i, N / 2); },
                             [&](int, int i, float2 v) { nyq[i] = v; });
    line_fft_warp<N, 1>(PairCols<N>{Z, c0}, tw, [&](int g, int i) { return scaled(Z.half(i, c0 + g), i, c0 + g); },
                        [&](int g, int i, float2 v) {
                          Z.half(i, c0 + g) = c0 + g == 0 ? make_float2(v.x, nyq[i].x) : v;
                        });
  }
  __syncthreads();

  // ---- pass E: inverse row transforms of the pairs, z = A + i B over the
  // Hermitian extensions of the half spectra, so that the result's halves are
  // the two rows; centred pixels and the plane-fit sums
  const float mu = S.mu;
  float fz = 0.f, fxz = 0.f, fyz = 0.f, fww = 0.f;
  for (int grp = warp; grp < RG; grp += NW) {
    const PairRows<N> R{Z, grp};
    line_fft_warp<N, 1>(
        R, tw,
        [&](int g, int j) {
          const int k = j <= N / 2 ? (j == N / 2 ? 0 : j) : N - j;
          const float2 a = R.at(g, k), b = R.at(g, N / 2 + k);
          if (j == 0) return make_float2(a.x, b.x);
          if (j == N / 2) return make_float2(a.y, b.y);
          return j < N / 2 ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, b.x - a.y);
        },
        [&](int g, int j, float2 z) {
          const int i1 = 2 * R.row(g);
          const float wa = fmaf(z.x, scale_e, -mu), wb = fmaf(z.y, scale_e, -mu);
          R.at(g, j) = make_float2(wa, wb);
          fz += wa + wb;
          fxz = fmaf((float)i1, wa, fmaf((float)(i1 + 1), wb, fxz));
          fyz = fmaf((float)j, wa + wb, fyz);
          fww = fmaf(wa, wa, fmaf(wb, wb, fww));
        });
  }
  // Least-squares plane over the full N x N grid in closed form: the grid is
  // a Cartesian product, so the centred row and column coordinates are
  // orthogonal and the normal equations of the reference's 3x3 solve
  // (rows as x, columns as y) decouple.
  const float4 s4 = block_sum_f4<NW>(make_float4(fz, fxz, fyz, fww), S.red4);
  constexpr float kMid = 0.5f * (float)(N - 1);
  constexpr float kSii = (float)((double)N * (double)N * ((double)N * (double)N - 1.0) / 12.0);
  const float pc0 = (s4.y - kMid * s4.x) / kSii;
  const float pc1 = (s4.z - kMid * s4.x) / kSii;
  const float pcm = s4.x * scale_e - (pc0 + pc1) * kMid;
  // Residual energy of the least-squares plane: sum (w - P)^2 = sum w^2 -
  // sum P w (the normal equations make the residual orthogonal to P). The
  // pixels are centred, so sum w^2 carries no DC term; where the plane
  // holds most of the energy the subtraction would cancel, and the residual
  // is summed directly instead (a block-uniform choice).
  float ssr = s4.w - fmaf(pc0, s4.y, fmaf(pc1, s4.z, pcm * s4.x));
  if (!(ssr > 0.25f * s4.w)) {
    float fsv = 0.f;
    for (int t = tid; t < N * N / 2; t += NT) {
      const int q = t / N, j = t - q * N;
      const float2 z = Z.at(q, j);
      const float pj = fmaf(pc1, (float)j, pcm);
      const float a = z.x - fmaf(pc0, (float)(2 * q), pj), b = z.y - fmaf(pc0, (float)(2 * q + 1), pj);
      fsv = fmaf(a, a, fmaf(b, b, fsv));
    }
    ssr = block_sum_f<NW>(fsv, S.red);
  }
  const float sd = sqrtf(ssr * scale_e);
  const float inv_sd = sd > 1e-12f ? 1.0f / sd : 1.0f;

  // ---- pass F: normalise and mask on load, forward row transforms
  for (int grp = warp; grp < RG; grp += NW) {
    const PairRows<N> R{Z, grp};
    line_fft_warp<N, -1>(
        R, tw,
        [&](int g, int j) {
          const int i1 = 2 * R.row(g);
          const float2 z = R.at(g, j);
          const float pj = fmaf(pc1, (float)j, pcm);
          float2 f = make_float2((z.x - fmaf(pc0, (float)i1, pj)) * inv_sd,
                                 (z.y - fmaf(pc0, (float)(i1 + 1), pj)) * inv_sd);
          if (P.mask != nullptr) {
            f.x *= __ldg(P.mask + i1 * N + j);
            f.y *= __ldg(P.mask + (i1 + 1) * N + j);
          }
          return f;
        },
        [&](int g, int j, float2 v) { R.at(g, j) = v; });
    pair_split_rows<N>(R);
  }
  __syncthreads();
  // ---- pass G: forward column transforms
  forward_columns();
  __syncthreads();
  // crop + FSC in place (packed column nb / 2 in nyq), L2 norm (float32 per
  // thread, fixed tree across the block), pre-shifted write
  const int hb = nb / 2;
  float fss = 0.f;
  for (int r = warp; r < nb; r += NW) {
    const int i = r < hb ? r : r + N - nb;
#pragma unroll 2
    for (int c = lane; c < hb; c += 32) {
      const float2 f = cscale(Z.half(i, c), __ldg(P.fsc + r * H + c));
      Z.half(i, c) = f;
      fss = fmaf(f.x, f.x, fmaf(f.y, f.y, fss));
    }
  }
  for (int r = tid; r < nb; r += NT) {
    const int i = r < hb ? r : r + N - nb;
    // cropped: the packed column is the negative frequency -nb / 2
    const float2 z = nb == N ? nyq[i] : cconj(Z.half(i == 0 ? 0 : N - i, hb));
    const float2 f = cscale(z, __ldg(P.fsc + r * H + hb));
    nyq[r] = f;
    fss = fmaf(f.x, f.x, fmaf(f.y, f.y, fss));
  }
  const float inv_norm = 1.0f / sqrtf(block_sum_f<NW>(fss, S.red));  // its barrier: every value is in place
  float2* out = P.bank + (size_t)slot * nb * H;
  for (int r = warp; r < nb; r += NW) {
    const int i = r < hb ? r : r + N - nb, rs = r < hb ? r + hb : r - hb;
#pragma unroll 2
    for (int c = lane; c <= hb; c += 32) {
      const int cs = c + H / 2 < H ? c + H / 2 : c + H / 2 - H;
      out[rs * H + cs] = cscale(c < hb ? Z.half(i, c) : nyq[r], inv_norm);
    }
  }
}

// Boxes 32, 64 and 128: one template per CTA, its plane written by rows_inverse.
template <int N>
__global__ void __launch_bounds__(tail_threads<N>(), tail_ctas<N>()) template_tail(ProjParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TailShared<N> S;
  float2* Zs = reinterpret_cast<float2*>(smem_raw);
  float* s_div = reinterpret_cast<float*>(Zs + pair_elems(N) + N);
  const int b = blockIdx.x;
  const float2* rows = P.planes + (size_t)b * N * plane_out_ld(N);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    rows_load<N>(Zs, rows, &S.bar);
  }
  tail_tables<N>(P.t, S);
  __syncthreads();
  const int dir = P.dirs[b], slot = P.out_slot ? P.out_slot[b] : dir;
  const bool ok = plane_wait(&S.bar, 0, P.wait_limit);
  if (__syncthreads_or(!ok)) {
    // rows that did not arrive in time: the status word reports it; the copies
    // still in flight get the default bound to land before the CTA's shared
    // memory is released; the template becomes NaN, so every score computed
    // from it is NaN
    if (threadIdx.x == 0) {
      if (P.status != nullptr) atomicExch(P.status, 1);
      plane_wait(&S.bar, 0, kPlaneWaitLimit);
    }
    __syncthreads();
    const float nan = __int_as_float(0x7fc00000);
    const int total = P.nb * (P.nb / 2 + 1);
    for (int t = threadIdx.x; t < total; t += blockDim.x) P.bank[(size_t)slot * total + t] = make_float2(nan, nan);
    return;
  }
  tail_passes<N>(P, rows, slot, Zs, s_div, S);
}

}  // namespace

// complex elements of the blocked copy of one [2N][2N][N+1] spectrum
size_t project_blocked_elems(int N) { return (size_t)4 * N * N * ((N + 1 + kBX - 1) / kBX) * kBX; }

// Dynamic shared memory of a tail CTA: plane, Nyquist column, divisors.
static size_t tail_smem_bytes(int N, int n_bins) {
  return (size_t)(pair_elems(N) + N) * sizeof(float2) + (size_t)n_bins * sizeof(float);
}

template <int N>
static cudaError_t launch_planes(ProjParams P, float2* planes, float2* blocked, cudaStream_t st) {
  constexpr int CC = ri_cols<N>();
  cudaError_t e = cudaSuccess;
  if (P.spectrum != nullptr) {  // else the blocked copy was written by the volume transform
    spectrum_blocked<N><<<8 * 152, 256, 0, st>>>(P.spectrum, blocked);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  rows_inverse<N><<<dim3((N + 1 + CC - 1) / CC, P.n_build), kRiWarps * 32, 0, st>>>(blocked, P.rot, P.dirs, P.t,
                                                                                      planes);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  P.planes = planes;
  static SmemLimit limit;
  const size_t smem = tail_smem_bytes(N, P.t.n_bins);
  e = allow_smem(template_tail<N>, smem, limit);
  if (e != cudaSuccess) return e;
  template_tail<N><<<P.n_build, tail_threads<N>(), smem, st>>>(P);
  return cudaGetLastError();
}

template <int N>
static cudaError_t launch_general(const ProjParams& P, int grid, cudaStream_t st) {
  static SmemLimit limit;
  const size_t smem = general_smem_bytes(N, P.t.n_bins);
  const cudaError_t e = allow_smem(project_templates<N>, smem, limit);
  if (e != cudaSuccess) return e;
  project_templates<N><<<grid, kThreads, smem, st>>>(P);
  return cudaGetLastError();
}

// Boxes 32, 64 and 128: the blocked copy (when a spectrum is given), the gather
// and the tail; boxes 96 and 192: one kernel on the cuFFT spectrum.
cudaError_t launch_project_templates(cudaStream_t st, const float2* spectrum, const float* rot, const int* dirs,
                                     int n_build, const int* out_slot, const float* mask, const float* fsc,
                                     const ProjTables& t, float2* bank, float2* scratch, int grid, int N, int nb,
                                     float2* planes, float2* blocked, int* status, unsigned wait_limit) {
  if (n_build <= 0) return cudaSuccess;
  ProjParams P;
  P.spectrum = spectrum; P.rot = rot; P.dirs = dirs; P.n_build = n_build; P.mask = mask; P.fsc = fsc; P.t = t;
  P.bank = bank; P.out_slot = out_slot; P.scratch = scratch; P.scratch_stride = project_scratch_elems(N, nb);
  P.status = status; P.wait_limit = wait_limit; P.planes = nullptr; P.N = N; P.nb = nb;
  if ((N == 32 || N == 64 || N == 128) && n_build > 65535) return cudaErrorInvalidValue;
  switch (N) {
    case 32: return launch_planes<32>(P, planes, blocked, st);
    case 64: return launch_planes<64>(P, planes, blocked, st);
    case 128: return launch_planes<128>(P, planes, blocked, st);
    case 96: return launch_general<96>(P, grid, st);
    case 192: return launch_general<192>(P, grid, st);
    default: return cudaErrorInvalidValue;  // box 256: launch_project_templates_planes
  }
}

// Box 256: the slice gather and pass A run in rows_inverse from the blocked
// spectrum (its plane [N][N+1] written to global memory, ``chunk`` templates
// at a time), passes B-G in the general kernel, which reads those planes.
cudaError_t launch_project_templates_planes(cudaStream_t st, const float2* spectrum, const float* rot,
                                            const int* dirs, int n_build, const int* out_slot,
                                            const float* mask, const float* fsc, const ProjTables& t,
                                            float2* bank, float2* scratch, int grid, int N, int nb, float2* planes,
                                            float2* blocked, int chunk) {
  constexpr int kN = 256, CC = ri_cols<kN>();
  if (n_build <= 0) return cudaSuccess;
  if (N != kN || chunk <= 0 || chunk > 65535 || grid <= 0) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (spectrum != nullptr) {  // else the blocked copy was written by the volume transform
    spectrum_blocked<kN><<<8 * 152, 256, 0, st>>>(spectrum, blocked);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  ProjParams P;
  P.status = nullptr; P.wait_limit = 0;
  P.spectrum = spectrum; P.rot = rot; P.mask = mask; P.fsc = fsc; P.t = t; P.bank = bank; P.scratch = scratch;
  P.scratch_stride = project_scratch_elems(N, nb); P.N = N; P.nb = nb; P.planes = planes;
  for (int b0 = 0; b0 < n_build; b0 += chunk) {
    const int n = min(chunk, n_build - b0);
    rows_inverse<kN><<<dim3((kN + 1 + CC - 1) / CC, n), kRiWarps * 32, 0, st>>>(blocked, rot, dirs + b0, t,
                                                                                 planes);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    P.dirs = dirs + b0; P.out_slot = out_slot ? out_slot + b0 : nullptr; P.n_build = n;
    e = launch_general<kN>(P, min(grid, n), st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
