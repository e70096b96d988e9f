// Two-dimensional transforms of a real N x N image held in one CTA's shared
// memory as N/2 complex lines, shared by the particle preparation
// (particles.cu) and the template tail (project.cu).
//
// Line q holds z = a + i b for the real rows a = 2q and b = 2q + 1. After the
// forward row transform, pair_split turns each line into the half spectra of
// its two rows, in place: row 2q at positions 0..N/2-1, row 2q + 1 at N/2..N-1,
// and the two real coefficients k = 0 and k = N/2 of a row packed as (DC,
// Nyquist) at its position 0. The plane therefore never grows past N/2 x N
// complex values (75 KB at N = 128, against 173 KB for N rows of N + 1), which
// is what lets several images be in flight per SM. A column of the half plane
// is then the N values at (i >> 1, k + (i & 1) N/2); column 0 carries the DC
// column as its real part and the Nyquist column as its imaginary part through
// the column transform, and col0_split takes the two apart.
//
// Layout: one spare slot after every 8 elements of a line, line stride a
// multiple of 16 plus 2, and one more slot every 4 lines: the four-step loads
// and stores of a half warp, along lines and along columns, then fall on
// distinct 8-byte bank pairs at N = 128 (but for one pair in the row pass).
#pragma once

#include "common.cuh"

// ---------------------------------------------------------------------------
// Codelets of length 3, 6 and 12 (boxes 96 and 192), as dft<R, DIR>.
// ---------------------------------------------------------------------------
template <int DIR>
GISAPR_DEV void dft3(float2& a, float2& b, float2& c) {
  constexpr float kS = 0.86602540378443864676f;  // sin(pi/3)
  const float2 s = cadd(b, c), d = cscale(csub(b, c), kS);
  const float2 h = make_float2(a.x - 0.5f * s.x, a.y - 0.5f * s.y), t = mul_dir_i<DIR>(d);
  a = cadd(a, s);
  b = cadd(h, t);
  c = csub(h, t);
}

// exp(DIR * i * k * pi / 6), k = 0..11 known at compile time
template <int DIR>
GISAPR_DEV float2 w12(int k) {
  constexpr float kC = 0.86602540378443864676f;
  float c = 1.f, s = 0.f;
  switch (k % 12) {
    case 1: c = kC; s = 0.5f; break;
    case 2: c = 0.5f; s = kC; break;
    case 3: c = 0.f; s = 1.f; break;
    case 4: c = -0.5f; s = kC; break;
    case 5: c = -kC; s = 0.5f; break;
    case 6: c = -1.f; break;
    case 7: c = -kC; s = -0.5f; break;
    case 8: c = -0.5f; s = -kC; break;
    case 9: c = 0.f; s = -1.f; break;
    case 10: c = 0.5f; s = -kC; break;
    case 11: c = kC; s = -0.5f; break;
    default: break;
  }
  return make_float2(c, DIR > 0 ? s : -s);
}

// 6 = 2 x 3: n = 3 n1 + n2, k = k1 + 2 k2
template <int DIR>
GISAPR_DEV void dft6_impl(float2 (&x)[6]) {
#pragma unroll
  for (int n2 = 0; n2 < 3; ++n2) dft2<DIR>(x[n2], x[n2 + 3]);  // x[n2 + 3 k1] = A[n2][k1]
  x[4] = cmul(x[4], w12<DIR>(2));
  x[5] = cmul(x[5], w12<DIR>(4));
  dft3<DIR>(x[0], x[1], x[2]);  // k1 = 0 -> X[0], X[2], X[4]
  dft3<DIR>(x[3], x[4], x[5]);  // k1 = 1 -> X[1], X[3], X[5]
  const float2 y[6] = {x[0], x[3], x[1], x[4], x[2], x[5]};
#pragma unroll
  for (int k = 0; k < 6; ++k) x[k] = y[k];
}
template <>
GISAPR_DEV void dft<6, 1>(float2 (&x)[6]) { dft6_impl<1>(x); }
template <>
GISAPR_DEV void dft<6, -1>(float2 (&x)[6]) { dft6_impl<-1>(x); }

// 12 = 3 x 4: n = 4 n1 + n2, k = k1 + 3 k2
template <int DIR>
GISAPR_DEV void dft12_impl(float2 (&x)[12]) {
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) dft3<DIR>(x[n2], x[n2 + 4], x[n2 + 8]);  // x[n2 + 4 k1] = A[n2][k1]
#pragma unroll
  for (int n2 = 1; n2 < 4; ++n2)
#pragma unroll
    for (int k1 = 1; k1 < 3; ++k1) x[n2 + 4 * k1] = cmul(x[n2 + 4 * k1], w12<DIR>(n2 * k1));
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) dft4<DIR>(x[4 * k1], x[4 * k1 + 1], x[4 * k1 + 2], x[4 * k1 + 3]);
  float2 y[12];
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) y[k1 + 3 * k2] = x[4 * k1 + k2];
#pragma unroll
  for (int k = 0; k < 12; ++k) x[k] = y[k];
}
template <>
GISAPR_DEV void dft<12, 1>(float2 (&x)[12]) { dft12_impl<1>(x); }
template <>
GISAPR_DEV void dft<12, -1>(float2 (&x)[12]) { dft12_impl<-1>(x); }

// ---------------------------------------------------------------------------
// Warp FFTs of N = 16 * (N / 16) points, N = 32, 64, 96, 128, 192 or 256.
// ---------------------------------------------------------------------------

// lines one warp transforms at once
template <int N>
__host__ __device__ constexpr int fft_lines() { return N == 96 ? 4 : (N == 192 ? 2 : 32 / (N / 16)); }

// The twiddles between the two steps, exp(-2 pi i n2 k1 / N), in the order the
// lanes of a warp read them (entry k1 N/16 + n2): one conflict-free load each,
// where a table by exponent put a warp's eight on two to eight banks.
template <int N>
__host__ __device__ constexpr int twiddle_exponent(int entry) { return (entry / (N / 16)) * (entry % (N / 16)); }

// One warp's four-step transform of fft_lines<N>() lines, natural order in
// and out: 16-point codelets over n1, twiddles, N/16-point codelets over n2.
// ``load(g, k)`` gives element k of line g, L.at holds the values between the
// two steps, ``store(g, k, v)`` takes the result. A load may read any element of
// the warp's lines (all loads come before the first write). LINES: fewer lines.
// ``tw`` is the table of twiddle_exponent, in shared memory; ``mul`` multiplies
// by its entries.
struct CMul {
  GISAPR_DEV float2 operator()(float2 a, float2 w) const { return cmul(a, w); }
};
template <int N, int DIR, int LINES = 0, class Lines, class Load, class Store, class Mul = CMul>
GISAPR_DEV void line_fft_warp(const Lines& L, const float2* tw, const Load& load, const Store& store,
                              const Mul& mul = Mul()) {
  constexpr int L2 = N / 16, G = LINES ? LINES : fft_lines<N>(), T = (G * 16 + 31) / 32;
  const int lane = threadIdx.x & 31;
  {
    const int g = lane / L2, n2 = lane % L2;
    float2 x[16];
    if (G * L2 == 32 || g < G) {
#pragma unroll
      for (int n1 = 0; n1 < 16; ++n1) x[n1] = load(g, L2 * n1 + n2);
      dft<16, DIR>(x);
    }
    __syncwarp();
    if (G * L2 == 32 || g < G) {
      L.at(g, n2) = x[0];
#pragma unroll
      for (int k1 = 1; k1 < 16; ++k1) {
        const float2 w = tw[k1 * L2 + n2];
        L.at(g, L2 * k1 + n2) = mul(x[k1], DIR < 0 ? w : cconj(w));
      }
    }
  }
  __syncwarp();
  float2 y[T][L2];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int task = lane + 32 * t, g = task / 16, k1 = task % 16;
    if (G * 16 % 32 == 0 || g < G) {
#pragma unroll
      for (int n2 = 0; n2 < L2; ++n2) y[t][n2] = L.at(g, L2 * k1 + n2);
      dft<L2, DIR>(y[t]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int task = lane + 32 * t, g = task / 16, k1 = task % 16;
    if (G * 16 % 32 == 0 || g < G) {
#pragma unroll
      for (int k2 = 0; k2 < L2; ++k2) store(g, k1 + 16 * k2, y[t][k2]);
    }
  }
  __syncwarp();
}

// The same in place.
template <int N, int DIR, class Lines>
GISAPR_DEV void line_fft_warp(const Lines& L, const float2* tw) {
  line_fft_warp<N, DIR>(L, tw, [&](int g, int k) { return L.at(g, k); },
                        [&](int g, int k, float2 v) { L.at(g, k) = v; });
}

// Staging lines of one warp (powers of two): element k of a line at
// k ^ (its row of 16), line stride N + N/16 and four slots more every two lines:
// the loads and stores of both steps, and the slice gather's, fall on distinct
// banks at N = 128.
__host__ __device__ constexpr int stage_ld(int N) { return N + N / 16; }
__host__ __device__ constexpr int stage_elems(int N, int lines) { return lines * stage_ld(N) + 2 * lines; }
template <int N>
struct StagedLines {
  float2* p;
  GISAPR_DEV static int slot(int k) { return k ^ ((k >> 4) & (N / 16 - 1)); }
  GISAPR_DEV float2* line(int g) const { return p + g * stage_ld(N) + (g >> 1) * 4; }
  GISAPR_DEV float2& at(int g, int k) const { return line(g)[slot(k)]; }
};

// exp(-2 pi i t / N), from the context's two tables
template <int N>
GISAPR_DEV float2 twiddle_of(const float2* __restrict__ tw, const float2* __restrict__ tw3, int t) {
  if constexpr ((N & (N - 1)) == 0) return tw_full<-1>(tw, t, N);
  return tw3[t * (kMaxFftLen3 / N)];
}

// ---------------------------------------------------------------------------
// The plane
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int pair_ld(int N) { return ((N + N / 8 + 13) / 16) * 16 + 2; }
__host__ __device__ constexpr int pair_elems(int N) { return (N / 2) * pair_ld(N) + N / 8; }

template <int N>
struct PairPlane {
  float2* p;
  GISAPR_DEV float2& at(int q, int j) const { return p[q * pair_ld(N) + (q >> 2) + j + (j >> 3)]; }
  // element (row i, column k < N/2) of the half plane
  GISAPR_DEV float2& half(int i, int k) const { return at(i >> 1, k + (i & 1) * (N / 2)); }
};

// Line g of row group ``grp``: lines 4 apart where the group count allows it
// (rows 4 apart fall on other banks), else consecutive ones.
template <int N>
struct PairRows {
  PairPlane<N> pl;
  int grp;
  static constexpr int G = fft_lines<N>();
  static constexpr bool kApart = (N / 2) % (4 * G) == 0;
  GISAPR_DEV int row(int g) const { return kApart ? (grp & 3) + (grp >> 2) * 4 * G + 4 * g : grp * G + g; }
  GISAPR_DEV float2& at(int g, int k) const { return pl.at(row(g), k); }
};
template <int N>
__host__ __device__ constexpr int pair_row_groups() { return (N / 2) / fft_lines<N>(); }

template <int N>
struct PairCols {
  PairPlane<N> pl;
  int c0;
  GISAPR_DEV float2& at(int g, int i) const { return pl.half(i, c0 + g); }
};
template <int N>
__host__ __device__ constexpr int pair_col_groups() { return (N / 2) / fft_lines<N>(); }

// Splits the transformed lines of one row group (see the top of the file).
// A task owns positions k, N/2 - k, N/2 + k and N - k of its line and reads
// and writes nothing else, so the split runs in place. One warp.
template <int N>
GISAPR_DEV void pair_split_rows(const PairRows<N>& R) {
  constexpr int Q = N / 4, G = fft_lines<N>();
  for (int idx = threadIdx.x & 31; idx < G * (Q + 1); idx += 32) {
    const int g = idx / (Q + 1), k = idx - g * (Q + 1);
    const float2 z1 = R.at(g, k);
    if (k == 0) {
      const float2 zh = R.at(g, N / 2);
      R.at(g, 0) = make_float2(z1.x, zh.x);
      R.at(g, N / 2) = make_float2(z1.y, zh.y);
    } else {
      const float2 zn = R.at(g, N - k);
      const float2 a = make_float2(0.5f * (z1.x + zn.x), 0.5f * (z1.y - zn.y));
      const float2 b = make_float2(0.5f * (z1.y + zn.y), 0.5f * (zn.x - z1.x));
      if (k == Q) {
        R.at(g, Q) = a;
        R.at(g, N - Q) = b;
      } else {
        const float2 y1 = R.at(g, N / 2 - k), yn = R.at(g, N / 2 + k);
        R.at(g, k) = a;
        R.at(g, N / 2 + k) = b;
        R.at(g, N / 2 - k) = make_float2(0.5f * (y1.x + yn.x), 0.5f * (y1.y - yn.y));
        R.at(g, N - k) = make_float2(0.5f * (y1.y + yn.y), 0.5f * (yn.x - y1.x));
      }
    }
  }
  __syncwarp();
}

// After the transform of column 0, takes the DC column (left in place) and the
// Nyquist column (to nyq[N]) apart: D(i) = (Z(i) + conj Z(-i)) / 2, Q(i) =
// (Z(i) - conj Z(-i)) / 2i. One warp; a task owns rows i and N - i.
template <int N>
GISAPR_DEV void col0_split(const PairPlane<N>& Z, float2* nyq) {
  for (int i = threadIdx.x & 31; i <= N / 2; i += 32) {
    const int o = i == 0 ? 0 : N - i;
    const float2 a = Z.half(i, 0), b = Z.half(o, 0);
    const float2 d = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
    const float2 q = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
    Z.half(i, 0) = d;
    Z.half(o, 0) = cconj(d);
    nyq[i] = q;
    nyq[o] = cconj(q);
  }
  __syncwarp();
}
