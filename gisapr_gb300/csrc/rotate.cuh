// The rotation of a particle image: source coordinates and bilinear sample in the
// float32 operations, order and roundings of affine_grid and grid_sample on the CPU
// (align_corners=True, zero padding; torch's vectorised 2-D kernel).
#pragma once

#include "common.cuh"

__device__ __forceinline__ float sample_bilinear_zero(const float* __restrict__ img, int N,
                                                      float iy, float ix) {
  const float fy = floorf(iy), fx = floorf(ix);
  const int y0 = (int)fy, x0 = (int)fx;
  const float w = __fsub_rn(ix, fx), e = __fsub_rn(1.0f, w);
  const float nn = __fsub_rn(iy, fy), s = __fsub_rn(1.0f, nn);
  const float wnw = __fmul_rn(s, e), wne = __fmul_rn(s, w);
  const float wsw = __fmul_rn(nn, e), wse = __fmul_rn(nn, w);
  auto at = [&](int yy, int xx) -> float {
    return (yy >= 0 && yy < N && xx >= 0 && xx < N) ? __ldg(img + (size_t)yy * N + xx) : 0.0f;
  };
  float acc = __fmul_rn(at(y0, x0), wnw);
  acc = __fadd_rn(acc, __fmul_rn(at(y0, x0 + 1), wne));
  acc = __fadd_rn(acc, __fmul_rn(at(y0 + 1, x0), wsw));
  acc = __fadd_rn(acc, __fmul_rn(at(y0 + 1, x0 + 1), wse));
  return acc;
}

// A staged image has a border of two zero pixels for the padding and rows of
// image_ld elements.
constexpr int kBorder = 2;
template <int N>
__host__ __device__ constexpr int image_ld() { return N + 9; }

// a / (N - 1), correctly rounded: one Newton correction of a * RN(1 / (N - 1))
// (Markstein's theorem; the remainder is exact in the fused multiply-add).
template <int N>
GISAPR_DEV float2 div_nm1(float2 a) {
  constexpr float d = (float)(N - 1), r = 1.0f / (float)(N - 1);
  const float2 q = mul2(a, dup2(r));
  return fma2(fma2(q, dup2(-d), a), dup2(r), q);
}

GISAPR_DEV float small_to_float(int i) {  // 0 <= i < 2^23, FP32 pipe
  return __int_as_float(0x4B000000 | i) - 8388608.0f;
}

// Packed product for a packed sum. A plain one may be fused into the sum (the
// assembler does), and then neither the floor and the fraction of a coordinate nor
// the sample's terms have the roundings they should; adding zero rounds nothing
// and leaves only a sum of sums (749 us for 6,000 spectra of box 128, 744 with
// plain products).
GISAPR_DEV float2 mul_alone(float2 a, float2 b) { return fma2(a, b, dup2(0.0f)); }

// Pixels (2 q, j) and (2 q + 1, j) of the image rotated by ``ps`` (cos, sin, offset
// of the row, of the column), as the halves of packed operations. ``img`` is staged
// (its first border pixel), or the image itself.
template <int N, bool STAGED>
GISAPR_DEV float2 rotated_pair(const float* img, float4 ps, int q, int j) {
  constexpr float half = 0.5f * (float)(N - 1);
  const float cth = ps.x, sth = ps.y;
  const float xx = small_to_float(j), y0f = small_to_float(2 * q);
  const float2 yy = make_float2(y0f, y0f + 1.0f);
  // source = [row, col] @ M^T + offset; M = [[c, -s], [s, c]]
  const float2 sy = add2(fma2(dup2(-sth), dup2(xx), mul2(dup2(cth), yy)), dup2(ps.z));
  const float2 sx = add2(fma2(dup2(cth), dup2(xx), mul2(dup2(sth), yy)), dup2(ps.w));
  const float2 yn = add2(div_nm1<N>(mul2(dup2(2.0f), sy)), dup2(-1.0f));
  const float2 xn = add2(div_nm1<N>(mul2(dup2(2.0f), sx)), dup2(-1.0f));
  const float2 iy = mul_alone(add2(yn, dup2(1.0f)), dup2(half)), ix = mul_alone(add2(xn, dup2(1.0f)), dup2(half));
  if constexpr (!STAGED) {
    return make_float2(sample_bilinear_zero(img, N, iy.x, ix.x), sample_bilinear_zero(img, N, iy.y, ix.y));
  } else {
    constexpr int ILD = image_ld<N>();
    // floor by adding 1.5 * 2^23 rounded down: the sum's low bits are the
    // integer, clamped as they are (the bits of positive floats are ordered)
    constexpr float kMagic = 12582912.0f;
    constexpr int kZero = 0x4B400000;  // the bits of kMagic
    const float2 ry = add2_down(iy, dup2(kMagic)), rx = add2_down(ix, dup2(kMagic));
    const float2 fy = add2(ry, dup2(-kMagic)), fx = add2(rx, dup2(-kMagic));
    const float2 w = sub2(ix, fx), ea = sub2(dup2(1.0f), w);
    const float2 nn = sub2(iy, fy), s = sub2(dup2(1.0f), nn);
    auto at = [&](float yb, float xb) {
      const int y0 = min(max(__float_as_int(yb), kZero - kBorder), kZero + N);
      const int x0 = min(max(__float_as_int(xb), kZero - kBorder), kZero + N);
      return img + ((y0 - kZero + kBorder) * ILD + (x0 - kZero + kBorder));
    };
    const float* a = at(ry.x, rx.x);
    const float* b = at(ry.y, rx.y);
    float2 v = mul_alone(make_float2(a[0], b[0]), mul2(s, ea));
    v = add2(v, mul_alone(make_float2(a[1], b[1]), mul2(s, w)));
    v = add2(v, mul_alone(make_float2(a[ILD], b[ILD]), mul2(nn, ea)));
    return add2(v, mul_alone(make_float2(a[ILD + 1], b[ILD + 1]), mul2(nn, w)));
  }
}
