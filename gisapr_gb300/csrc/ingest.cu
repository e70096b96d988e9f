// Particle stack preparation (read_star_shift_crop_and_generate_new_star_v5.py).
//
// One batched pipeline per stack chunk, in float64 as the reference's numpy
// code computes it:
//   load       integer shift (zero fill) and centred crop, one element per
//              thread, as float64 rows padded to 2 (cw/2 + 1) values;
//   spectrum   one real-to-complex 2-D transform per image (cuFFT D2Z, batched,
//              in place), everything in the half spectrum by one CTA per image,
//              and one inverse (Z2D):
//     whiten     the mean |F| of every radial bin (round(distance) on the
//                centred grid) and F *= 1 / mean (bin 0 keeps 1) (v5:42-59). The
//                bins come as a CSR list of pixels per bin, built once on the
//                host; a bin is summed with a fixed lane order and shuffle tree;
//     normalize  least-squares plane over (column, row, value), subtracted, then
//                (v - mean) / population sigma when sigma > 0 (v5:61-106). The
//                sums of v, x v and y v are sums over the spectrum's two axes
//                (the transform of a ramp lives there), and so is the plane that
//                is taken out; the sum of v^2 is Parseval's;
//     highpass   times the raised-cosine edge mask (a host table) (v5:107-134);
//   normalize  alone: on the pixels, one CTA per image;
//   store      the result as float32.
// The transforms are what it costs: GB300 computes FP64 at 1/64 of its FP32
// rate, and they run at that limit. Real data in place of complex and one pair
// of transforms in place of two (whitening and high-pass each had its own) cut
// them to a quarter. Measured on GB300, 500 images of 256 cropped to 128,
// whitened and high-passed: 5.47 -> 1.89 ms (1.25 of it the transforms).
#include "common.cuh"

namespace {

constexpr int kIngestThreads = 256;
constexpr int kSpectrumThreads = 512;

// round(distance from the origin) of a pixel of the unshifted grid; y and x are
// distances along the axes. No distance is half way between two integers.
__device__ __forceinline__ int radius_bin(int y, int x) {
  const long long d4 = 4 * ((long long)y * y + (long long)x * x);
  int b = __float2int_rn(sqrtf(0.25f * (float)d4));
  const long long up = 2LL * b + 1, down = 2LL * b - 1;
  if (up * up < d4) ++b;
  else if (b > 0 && down * down > d4) --b;
  return b;
}

// What the spectrum kernel has to know of the caller's tables. bins_other and
// mask_other hold the call's number if the bins are not the radial ones (in the
// order of their lists or in number), if the mask is not its own mirror image.
struct TableNotes {
  const int* bin_ptr;      // null: no whitening
  const int* bin_pix;
  int n_bins;
  const double* mask;      // or null
  int call;
  int* bins_other;
  int* mask_other;
  int* entry;              // [ch * cw] where a listed pixel stands in bin_pix
};

__device__ __forceinline__ int mirrored(int k, int n) { return k == 0 ? 0 : n - k; }

// One pass over both tables by the threads of the load. An entry is where it
// should be if it lies in the list of its pixel's radius.
__device__ __forceinline__ void note_tables(const TableNotes& T, int ch, int cw, long long first, long long step) {
  if (T.bin_ptr != nullptr) {
    const int e0 = T.bin_ptr[0], e1 = T.bin_ptr[T.n_bins];
    if (first == 0 && e1 - e0 != ch * cw) *T.bins_other = T.call;
    for (long long e = e0 + first; e < e1; e += step) {
      const int p = T.bin_pix[e];
      if (p < 0 || p >= ch * cw) continue;
      T.entry[p] = (int)e;
      const int ky = p / cw, kx = p - ky * cw;
      const int b = min(radius_bin(min(ky, ch - ky), min(kx, cw - kx)), T.n_bins - 1);
      if (e < T.bin_ptr[b] || e >= T.bin_ptr[b + 1]) *T.bins_other = T.call;
    }
  }
  if (T.mask != nullptr)
    for (long long p = first; p < (long long)ch * cw; p += step) {
      const int ky = (int)(p / cw), kx = (int)(p - (long long)ky * cw);
      const double a = T.mask[p], b = T.mask[(size_t)mirrored(ky, ch) * cw + mirrored(kx, cw)];
      if (__double_as_longlong(a) != __double_as_longlong(b)) *T.mask_other = T.call;
    }
}

// ld: row stride of the result
__global__ void ingest_load(const float* __restrict__ images, int n, int h, int w, const int* __restrict__ shifts,
                            int ch, int cw, double* __restrict__ work, int ld, TableNotes T) {
  note_tables(T, ch, cw, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
  const long long total = (long long)n * ch * cw;
  const int y0 = h / 2 - ch / 2, x0 = w / 2 - cw / 2;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(t % cw), r = (int)((t / cw) % ch);
    const long long img = t / ((long long)ch * cw);
    const int tx = shifts ? shifts[2 * img] : 0, ty = shifts ? shifts[2 * img + 1] : 0;
    // translated[y][x] = image[y - ty][x - tx] inside the image, else 0
    const int sy = y0 + r - ty, sx = x0 + c - tx;
    double v = 0.0;
    if (sy >= 0 && sy < h && sx >= 0 && sx < w) v = (double)images[(img * h + sy) * w + sx];
    work[(t / cw) * ld + c] = v;
  }
}

__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum with a fixed tree (every thread gets the result).
__device__ double block_sum_d(double v, double* red) {
  v = warp_sum_d(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
  for (int k = 0; k < nw; ++k) t += red[k];
  return t;
}

struct PlaneSums {
  double D, E, F, G, H, I;  // sums of x^2, xy, x, y^2, y, 1 over the pixel grid
};

// Coefficients of the plane pa x + pb y + pc through the sums J = sum x z,
// K = sum y z, L = sum z (x = column, y = row).
__device__ __forceinline__ void plane_fit(const PlaneSums& ps, double J, double K, double L, double& pa, double& pb,
                                          double& pc) {
  const double D = ps.D, E = ps.E, F = ps.F, G = ps.G, H = ps.H, I = ps.I;
  const double denom = F * F * G - 2 * E * F * H + D * H * H + E * E * I - D * G * I;
  pa = (H * H * J - G * I * J + E * I * K + F * G * L - H * (F * K + E * L)) / denom;
  pb = (E * I * J + F * F * K - D * I * K + D * H * L - F * (H * J + E * L)) / denom;
  pc = (F * G * J - E * H * J - E * F * K + D * H * K + E * E * L - D * G * L) / denom;
}

// Plane fit, subtraction, mean and sigma normalisation of one image per CTA
// (v5:61-106). x = column, y = row.
__global__ void __launch_bounds__(kIngestThreads) ingest_normalize(double* __restrict__ work, int ch, int cw, int ld,
                                                                   PlaneSums ps) {
  __shared__ double red[kIngestThreads / 32];
  const int pixels = ch * cw;
  double* img = work + (size_t)blockIdx.x * ch * ld;
  double J = 0.0, K = 0.0, L = 0.0;
  for (int p = threadIdx.x; p < pixels; p += blockDim.x) {
    const int r = p / cw, c = p - r * cw;
    const double z = img[(size_t)r * ld + c], x = (double)c, y = (double)r;
    J = __dadd_rn(J, __dmul_rn(x, z));
    K = __dadd_rn(K, __dmul_rn(y, z));
    L = __dadd_rn(L, z);
  }
  J = block_sum_d(J, red);
  K = block_sum_d(K, red);
  L = block_sum_d(L, red);
  double pa, pb, pc;
  plane_fit(ps, J, K, L, pa, pb, pc);
  double s1 = 0.0, s2 = 0.0;
  for (int p = threadIdx.x; p < pixels; p += blockDim.x) {
    const int r = p / cw, c = p - r * cw;
    const double x = (double)c, y = (double)r;
    const double plane = __dadd_rn(__dadd_rn(__dmul_rn(pa, x), __dmul_rn(pb, y)), pc);
    const double v = __dsub_rn(img[(size_t)r * ld + c], plane);
    img[(size_t)r * ld + c] = v;
    s1 = __dadd_rn(s1, v);
    s2 = __dadd_rn(s2, __dmul_rn(v, v));
  }
  s1 = block_sum_d(s1, red);
  s2 = block_sum_d(s2, red);
  const double n = (double)pixels;
  const double ave = s1 / n;
  const double sd = sqrt(__dsub_rn(s2 / n, __dmul_rn(ave, ave)));
  if (sd > 0.0) {
    for (int p = threadIdx.x; p < pixels; p += blockDim.x) {
      double& v = img[(size_t)(p / cw) * ld + p % cw];
      v = (v - ave) / sd;
    }
  }
}

// Imaginary part of entry k of the transform of the ramp 0, 1, ..., n - 1
// (sum_j j exp(-2 pi i j k / n)), k > 0; the real part is -n/2, and entry 0 is
// n (n - 1) / 2.
__device__ __forceinline__ double ramp_imag(int k, int n) {
  double s, c;
  sincospi((double)k / (double)n, &s, &c);
  return 0.5 * (double)n * (c / s);
}

struct SpectrumSteps {
  const int* bin_ptr;       // null: no whitening
  const int* bin_pix;
  const double* bin_count;
  int n_bins;
  int normalize;
  PlaneSums plane;
  int ramps;                // the axes' ramp transforms are kept in shared memory
  int amplitudes;           // the half spectrum's |F| are kept there too
  const double* mask;       // [ch][cw] or null
  TableNotes notes;
};

// The steps of one image in its half spectrum [ch][cw/2 + 1], scaled by
// 1 / pixels for the inverse. Dynamic shared memory: n_bins doubles, cw/2 + 1 +
// ch of ramp transforms, ch (cw/2 + 1) amplitudes. With the amplitudes there, the
// spectrum is read and written in order, and only they are gathered bin by bin
// (gathering the spectrum itself took the latency of two dependent loads from
// memory an entry, 594 us for 500 spectra of 128 where this takes 475);
// larger spectra are gathered. A pixel of
// the full grid right of column cw/2 stands for its mirror, which has the same
// magnitude and, where bins and mask are radial, the same bin and mask value: the
// columns that have a mirror count twice.
//
// Bins and mask may be any (ANY: the bins are not the radial ones, or the mask is
// not its own mirror image). The result of a step is the real part of its inverse
// transform, that is, of a spectrum F(k) m(k) with real m the half of F(k) (m(k) +
// m(-k)): the mean of a factor and its mirror image's stands for both, and a bin's
// sum takes every pixel that it lists.
template <bool ANY>
__device__ __forceinline__ void spectrum_steps(double2* F, int ch, int cw, const SpectrumSteps& P, double* s_div,
                                               double* red) {
  const int hc = cw / 2 + 1, pixels = ch * cw;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const double inv = 1.0 / (double)pixels;
  auto doubled = [&](int kx) { return kx != 0 && 2 * kx != cw; };
  double* s_ramp = s_div + (P.bin_ptr != nullptr ? P.n_bins : 0);
  if (P.ramps && P.normalize)
    for (int k = threadIdx.x; k < hc + ch; k += blockDim.x) {
      const int j = k < hc ? k : k - hc;
      s_ramp[k] = j == 0 ? 0.0 : ramp_imag(j, k < hc ? cw : ch);
    }
  auto ramp_x = [&](int k) {
    return k == 0 ? make_double2(0.5 * (double)cw * (double)(cw - 1), 0.0)
                  : make_double2(-0.5 * (double)cw, P.ramps ? s_ramp[k] : ramp_imag(k, cw));
  };
  auto ramp_y = [&](int k) {
    return k == 0 ? make_double2(0.5 * (double)ch * (double)(ch - 1), 0.0)
                  : make_double2(-0.5 * (double)ch, P.ramps ? s_ramp[hc + k] : ramp_imag(k, ch));
  };
  double* s_amp = s_ramp + (P.ramps ? hc + ch : 0);
  if (P.amplitudes) {
    for (int t = threadIdx.x; t < ch * hc; t += blockDim.x) {
      const double2 f = F[t];
      s_amp[t] = sqrt_fp64(fma(f.x, f.x, f.y * f.y));
    }
    __syncthreads();
  }
  // the divisor of a pixel by its entry in the lists (an entry left by an earlier
  // call does not name the pixel), 1 if it has none
  auto listed = [&](int ky, int kx) {
    const int p = ky * cw + kx, e = P.notes.entry[p];
    if (e < P.bin_ptr[0] || e >= P.bin_ptr[P.n_bins] || P.bin_pix[e] != p) return 1.0;
    int lo = 0, hi = P.n_bins;  // the last bin that starts at e or before
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (P.bin_ptr[mid] <= e) lo = mid;
      else hi = mid;
    }
    return s_div[lo];
  };
  auto factor = [&](int ky, int kx) {
    return P.bin_ptr == nullptr ? 1.0 : 0.5 * (listed(ky, kx) + listed(mirrored(ky, ch), mirrored(kx, cw)));
  };
  double s2 = 0.0;  // this lane's part of the sum over the full grid of |V|^2, the axes added below
  for (int b = warp; P.bin_ptr != nullptr && b < P.n_bins; b += nw) {
    double s = 0.0, q = 0.0;
    for (int i = P.bin_ptr[b] + lane; i < P.bin_ptr[b + 1]; i += 32) {
      const int p = P.bin_pix[i];
      int ky = p / cw, kx = p - ky * cw;
      const bool right = kx >= hc;
      if (right) {
        if (!ANY) continue;
        ky = mirrored(ky, ch);
        kx = cw - kx;
      }
      double e, a;
      if (P.amplitudes) {
        a = s_amp[ky * hc + kx];
        e = a * a;
      } else {
        const double2 f = F[(size_t)ky * hc + kx];
        e = fma(f.x, f.x, f.y * f.y);
        a = sqrt_fp64(e);
      }
      s += !ANY && doubled(kx) ? 2.0 * a : a;
      if (!ANY && ky != 0 && kx != 0) q += doubled(kx) ? 2.0 * e : e;
    }
    s = warp_sum_d(s);
    const double d = (b == 0 || P.bin_count[b] <= 0.0) ? 1.0 : 1.0 / (s / P.bin_count[b]);
    if (!ANY) s2 = fma(d * d, q, s2);
    if (lane == 0) s_div[b] = d;
  }
  __syncthreads();
  auto divisor = [&](int bin) { return P.bin_ptr != nullptr ? s_div[min(bin, P.n_bins - 1)] : 1.0; };
  auto axis_y = [&](int ky) { return min(ky, ch - ky); };
  auto axis_divisor = [&](int ky, int kx) { return ANY ? factor(ky, kx) : divisor(ky == 0 ? kx : axis_y(ky)); };
  double pa = 0.0, pb = 0.0, pc = 0.0, scale = inv;
  bool centre = false;
  if (P.normalize) {
    if (ANY || P.bin_ptr == nullptr) {
      for (long long t = threadIdx.x; t < (long long)ch * hc; t += blockDim.x) {
        const int ky = (int)(t / hc), kx = (int)(t - (long long)ky * hc);
        if (ky == 0 || kx == 0) continue;
        const double2 f = F[t];
        const double d = ANY ? factor(ky, kx) : 1.0, e = d * d * fma(f.x, f.x, f.y * f.y);
        s2 += doubled(kx) ? 2.0 * e : e;
      }
    }
    // sum x z = 1/cw sum_kx G(0, kx) conj X(kx) and sum y z = 1/ch sum_ky G(ky, 0) conj Y(ky)
    double J = 0.0, K = 0.0;
    for (int kx = threadIdx.x; kx < hc; kx += blockDim.x) {
      const double2 f = F[kx], x = ramp_x(kx);
      const double v = (f.x * x.x + f.y * x.y) * axis_divisor(0, kx);
      J += doubled(kx) ? 2.0 * v : v;
    }
    for (int ky = threadIdx.x; ky < ch; ky += blockDim.x) {
      const double2 f = F[(size_t)ky * hc], y = ramp_y(ky);
      K += (f.x * y.x + f.y * y.y) * axis_divisor(ky, 0);
    }
    J = block_sum_d(J, red) / (double)cw;
    K = block_sum_d(K, red) / (double)ch;
    const double L = F[0].x * axis_divisor(0, 0);
    plane_fit(P.plane, J, K, L, pa, pb, pc);
  }
  // value of the plane-free spectrum on an axis
  auto axis_value = [&](int ky, int kx, double d) {
    const double2 f = F[(size_t)ky * hc + kx];
    double2 v = make_double2(f.x * d, f.y * d);
    if (P.normalize) {
      if (ky == 0) {
        const double2 x = ramp_x(kx);
        v.x -= pa * (double)ch * x.x;
        v.y -= pa * (double)ch * x.y;
      }
      if (kx == 0) {
        const double2 y = ramp_y(ky);
        v.x -= pb * (double)cw * y.x;
        v.y -= pb * (double)cw * y.y;
      }
      if (ky == 0 && kx == 0) v.x -= pc * (double)pixels;
    }
    return v;
  };
  if (P.normalize) {
    for (int k = threadIdx.x; k < hc + ch - 1; k += blockDim.x) {
      const int kx = k < hc ? k : 0, ky = k < hc ? 0 : k - hc + 1;
      const double2 v = axis_value(ky, kx, axis_divisor(ky, kx));
      const double e = fma(v.x, v.x, v.y * v.y);
      s2 += doubled(kx) ? 2.0 * e : e;
    }
    s2 = block_sum_d(s2, red) * inv;  // sum of v^2 over the pixels
    const double ave = axis_value(0, 0, axis_divisor(0, 0)).x * inv;
    const double sd = sqrt(__dsub_rn(s2 * inv, __dmul_rn(ave, ave)));
    if (sd > 0.0) {
      scale = inv / sd;
      centre = true;
    }
  }
  __syncthreads();  // the axes have been read
  auto finish = [&](int ky, int kx, double d) {
    const size_t o = (size_t)ky * hc + kx;
    double m = P.mask != nullptr ? P.mask[(size_t)ky * cw + kx] * scale : scale;
    if (ANY && P.mask != nullptr) m = 0.5 * (m + P.mask[(size_t)mirrored(ky, ch) * cw + mirrored(kx, cw)] * scale);
    double2 v;
    if (ky == 0 || kx == 0) {
      v = axis_value(ky, kx, d);
      if (ky == 0 && kx == 0 && centre) v.x = 0.0;  // the mean
    } else {
      v = F[o];
      m *= d;
    }
    F[o] = make_double2(v.x * m, v.y * m);
  };
  if (ANY) {
    for (long long t = threadIdx.x; t < (long long)ch * hc; t += blockDim.x) {
      const int ky = (int)(t / hc), kx = (int)(t % hc);
      finish(ky, kx, factor(ky, kx));
    }
  } else if (P.amplitudes) {
    // in order; the bin by its definition, round(distance): a distance of an
    // integer d2 < 2^16 is at least 2^-11 from a half, float32's square root
    // within 2^-15 of it
    for (int t = threadIdx.x; t < ch * hc; t += blockDim.x) {
      const int ky = t / hc, kx = t - ky * hc, y = axis_y(ky);
      finish(ky, kx, divisor(__float2int_rn(sqrtf((float)(y * y + kx * kx)))));
    }
  } else if (P.bin_ptr != nullptr) {
    for (int b = warp; b < P.n_bins; b += nw) {
      const double d = s_div[b];
      for (int i = P.bin_ptr[b] + lane; i < P.bin_ptr[b + 1]; i += 32) {
        const int p = P.bin_pix[i], ky = p / cw, kx = p - ky * cw;
        if (kx < hc) finish(ky, kx, d);
      }
    }
  } else {
    for (long long t = threadIdx.x; t < (long long)ch * hc; t += blockDim.x)
      finish((int)(t / hc), (int)(t % hc), 1.0);
  }
}

__global__ void __launch_bounds__(kSpectrumThreads) ingest_spectrum(double2* __restrict__ work, int ch, int cw,
                                                                    SpectrumSteps P) {
  extern __shared__ double s_div[];
  __shared__ double red[kSpectrumThreads / 32];
  double2* F = work + (size_t)blockIdx.x * ch * (cw / 2 + 1);
  const bool any = (P.bin_ptr != nullptr && *P.notes.bins_other == P.notes.call) ||
                   (P.mask != nullptr && *P.notes.mask_other == P.notes.call);
  if (any) spectrum_steps<true>(F, ch, cw, P, s_div, red);
  else spectrum_steps<false>(F, ch, cw, P, s_div, red);
}

__global__ void ingest_store(const double* __restrict__ work, long long total, int cw, int ld, float* __restrict__ out) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const long long r = t / cw;
    out[t] = (float)work[r * ld + (t - r * cw)];
  }
}

int grid_of(long long total, int sm_count) {
  long long g = (total + kIngestThreads - 1) / kIngestThreads;
  const long long cap = 8LL * sm_count;
  return (int)(g < cap ? (g > 0 ? g : 1) : cap);
}

}  // namespace

// ints of the notes on a call's tables
size_t ingest_note_elems(int ch, int cw) { return 2 + (size_t)ch * cw; }

static TableNotes table_notes(const int* bin_ptr, const int* bin_pix, int n_bins, const double* mask, int* notes,
                              int call) {
  return TableNotes{bin_ptr, bin_pix, n_bins, mask, call, notes, notes + 1, notes + 2};
}

// sums over the pixel grid of x^2, xy, x, y^2, y and 1, exact in integers
static PlaneSums plane_sums(int ch, int cw) {
  const long long h = ch, w = cw;
  const long long sx = w * (w - 1) / 2, sy = h * (h - 1) / 2;
  const long long sxx = (w - 1) * w * (2 * w - 1) / 6, syy = (h - 1) * h * (2 * h - 1) / 6;
  return PlaneSums{(double)(sxx * h), (double)(sx * sy), (double)(sx * h), (double)(syy * w), (double)(sy * w),
                   (double)(h * w)};
}

cudaError_t launch_ingest_load(cudaStream_t st, const float* images, int n, int h, int w, const int* shifts, int ch,
                               int cw, double* work, int ld, const int* bin_ptr, const int* bin_pix, int n_bins,
                               const double* mask, int* notes, int call, int sm_count) {
  ingest_load<<<grid_of((long long)n * ch * cw, sm_count), kIngestThreads, 0, st>>>(
      images, n, h, w, shifts, ch, cw, work, ld, table_notes(bin_ptr, bin_pix, n_bins, mask, notes, call));
  return cudaGetLastError();
}

cudaError_t launch_ingest_spectrum(cudaStream_t st, double2* work, int n, int ch, int cw, const int* bin_ptr,
                                   const int* bin_pix, const double* bin_count, int n_bins, int normalize,
                                   const double* mask, int* notes, int call) {
  const size_t bins = bin_ptr != nullptr ? (size_t)n_bins * sizeof(double) : 0;
  const size_t ramps = normalize ? (size_t)(cw / 2 + 1 + ch) * sizeof(double) : 0;
  const bool keep = bins + ramps <= 96 * 1024;  // else the ramps are computed where they are used
  const size_t amps = (size_t)ch * (cw / 2 + 1) * sizeof(double);
  const bool hold = bin_ptr != nullptr && keep && ch <= 256 && cw <= 256 && bins + ramps + amps <= 200 * 1024;
  const size_t smem = bins + (keep ? ramps : 0) + (hold ? amps : 0);
  static SmemLimit limit;
  const cudaError_t e = allow_smem(ingest_spectrum, smem, limit);
  if (e != cudaSuccess) return e;
  const SpectrumSteps P{bin_ptr, bin_pix, bin_count, n_bins, normalize, plane_sums(ch, cw), keep && normalize ? 1 : 0, hold ? 1 : 0, mask,
                        table_notes(bin_ptr, bin_pix, n_bins, mask, notes, call)};
  ingest_spectrum<<<n, kSpectrumThreads, smem, st>>>(work, ch, cw, P);
  return cudaGetLastError();
}

cudaError_t launch_ingest_normalize(cudaStream_t st, double* work, int n, int ch, int cw, int ld) {
  ingest_normalize<<<n, kIngestThreads, 0, st>>>(work, ch, cw, ld, plane_sums(ch, cw));
  return cudaGetLastError();
}

cudaError_t launch_ingest_store(cudaStream_t st, const double* work, int n, int ch, int cw, int ld, float* out,
                                int sm_count) {
  const long long total = (long long)n * ch * cw;
  ingest_store<<<grid_of(total, sm_count), kIngestThreads, 0, st>>>(work, total, cw, ld, out);
  return cudaGetLastError();
}
