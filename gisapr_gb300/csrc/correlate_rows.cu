// Plain FP32 correlation (correlate.cu has the mathematics) with the particle's
// spectrum in registers, for the sizes and windows that are searched with.
//
// A thread owns one column of one psi spectrum and Q = 2 or 3 of the residues q
// of the rows r = M j + q (M = n/16): 16 Q complex values that stay in registers
// over a group of directions. Per direction it multiplies them by the template's
// column from shared memory, transforms the 16 rows of each residue, adds the
// wanted rows of its residues up by powers of w_n^y, which all lanes share, and
// turns the sum by w_n^{Q l y}; the L = M/Q lanes that
// share a column then halve the rows among them until each holds the whole sum
// of C/L rows (an exchange by shuffles that moves every value once). The next
// template's columns are on their way by asynchronous copies meanwhile. After a
// few directions one thread per (map, y) contracts its row of columns with the
// column twiddles, using x and -x together, and adds it to the partial map.
//
// A CTA goes through the column tiles of its particle one after the other; with
// few particles the tiles are spread over a cluster, whose partial maps are added
// over distributed shared memory, and psi angles and directions over more CTAs.
//
// 90,000 maps at box 128 (5,000 particles, 5.8 directions, three angles, window
// 12) take 0.99 ms; the form with all psi spectra in shared memory takes 1.79.
// Their multiply-adds are 0.39 ms of the FP32 pipes; what is left is latency
// (ten warps on an SM, a barrier per direction), 0.1 ms of copies, 0.1 ms of the
// contraction over columns and 0.05 ms of the particles' first reading. Reading
// the particle's tiles through the same ring as the templates' hid that and cost
// 0.15 ms more in copies.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kGroup = 8;  // directions whose partial maps are held together
constexpr int kPsi = 3;    // psi angles of a CTA at most

struct RowsParams {
  const float2* bank;      // [n_cand][..][n][H]
  const float2* stack;     // [n_particles][n_psi][n][H]
  const int* local_ptr;    // [n_particles + 1]
  const int* local_idx;
  const float2* tw_outer;  // [M][C]  exp(+2 pi i q y / n), y = -C/2 ..
  const float2* tw_col;    // [H][C]  w_c exp(+2 pi i c x / n)
  float* out_score;        // [n_cand][nnz][n_psi]
  int* out_y;
  int* out_x;
  int n_particles, n_psi, cluster, n_cand;
  long long bank_stride;
  int nnz;
  const unsigned char* subset;
  int psi_per_cta;         // blockIdx.y: chunk of psi angles, blockIdx.z: chunk of directions
  float2 step[16];         // exp(+2 pi i y / n), y = -C/2 ..
};

template <int C, int M, int Q>
struct Rows {
  static constexpr int n = 16 * M, H = n / 2 + 1, L = M / Q, h = C / 2;
  static constexpr int tile = M <= 6 ? 17 : 13;             // columns of a pass
  static constexpr int batch = M == 6 || C == 16 ? 4 : 8;   // directions between two contractions over the columns
  static constexpr int tiles = (H + tile - 1) / tile;
  static constexpr int chunks = (tile + 2) / 2;             // 16-byte pieces of a tile's row
  static constexpr int CL = (C + L - 1) / L;                // rows of the window per lane after the exchange
  static constexpr int TWS = C % 4 == 0 ? C + 2 : C;        // lanes of one column read their twiddles in different banks
  // Lane l of a column has the residues q = Q l + i. A half warp reads, for one i, L rows x 16/L columns of a
  // template; with Q = 2 the rows have one parity, and the (even) stride puts them in different banks for L <= 4.
  static constexpr int spread = Q == 2 && L <= 4 ? 8 / L : 2;
  static constexpr int TS = (tile + 1 - spread + 7) / 8 * 8 + spread;
  static constexpr int WS = (h + 2) / 2 * 2;                // stride of the column twiddles: x = 0, -1, .. -h
  static constexpr int RS = C % 8 == 0 ? C + 4 : C;         // stride of a partial map's rows
  static constexpr int ZS = tile;                           // odd: rows of one column in different banks
  static constexpr int max_threads = (tile * L * kPsi + 31) / 32 * 32;
  // 12 warps of 168 registers on an SM; 16 of 128 registers spilled and took 1.32 against 1.08 ms
  static constexpr int min_ctas = 12 / (max_threads / 32);
  static size_t smem(int np) {
    return sizeof(float2) * (2 * (size_t)n * TS + (size_t)L * TWS + (size_t)tile * WS + (size_t)batch * np * C * ZS) +
           sizeof(float) * (size_t)kGroup * np * C * RS;
  }
};

// The directions of a group: where their templates start in the bank and their
// scores in the output.
struct Group {
  long long src[kGroup];
  size_t out[kGroup];
  int count, next_cand, next_e;  // and where the group after it starts
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <int C, int M, int Q>
__global__ void __launch_bounds__(Rows<C, M, Q>::max_threads, Rows<C, M, Q>::min_ctas) correlate_rows(RowsParams P) {
  using R = Rows<C, M, Q>;
  constexpr int n = R::n, H = R::H, L = R::L, CL = R::CL, h = R::h, TS = R::TS, ZS = R::ZS, WS = R::WS, RS = R::RS, tile = R::tile, batch = R::batch;
  extern __shared__ __align__(16) float2 smem[];
  __shared__ Group s_group[3];
  cg::cluster_group cluster = cg::this_cluster();
  const int K = P.cluster, rank = (int)cluster.block_rank(), b = blockIdx.x / K;
  const int np = P.psi_per_cta, psi0 = blockIdx.y * np, pn = min(np, P.n_psi - psi0);
  float2* s_t = smem;                                        // [2][n][TS]
  float2* s_two = s_t + 2 * n * TS;                          // [L][TWS]: q = Q l
  float2* s_twc = s_two + L * R::TWS;                        // [tile][WS]
  float2* s_z = s_twc + tile * WS;                           // [batch][np][C][ZS]
  float* s_raw = reinterpret_cast<float*>(s_z + (size_t)batch * np * C * ZS);  // [kGroup][np][C][RS]

  const int first = P.local_ptr[b], d = P.local_ptr[b + 1] - first;
  const int e0 = first + (int)((long long)d * blockIdx.z / gridDim.z);
  const int e1 = first + (int)((long long)d * (blockIdx.z + 1) / gridDim.z);
  const unsigned char* subset = P.subset == nullptr ? nullptr : P.subset + b;
  auto next_cand = [&](int c) {
    if (subset != nullptr)
      while (c < P.n_cand && subset[(size_t)c * P.n_particles] == 0) ++c;
    return c;
  };
  if (e1 <= e0) return;  // the same in the whole cluster, as is the next
  if (next_cand(0) >= P.n_cand) return;

  const int tid = threadIdx.x, ql = tid % L, cl = (tid / L) % tile, psi = tid / (L * tile);
  const float2* stack = P.stack + ((size_t)b * P.n_psi + psi0) * n * H;
  // warp 0: the directions from (cand, e) on
  auto fill = [&](Group& G, int cand, int e) {
    if (tid >= 32) return;
    auto walk = [&](int ahead, int& c, int& x) {
      c = cand;
      x = e + ahead;
      while (x >= e1 && c < P.n_cand) {
        x -= e1 - e0;
        c = next_cand(c + 1);
      }
      return c < P.n_cand;
    };
    int c, x;
    const bool in = tid < kGroup && walk(tid, c, x);
    if (in) {
      G.src[tid] = c * P.bank_stride + (long long)P.local_idx[x] * (n * H);
      G.out[tid] = ((size_t)c * P.nnz + x) * P.n_psi + psi0;
    }
    const unsigned all = __ballot_sync(0xffffffffu, in);
    if (tid == 0) {
      walk(kGroup, c, x);
      G.count = __popc(all);
      G.next_cand = c;
      G.next_e = x;
    }
  };
  // Columns [clo, clo + cw) of a template into shared memory in pieces of 16
  // bytes; a row that starts in the middle of a piece is kept one place later.
  const int t_rows = blockDim.x / R::chunks, t_row = tid / R::chunks, t_piece = tid % R::chunks;
  auto stage = [&](int buf, const float2* t, int clo) {
    const int cw = min(tile, H - clo);
    if (t_row < t_rows) {
      float2* dst = s_t + buf * (n * TS) + 2 * t_piece;
      for (int r = t_row; r < n; r += t_rows) {
        const int odd = (r + clo) & 1;  // H is odd
        if (2 * t_piece < cw + odd) cp_async16(dst + r * TS, t + r * H + clo - odd + 2 * t_piece);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  fill(s_group[0], next_cand(0), e0);
  for (int t = tid; t < L * C; t += blockDim.x) s_two[(t / C) * R::TWS + t % C] = P.tw_outer[(t / C) * Q * C + t % C];
  __syncthreads();
  stage(0, P.bank + s_group[0].src[0], rank * tile);

  int buf = 0;
  for (int gi = 0;; gi = gi == 2 ? 0 : gi + 1) {
    const Group& G = s_group[gi];
    Group& N = s_group[gi == 2 ? 0 : gi + 1];
    const int count = G.count;
    const bool last = G.next_cand >= P.n_cand;
    if (!last) fill(N, G.next_cand, G.next_e);
    for (int ti = rank; ti < R::tiles; ti += K) {
      const int clo = ti * tile, cw = min(tile, H - clo);
      const bool act = psi < pn && cl < cw;
      float2 p[Q][16];
      {
        const float2* src = stack + (psi * n + Q * ql) * H + clo + cl;
#pragma unroll
        for (int i = 0; i < Q; ++i)
#pragma unroll
          for (int j = 0; j < 16; ++j) p[i][j] = act ? src[(M * j + i) * H] : make_float2(0.f, 0.f);
      }
      for (int t = tid; t < cw * (h + 1); t += blockDim.x) {  // read after the next barriers
        const int c = t / (h + 1), k = t % (h + 1);
        s_twc[c * WS + k] = P.tw_col[(size_t)(clo + c) * C + h - k];
      }
      for (int item = 0; item < count; ++item) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // this template is in; the other buffer and the sums are free
        if (item + 1 < count)
          stage(buf ^ 1, P.bank + G.src[item + 1], clo);
        else if (ti + K < R::tiles)
          stage(buf ^ 1, P.bank + G.src[0], (ti + K) * tile);
        else if (!last)
          stage(buf ^ 1, P.bank + N.src[0], rank * tile);
        const float2* T = s_t + buf * (n * TS) + Q * ql * TS + cl;
        float2 z[CL * L];
// Z(y) = w^{Q l y} (G_0 + w^y (G_1 + w^y G_2)): w^y is the same in all lanes and comes from the parameters
#pragma unroll
        for (int i = Q - 1; i >= 0; --i) {
          float2 x[16];
          const float2* Ti = T + ((Q * ql + i + clo) & 1);
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = cmul(Ti[(M * j + i) * TS], p[i][j]);
          idft16(x);
#pragma unroll
          for (int y = 0; y < C; ++y) {
            const float2 gq = x[idft16_slot((y - h) & 15)], c = P.step[y];
            if (i == Q - 1) {
              z[y] = gq;
            } else if (y == h) {
              z[y] = cadd(gq, z[y]);
            } else {
              const float2 v = z[y];
              z[y].x = fmaf(v.x, c.x, fmaf(-v.y, c.y, gq.x));
              z[y].y = fmaf(v.x, c.y, fmaf(v.y, c.x, gq.y));
            }
          }
        }
        const float2* w = s_two + ql * R::TWS;
#pragma unroll
        for (int y = 0; y < C; ++y) z[y] = cmul(z[y], w[y]);
#pragma unroll
        for (int y = C; y < CL * L; ++y) z[y] = make_float2(0.f, 0.f);
        // lane ql ends with rows CL ql ..
#pragma unroll
        for (int m = L / 2, half = CL * L / 2; m >= 1; m /= 2, half /= 2) {
          const bool up = (ql & m) != 0;
#pragma unroll
          for (int s = 0; s < half; ++s) {
            const float2 give = up ? z[s] : z[s + half], keep = up ? z[s + half] : z[s];
            float2 got;
            got.x = __shfl_xor_sync(0xffffffffu, give.x, m);
            got.y = __shfl_xor_sync(0xffffffffu, give.y, m);
            z[s] = cadd(keep, got);
          }
        }
        const int zi = item % batch;
        if (act) {
          float2* zo = s_z + ((zi * np + psi) * C + ql * CL) * ZS + cl;
#pragma unroll
          for (int s = 0; s < CL; ++s)
            if (C % L == 0 || ql * CL + s < C) zo[s * ZS] = z[s];
        }
        buf ^= 1;
        if (zi == batch - 1 || item + 1 == count) {
          __syncthreads();
          // columns: raw(-k) = A_k + B_k, raw(k) = A_k - B_k; a row stays with its thread over the tiles
          for (int t = tid; t < (zi + 1) * pn * C; t += blockDim.x) {
            const int gp = t / C, y = t % C;  // gp = direction * pn + psi
            const int slot = gp / pn, ps = gp % pn;
            const float2* row = s_z + ((slot * np + ps) * C + y) * ZS;
            float A[h + 1], B[h + 1];
#pragma unroll
            for (int k = 0; k <= h; ++k) A[k] = B[k] = 0.f;
#pragma unroll 2
            for (int c = 0; c < cw; ++c) {
              const float2 v = row[c];
              const float4* w = reinterpret_cast<const float4*>(s_twc + c * WS);
#pragma unroll
              for (int k = 0; k <= h; k += 2) {
                const float4 u = w[k / 2];
                A[k] = fmaf(v.x, u.x, A[k]);
                B[k] = fmaf(-v.y, u.y, B[k]);
                if (k + 1 <= h) {
                  A[k + 1] = fmaf(v.x, u.z, A[k + 1]);
                  B[k + 1] = fmaf(-v.y, u.w, B[k + 1]);
                }
              }
            }
            float* out = s_raw + (((item - zi + slot) * np + ps) * C + y) * RS;
            auto value = [&](int xi) { return xi < h ? A[h - xi] + B[h - xi] : A[xi - h] - B[xi - h]; };
            if (C % 4 == 0) {
#pragma unroll
              for (int xi = 0; xi < C; xi += 4) {
                float4 v = make_float4(value(xi), value(xi + 1), value(xi + 2), value(xi + 3));
                float4* o = reinterpret_cast<float4*>(out + xi);
                if (ti != rank) {
                  const float4 w = *o;
                  v = make_float4(w.x + v.x, w.y + v.y, w.z + v.z, w.w + v.w);
                }
                *o = v;
              }
            } else {
#pragma unroll
              for (int xi = 0; xi < C; xi += 2) {
                float2 v = make_float2(value(xi), value(xi + 1));
                float2* o = reinterpret_cast<float2*>(out + xi);
                *o = ti == rank ? v : cadd(*o, v);
              }
            }
          }
          if (item + 1 == count) __syncthreads();  // s_twc may change
        }
      }
    }
    if (K > 1) cluster.sync();
    // partial maps: dealt out to the CTAs, summed in rank order, first maximum in row-major order
    {
      const int warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
      for (int mp = rank + K * warp; mp < count * pn; mp += K * nw) {
        const int item = mp / pn, ps = mp % pn;
        float* raw = s_raw + (item * np + ps) * C * RS;
        float best = -INFINITY;
        int bi = C * C;
        for (int t = lane; t < C * C; t += 32) {
          const int at = t / C * RS + t % C;
          float v;
          if (K == 1) {
            v = raw[at];
          } else {
            v = 0.f;
            for (int r = 0; r < K; ++r) v += cluster.map_shared_rank(raw, r)[at];
          }
          if (v > best) { best = v; bi = t; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) {
          const size_t o = G.out[item] + ps;
          P.out_score[o] = best * 1024.0f;
          P.out_y[o] = bi / C;
          P.out_x[o] = bi % C;
        }
      }
    }
    if (K > 1) cluster.sync();
    if (last) return;
  }
}

template <int C, int M, int Q>
cudaError_t launch(RowsParams P, int sm_count, cudaStream_t st, bool* taken) {
  using R = Rows<C, M, Q>;
  // Cluster size: rounds of resident CTAs times passes over the tiles, plus 0.4 of a pass for adding the partial maps up.
  // Clusters of three and more fill about nine tenths of the SMs. Box 128, three psi angles, six directions: 100
  // particles take 34 us with 5 CTAs each and 42 with 2, 150 take 50 and 42, 400 take 120 with 5 and 107 with one.
  const long long slots = (long long)R::min_ctas * sm_count;
  int chunks = (P.n_psi + kPsi - 1) / kPsi;
  long long ctas = (long long)P.n_particles * chunks;
  int K = 1, top = std::min(R::tiles, 8);
  if (P.cluster > 0) {
    const int passes = (R::tiles + std::min(P.cluster, top) - 1) / std::min(P.cluster, top);
    K = (R::tiles + passes - 1) / passes;  // as many as have a tile in every pass but the last
  } else {
    double best = 0;
    for (int k = 1; k <= top; ++k) {
      const int passes = (R::tiles + k - 1) / k;
      if (passes > 1 && (R::tiles + passes - 1) / passes != k) continue;
      const long long fit = k < 3 ? slots : slots * 9 / 10;
      const double cost = (double)((ctas * k + fit - 1) / fit) * (passes + (k > 1 ? 0.4 : 0.0));
      if (k == 1 || cost < best) {
        best = cost;
        K = k;
      }
    }
  }
  P.cluster = K;
  for (int y = 0; y < C; ++y) {
    const double a = 2.0 * 3.14159265358979323846 * (y - C / 2) / R::n;
    P.step[y] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  ctas *= K;
  // Still few: the maps are spread, first by psi, then by direction.
  if (ctas < slots) chunks = (int)std::min<long long>(P.n_psi, chunks * (slots / ctas));
  P.psi_per_cta = (P.n_psi + chunks - 1) / chunks;
  chunks = (P.n_psi + P.psi_per_cta - 1) / P.psi_per_cta;
  const long long now = (long long)P.n_particles * K * chunks;
  const int splits = (int)std::min<long long>(8, std::max<long long>(1, slots / now));
  const size_t smem = R::smem(P.psi_per_cta);
  if (chunks > 65535) return cudaSuccess;
  static SmemLimit limit;
  const cudaError_t e = allow_smem(correlate_rows<C, M, Q>, R::smem(kPsi), limit);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(P.n_particles * K), chunks, splits);
  cfg.blockDim = dim3((R::tile * R::L * P.psi_per_cta + 31) / 32 * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)K;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  *taken = true;
  return cudaLaunchKernelEx(&cfg, correlate_rows<C, M, Q>, P);
}

// The sizes of the searches. us in this form and in the one of correlate.cu, six
// directions and three angles: 64 (4,000 particles, window 10) 236 / 533, 96
// (2,000, 12) 307 / 526, 128 (2,000, 12) 442 / 800, 192 (1,000, 12) 716 / 1397,
// 256 (500 with eight directions, 14) 920 / 1526; one particle at 128 8.7 / 24.
// Other sizes and windows below 8 stay with the other, which takes any.
template <int C>
cudaError_t launch_size(const RowsParams& P, int n, int sm_count, cudaStream_t st, bool* taken) {
  switch (n) {
    case 64: return launch<C, 4, 2>(P, sm_count, st, taken);
    case 96: return launch<C, 6, 3>(P, sm_count, st, taken);
    case 128: return launch<C, 8, 2>(P, sm_count, st, taken);
    case 192: return launch<C, 12, 3>(P, sm_count, st, taken);
    case 256: return launch<C, 16, 2>(P, sm_count, st, taken);
    default: return cudaSuccess;
  }
}

}  // namespace

// Whether this form has the size and window.
bool correlate_rows_takes(int n, int crop) {
  return (n == 64 || n == 96 || n == 128 || n == 192 || n == 256) && crop >= 8 && crop <= 16 && crop % 2 == 0;
}

// *taken: this form has the size and window, and was launched. Templates must
// start on 16 bytes.
cudaError_t launch_correlate_rows(cudaStream_t st, const float2* bank, const float2* stack, const int* local_ptr,
                                  const int* local_idx, int n_particles, int n_psi, int n, int crop,
                                  const float2* tw_outer, const float2* tw_col, float* out_score, int* out_y,
                                  int* out_x, int n_cand, long long bank_stride, int nnz, int cluster,
                                  const unsigned char* subset, int sm_count, bool* taken) {
  *taken = false;
  if (n_particles <= 0 || n_cand <= 0 || !correlate_rows_takes(n, crop)) return cudaSuccess;
  if (reinterpret_cast<uintptr_t>(bank) % 16 != 0 || bank_stride % 2 != 0) return cudaSuccess;
  RowsParams P{bank, stack, local_ptr, local_idx, tw_outer, tw_col, out_score, out_y, out_x, n_particles, n_psi, cluster,
               n_cand, bank_stride, nnz, subset, 0};
  switch (crop) {
    case 8: return launch_size<8>(P, n, sm_count, st, taken);
    case 10: return launch_size<10>(P, n, sm_count, st, taken);
    case 12: return launch_size<12>(P, n, sm_count, st, taken);
    case 14: return launch_size<14>(P, n, sm_count, st, taken);
    case 16: return launch_size<16>(P, n, sm_count, st, taken);
    default: return cudaSuccess;
  }
}
