// Building blocks of the recycled PCG start (Galerkin projection onto vectors
// whose Sigma-image is known without a GRM product) and diag(K).
#include <algorithm>

#include "engine.cuh"
#include "warm.cuh"

namespace saige {
namespace {

constexpr int kG = 32;  // Gram: rows per stage; the chunks of rows are counted in 32 x 32 tiles

// Row chunks: at least 2,048 rows each, and at most kGramBlocks blocks of 32 x 32 tiles.
constexpr int kGramBlocks = 148 * 4;

int gram_chunks(int64_t n, int a, int b) {
  const int tiles = ((a + kG - 1) / kG) * ((b + kG - 1) / kG);
  const int64_t by_rows = (n + 2047) / 2048;
  const int64_t want = std::max<int64_t>(1, kGramBlocks / std::max(tiles, 1));
  return (int)std::max<int64_t>(1, std::min(by_rows, want));
}

// 16 bytes global -> shared (cp.async); bytes past `valid` (0, 8 or 16) are zero.
__device__ __forceinline__ void cp_async16_zfill(void* smem, const void* gmem, int valid) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(valid)
               : "memory");
}

// Block (chunk x, tile y): the sums over rows [x*chunk, (x+1)*chunk) of output tile y,
// 8R x 8R entries, 8 x 8 threads of R x R.  Each entry is one chain of fused multiply-adds
// in row order (a start's coefficients are sensitive to the last bit, so neither the
// chains nor the chunks may depend on the tile), which sets the pace: 32 rows are staged
// column by column while the ones before them are multiplied (cp.async, 8 / R buffers; column
// pitch 34 doubles: the eight columns that a quarter warp reads lie in different banks),
// and two rows are read per 16-byte load.
// Bound: the FP64 pipe for many rows and columns (R = 4: 16 chains per thread), the
// latency of the chains and of the stages' loads for few (R = 2, four times the blocks).  With 32 x 32 tiles of 256
// threads, unstaged loads and five 8-byte shared loads per four multiply-adds: 302 us at
// n = 200,000 (bases of up to about 120 columns, mean of a fit's ten) and 123 us at n = 2,000;
// now 158 and 29 us.
constexpr int kGramPitch = kG + 2;

template <int R>
__global__ void __launch_bounds__(64)
    gram_kernel(const double* __restrict__ A, int a, const double* __restrict__ B, int b,
                int64_t n, int64_t ld, int64_t chunk, double* __restrict__ partial) {
  constexpr int kTile = 8 * R, kStages = 8 / R;
  __shared__ __align__(16) double as[kStages][kTile][kGramPitch], bs[kStages][kTile][kGramPitch];
  const int tiles_b = (b + kTile - 1) / kTile;
  const int i0 = (blockIdx.y / tiles_b) * kTile, j0 = (blockIdx.y % tiles_b) * kTile;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  const int64_t lo = (int64_t)blockIdx.x * chunk;
  const int64_t hi = lo + chunk < n ? lo + chunk : n;
  // stage rows r0 .. r0+31 of the tile's columns, 16 pieces of two rows per column; rows
  // past hi and columns past the end are zero.  A thread takes piece pc of the columns
  // c0 + 4k of both operands: their addresses differ by a constant.
  const int pc = threadIdx.x & 15, c0 = threadIdx.x >> 4;
  const double* const pa = A + (int64_t)(i0 + c0) * ld + 2 * pc;
  const double* const pb = B + (int64_t)(j0 + c0) * ld + 2 * pc;
  const int na = a - i0 - c0, nb = b - j0 - c0;  // column 4k exists when 4k < na (nb)
  auto stage = [&](int buf, int64_t r0) {
    const int64_t left = hi - (r0 + 2 * pc);
    const int rows = left >= 2 ? 16 : (left == 1 ? 8 : 0);
#pragma unroll
    for (int k = 0; k < 2 * R; ++k) {
      const bool in = 4 * k < na && rows > 0;
      cp_async16_zfill(&as[buf][c0 + 4 * k][2 * pc], in ? pa + 4 * k * ld + r0 : A, in ? rows : 0);
    }
#pragma unroll
    for (int k = 0; k < 2 * R; ++k) {
      const bool in = 4 * k < nb && rows > 0;
      cp_async16_zfill(&bs[buf][c0 + 4 * k][2 * pc], in ? pb + 4 * k * ld + r0 : A, in ? rows : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[R][R];
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int l = 0; l < R; ++l) acc[k][l] = 0.0;
  // kStages - 1 stages ahead; an empty group where there is no further stage keeps the
  // count of groups in flight the same
  auto ahead = [&](int buf, int64_t r0) {
    if (r0 < hi) stage(buf, r0);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int k = 0; k < kStages - 1; ++k) ahead(k, lo + k * kG);
  int buf = 0;
  for (int64_t r0 = lo; r0 < hi; r0 += kG, buf = buf + 1 == kStages ? 0 : buf + 1) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // stage r0 has landed, and every thread is done with the one before
    ahead(buf == 0 ? kStages - 1 : buf - 1, r0 + (kStages - 1) * kG);
#pragma unroll
    for (int r = 0; r < kG; r += 2) {
      double2 x[R], y[R];
#pragma unroll
      for (int k = 0; k < R; ++k) x[k] = *reinterpret_cast<const double2*>(&as[buf][ty + 8 * k][r]);
#pragma unroll
      for (int l = 0; l < R; ++l) y[l] = *reinterpret_cast<const double2*>(&bs[buf][tx + 8 * l][r]);
#pragma unroll
      for (int k = 0; k < R; ++k)
#pragma unroll
        for (int l = 0; l < R; ++l) acc[k][l] = fma(x[k].x, y[l].x, acc[k][l]);
#pragma unroll
      for (int k = 0; k < R; ++k)
#pragma unroll
        for (int l = 0; l < R; ++l) acc[k][l] = fma(x[k].y, y[l].y, acc[k][l]);
    }
  }
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int l = 0; l < R; ++l) {
      const int i = i0 + ty + 8 * k, j = j0 + tx + 8 * l;
      if (i < a && j < b) partial[((int64_t)i * b + j) * gridDim.x + blockIdx.x] = acc[k][l];
    }
}

// out[e] = sum over chunks, in chunk order.
__global__ void gram_reduce(const double* __restrict__ partial, int nchunks, int64_t count,
                            double* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= count) return;
  double s = 0.0;
  for (int c = 0; c < nchunks; ++c) s += partial[e * nchunks + c];
  out[e] = s;
}

__global__ void combo_kernel(const double* __restrict__ V, int m, const double* __restrict__ G,
                             int q, double* __restrict__ Y, int add, int64_t n, int64_t ld) {
  extern __shared__ double g[];  // m x 8 slice of G
  const int c0 = blockIdx.y * 8;
  for (int t = threadIdx.x; t < m * 8; t += blockDim.x) {
    const int j = t >> 3, c = t & 7;
    g[t] = (c0 + c < q) ? G[(int64_t)j * q + c0 + c] : 0.0;
  }
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = (add && c0 + c < q) ? Y[(int64_t)(c0 + c) * ld + i] : 0.0;
  // eight columns' loads at a time: at n = 9,001 a thread's chain of loads is what the
  // kernel takes (7.9 -> 6.5 us)
  int j = 0;
  for (; j + 8 <= m; j += 8) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = V[(int64_t)(j + k) * ld + i];
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] += v[k] * g[(j + k) * 8 + c];
  }
  for (; j < m; ++j) {
    const double v = V[(int64_t)j * ld + i];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] += v * g[j * 8 + c];
  }
#pragma unroll
  for (int c = 0; c < 8; ++c)
    if (c0 + c < q) Y[(int64_t)(c0 + c) * ld + i] = acc[c];
}

// out = tau0 v / wmax + tau1 kv, and v and kv copied beside it; no output overlaps an input.
__global__ void sigma_image_kernel(const double* __restrict__ v, const double* __restrict__ kv,
                                   const double* __restrict__ wmax, double tau0, double tau1,
                                   double* __restrict__ v_out, double* __restrict__ kv_out,
                                   double* __restrict__ out, int64_t n, int64_t ld) {
  const int64_t c = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ld) return;
  const double x = v[c * ld + i], kx = kv[c * ld + i];
  v_out[c * ld + i] = x;
  kv_out[c * ld + i] = kx;
  if (i < n) out[c * ld + i] = tau0 * x / wmax[i] + tau1 * kx;
}

__global__ void sub_cols_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                double* __restrict__ out, int64_t n, int64_t ld) {
  const int64_t c = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[c * ld + i] = a[c * ld + i] - b[c * ld + i];
}

// scales: sx[q], sb[q], sk0, sk1
__global__ void learn_features_kernel(const double* __restrict__ x, const double* __restrict__ b,
                                      const double* __restrict__ bnext,
                                      const double* __restrict__ w,
                                      const double* __restrict__ wnext,
                                      const double* __restrict__ diagk,
                                      const double* __restrict__ ku, int n_sk,
                                      const double* __restrict__ scales, double tau0, double tau1,
                                      double dmean, int64_t n, int64_t ld, int q,
                                      float* __restrict__ F) {
  const int c = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t e = (int64_t)c * n + i, a = (int64_t)c * ld + i;
  const double sx = scales[c], sb = scales[q + c];
  const double wi = w[i] > 1e-30 ? w[i] : 1e-30, wn = wnext[i] > 1e-30 ? wnext[i] : 1e-30;
  const double d = 1.0 / (tau0 / wi + tau1);
  float f[16];
  f[0] = (float)(sx > 0.0 ? x[a] / sx : 0.0);
  f[1] = (float)(sb > 0.0 ? b[a] / sb : 0.0);
  f[2] = (float)(sb > 0.0 ? (bnext[a] - b[a]) / sb : 0.0);
  f[3] = (float)log(wn / wi);
  f[4] = (float)(d / dmean - 1.0);
  f[5] = (float)(diagk[i] - 1.0);
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const double sk = scales[2 * q + s];
    f[6 + s] = (float)(s < n_sk && sk > 0.0 ? ku[(int64_t)s * ld + i] / sk : 0.0);
  }
  f[14] = (float)tau1;
  f[15] = 0.f;
  float4* dst = reinterpret_cast<float4*>(F + e * 16);
#pragma unroll
  for (int k = 0; k < 4; ++k) dst[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
}

__global__ void learn_targets_kernel(const double* __restrict__ x1, const double* __restrict__ x0,
                                     const double* __restrict__ s, int64_t n, int64_t ld,
                                     float* __restrict__ T) {
  const int c = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t a = (int64_t)c * ld + i;
  T[(int64_t)c * n + i] = (float)(s[c] > 0.0 ? (x1[a] - x0[a]) / s[c] : 0.0);
}

__global__ void learn_to_cols_kernel(const float* __restrict__ y, int64_t n, int64_t ld,
                                     double* __restrict__ out) {
  const int c = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[(int64_t)c * ld + i] = (double)y[(int64_t)c * n + i];
}

// The live rows of a handle, in order: those with a standardised column (1/s != 0) that the
// mask does not leave out.  Block b's count of kLiveRows rows, then, from the counts, their
// list and how many there are.
constexpr int kLiveRows = 1024;

__device__ __forceinline__ bool live_row(const double* inv_s, const uint8_t* excl, int64_t j,
                                         int64_t m) {
  return j < m && inv_s[j] != 0.0 && !(excl && excl[j]);
}

__global__ void __launch_bounds__(kLiveRows)
    live_count_kernel(const double* __restrict__ inv_s, const uint8_t* __restrict__ excl,
                      int64_t m, int32_t* __restrict__ counts) {
  const int c = __syncthreads_count(
      live_row(inv_s, excl, (int64_t)blockIdx.x * kLiveRows + threadIdx.x, m));
  if (threadIdx.x == 0) counts[blockIdx.x] = c;
}

__global__ void __launch_bounds__(kLiveRows)
    live_list_kernel(const double* __restrict__ inv_s, const uint8_t* __restrict__ excl,
                     int64_t m, const int32_t* __restrict__ counts, int32_t* __restrict__ rows,
                     int32_t* __restrict__ n_live) {
  __shared__ int before[kLiveRows / 32], in_warp[kLiveRows / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int s = 0;  // rows in the blocks before
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += kLiveRows) s += counts[k];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const int64_t j = (int64_t)blockIdx.x * kLiveRows + threadIdx.x;
  const bool live = live_row(inv_s, excl, j, m);
  const unsigned int votes = __ballot_sync(0xffffffffu, live);
  if (lane == 0) {
    before[warp] = s;
    in_warp[warp] = __popc(votes);
  }
  __syncthreads();
  int at = 0;
  for (int k = 0; k < kLiveRows / 32; ++k) at += before[k] + (k < warp ? in_warp[k] : 0);
  at += __popc(votes & ((1u << lane) - 1u));
  if (live) rows[at] = (int32_t)j;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kLiveRows - 1) *n_live = at + (live ? 1 : 0);
}

// Sums of z^2 over a range of the live rows, for 16 samples per thread (one packed word per
// row): z^2 of the four codes (00 -> 2, 10 -> 1, 11 -> 0, 01 missing -> 0) sits in shared
// memory for kDiagChunk rows at a time, so an entry costs a
// bit-field extract, one 8-byte lookup (four addresses per row: no bank conflicts)
// and one FP64 add.  Block y sums the (first + y)-th range of `per` live rows into row y of
// partial; grm_diag_finish adds the rows in order.  The ranges count live rows, so that a handle with
// markers left out forms the sums of a handle without them, to the bit.  Bound: the lookups.
// One thread per sample over all markers (a 4-byte load per 2-bit code, one serial chain) took
// 22.9 ms at n = 60,013, m = 39,000; this takes 0.62 ms (0.64 with the 51 registers that the
// compiler takes for five blocks per SM), and the list 5 us.
constexpr int kDiagThreads = 256;
constexpr int kDiagChunk = 64;

__global__ void __launch_bounds__(kDiagThreads, 4)
    grm_diag_kernel(const uint32_t* __restrict__ geno, int64_t wpr,
                    const double* __restrict__ two_p, const double* __restrict__ inv_s,
                    const int32_t* __restrict__ rows, const int32_t* __restrict__ n_live,
                    int64_t per, int64_t first, double* __restrict__ partial) {
  __shared__ double tab[kDiagChunk][4];
  __shared__ int64_t at[kDiagChunk];  // the rows' first words
  const int64_t w = (int64_t)blockIdx.x * kDiagThreads + threadIdx.x;
  const int64_t lo = (first + blockIdx.y) * per;
  const int64_t n_rows = *n_live, hi = lo + per < n_rows ? lo + per : n_rows;
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  for (int64_t c0 = lo; c0 < hi; c0 += kDiagChunk) {
    const int cnt = hi - c0 < kDiagChunk ? (int)(hi - c0) : kDiagChunk;
    __syncthreads();
    {
      const int mk = threadIdx.x >> 2, code = threadIdx.x & 3;
      double z = 0.0;
      if (mk < cnt) {
        const int32_t j = rows[c0 + mk];
        if (code != 1) {
          const double g = code == 0 ? 2.0 : (code == 2 ? 1.0 : 0.0);
          z = (g - two_p[j]) * inv_s[j];
        }
        if (code == 0) at[mk] = j * wpr;
      }
      tab[mk][code] = z * z;
    }
    __syncthreads();
    if (w >= wpr) continue;
    auto add = [&](int k, uint32_t x) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int shift = 16 * (e >> 3) + 2 * ((e >> 2) & 1) + 4 * (e & 3);
        acc[e] += tab[k][(x >> shift) & 3u];
      }
    };
    // neighbouring rows (most chunks): addresses that do not wait for a lookup (0.78 ms with)
    const uint32_t* p = geno + at[0] + w;
    if (at[cnt - 1] - at[0] == (cnt - 1) * wpr) {
#pragma unroll 8
      for (int k = 0; k < cnt; ++k) add(k, __ldg(p + (int64_t)k * wpr));
    } else {
#pragma unroll 8
      for (int k = 0; k < cnt; ++k) add(k, __ldg(geno + at[k] + w));
    }
  }
  if (w >= wpr) return;
  double2* o = reinterpret_cast<double2*>(partial + ((int64_t)blockIdx.y * wpr + w) * 16);
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = make_double2(acc[2 * e], acc[2 * e + 1]);
}

// (more: after the ranges that out already has)
__global__ void grm_diag_finish(const double* __restrict__ partial, int splits, int64_t n_pad,
                                int64_t n, bool more, double scale, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = more ? out[i] : 0.0;
#pragma unroll 4
  for (int k = 0; k < splits; ++k) s += partial[(int64_t)k * n_pad + i];
  out[i] = s * scale;
}

}  // namespace

size_t gram_partial_doubles(int64_t n, int a, int b) {
  return (size_t)gram_chunks(n, a, b) * (size_t)a * (size_t)b;
}

// A product is cut into more than one chunk only while chunks x tiles <= kGramBlocks, and has at
// most kG^2 sums per tile: more than one chunk's sums are at most kGramBlocks kG^2 in all.
size_t gram_partial_most(int64_t n, int a, int b) {
  const size_t sums = (size_t)a * (size_t)b, by_rows = (size_t)ceil_div(n, (int64_t)2048);
  return std::min(by_rows * sums, std::max(sums, (size_t)kGramBlocks * kG * kG));
}

cudaError_t gram(const double* A, int a, const double* B, int b, int64_t n, int64_t ld,
                 double* partial, size_t cap, double* out, cudaStream_t st, int tile) {
  if (gram_partial_doubles(n, a, b) > cap) return cudaErrorInvalidValue;
  const int nch = gram_chunks(n, a, b);
  const int64_t chunk = round_up(ceil_div(n, nch), kG);
  // 32 x 32 tiles while they give every SM two blocks, else 16 x 16
  const int64_t tiles4 = ceil_div(a, 32) * ceil_div(b, 32);
  if (tile ? tile == 32 : tiles4 * nch >= 296)
    gram_kernel<4><<<dim3((unsigned)nch, (unsigned)tiles4), 64, 0, st>>>(A, a, B, b, n, ld, chunk,
                                                                          partial);
  else
    gram_kernel<2><<<dim3((unsigned)nch, (unsigned)(ceil_div(a, 16) * ceil_div(b, 16))), 64, 0, st>>>(
        A, a, B, b, n, ld, chunk, partial);
  const int64_t count = (int64_t)a * b;
  gram_reduce<<<(unsigned)ceil_div(count, 256), 256, 0, st>>>(partial, nch, count, out);
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t combo(const double* V, int m, const double* G, int q, double* Y, bool add, int64_t n,
                  int64_t ld, cudaStream_t st) {
  if (m <= 0 || q <= 0) return cudaSuccess;
  const dim3 grid((unsigned)ceil_div(n, 256), (unsigned)ceil_div(q, 8));
  combo_kernel<<<grid, 256, (size_t)m * 8 * sizeof(double), st>>>(V, m, G, q, Y, add ? 1 : 0, n,
                                                                  ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t sigma_image(const double* v, const double* kv, const double* wmax, double tau0,
                        double tau1, double* v_out, double* kv_out, double* out, int64_t n,
                        int64_t ld, int q, cudaStream_t st) {
  if (q <= 0) return cudaSuccess;
  sigma_image_kernel<<<dim3((unsigned)ceil_div(ld, 256), (unsigned)q), 256, 0, st>>>(
      v, kv, wmax, tau0, tau1, v_out, kv_out, out, n, ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t sub_cols(const double* a, const double* b, double* out, int64_t n, int64_t ld, int q,
                     cudaStream_t st) {
  if (q <= 0) return cudaSuccess;
  sub_cols_kernel<<<dim3((unsigned)ceil_div(n, 256), (unsigned)q), 256, 0, st>>>(a, b, out, n, ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t learn_features(const double* x, const double* b, const double* bnext, const double* w,
                           const double* wnext, const double* diagk, const double* ku, int n_sk,
                           const double* scales, double tau0, double tau1, double dmean,
                           int64_t n, int64_t ld, int q, float* F, cudaStream_t st) {
  learn_features_kernel<<<dim3((unsigned)ceil_div(n, 256), (unsigned)q), 256, 0, st>>>(
      x, b, bnext, w, wnext, diagk, ku, n_sk, scales, tau0, tau1, dmean, n, ld, q, F);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t learn_targets(const double* x1, const double* x0, const double* s, int64_t n,
                          int64_t ld, int q, float* T, cudaStream_t st) {
  learn_targets_kernel<<<dim3((unsigned)ceil_div(n, 256), (unsigned)q), 256, 0, st>>>(x1, x0, s, n,
                                                                                     ld, T);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t learn_to_cols(const float* y, int64_t n, int64_t ld, int q, double* out,
                          cudaStream_t st) {
  learn_to_cols_kernel<<<dim3((unsigned)ceil_div(n, 256), (unsigned)q), 256, 0, st>>>(y, n, ld, out);
  count_launches(1);
  return cudaGetLastError();
}

Status grm_diag(saige_grm* h, double* out, cudaStream_t st) {
  const int64_t m_used = h->masked ? h->m_active : h->m_eff;
  const double scale = m_used > 0 ? 1.0 / (double)m_used : 0.0;
  // about eight blocks per SM over (windows of 4,096 samples) x (marker ranges)
  // (at most m_used rows are live)
  const int64_t windows = ceil_div(h->wpr, (int64_t)kDiagThreads);
  const int64_t most = std::max<int64_t>(1, ceil_div(m_used, (int64_t)kDiagChunk));
  const int64_t want = std::min(most, ceil_div((int64_t)148 * 8, windows));
  const int64_t per = round_up(ceil_div(std::max<int64_t>(m_used, 1), want), kDiagChunk);
  const int64_t splits = std::max<int64_t>(1, ceil_div(m_used, per));
  const int64_t blocks = std::max<int64_t>(1, ceil_div(h->m, (int64_t)kLiveRows));
  DevBuf partial, list;
  SG_TRY(list.reserve((size_t)(h->m + blocks + 1) * sizeof(int32_t)));
  // all ranges at once; when memory is short, as many at a time as fit
  int64_t at_once = splits;
  Status room = partial.reserve((size_t)at_once * h->n_pad * sizeof(double));
  while (room.code == SAIGE_ENOMEM && at_once > 1) {
    at_once = ceil_div(at_once, (int64_t)2);
    set_error("");
    room = partial.reserve((size_t)at_once * h->n_pad * sizeof(double));
  }
  SG_TRY(room);
  int32_t *rows = list.as<int32_t>(), *counts = rows + h->m, *n_live = counts + blocks;
  const uint8_t* excl = h->masked ? h->excl.as<uint8_t>() : nullptr;
  // the buffers are used on st only
  ReleaseScope rs(ReleaseMode::kStream, st);
  live_count_kernel<<<(unsigned)blocks, kLiveRows, 0, st>>>(h->inv_s, excl, h->m, counts);
  live_list_kernel<<<(unsigned)blocks, kLiveRows, 0, st>>>(h->inv_s, excl, h->m, counts, rows,
                                                           n_live);
  for (int64_t s0 = 0; s0 < splits; s0 += at_once) {
    const int64_t k = std::min(at_once, splits - s0);
    grm_diag_kernel<<<dim3((unsigned)windows, (unsigned)k), kDiagThreads, 0, st>>>(
        h->geno, h->wpr, h->two_p, h->inv_s, rows, n_live, per, s0, partial.as<double>());
    grm_diag_finish<<<(unsigned)ceil_div(h->n, 256), 256, 0, st>>>(
        partial.as<double>(), (int)k, h->n_pad, h->n, s0 > 0, s0 + k == splits ? scale : 1.0, out);
    count_launches(2);
  }
  count_launches(2);
  SG_CHECK_LAUNCH();
  partial.release();
  list.release();
  return Status();
}

}  // namespace saige
