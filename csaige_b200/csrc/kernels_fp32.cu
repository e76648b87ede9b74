// FP32 GRM product on CUDA cores: the saige-rs arithmetic of
// OnTheFlyGrm::mat_vec (saige-core/src/glmm/pcg.rs:128-180) — z rounded to
// f32 per marker and code exactly as OnTheFlyGrm::new (pcg.rs:101-122), v
// rounded to f32, f32 products and sums — read straight from the 2-bit rows.
//
// Decode: each nibble of a packed word holds two samples' codes (the device
// word layout pairs samples (k, k+4) and (k+4, k+8)); the nibble indexes a
// per-marker table of 16 float2 entries (z(code_lo), z(code_hi)) held in
// shared memory: one 64-bit shared load per two samples.  The 16 entries span all 32
// banks, so a warp's lookups never conflict.
//   pass A  u_m  = sum_i z_mi v_i        (block = kMarkersA markers x all samples)
//   pass B  y_i  = sum_m z_mi u_m        (block = a window of samples x a marker split)
// Up to eight columns (C; pass B: four) share one decode.  A column's f32 operations and their order do
// not depend on C or on the block shapes below: pass A keeps one packed f32x2 chain per
// (marker, warp slice, lane) over the slice's words and nibbles, pass B one per (nibble of
// a word, marker split) over the split's markers, with every product rounded before it is
// added.  Pass B writes per-split partial sums, summed in a fixed order by the finish
// kernel, so results are run-to-run deterministic.
//
// Bound: the lookups' shared-memory wavefronts (two per pair of samples and warp) for one
// column, the FP32 pipe and the loads of v for many.  At 20,011 x 29,000, pass A / pass B:
// 170 / 93 us per column when each column decoded for itself, with 64-byte strided loads of
// v and four words in flight; now 123 / 96 us for one column, 204 / 211 us for four, 344 /
// 416 us for eight (43 / 52 us per column).
#include "common.cuh"
#include "kernels.cuh"

namespace saige {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kChunkB = 128;    // markers per table chunk in pass B

__device__ __forceinline__ float zsel(const float4& z, int c) {
  return c == 0 ? z.x : (c == 1 ? z.y : (c == 2 ? z.z : z.w));
}

// v32 layout: the 16 samples of word wo as eight pairs k (the codes of nibble k), pairs
// 2h and 2h + 1 as one float4 at ((wo / 32) 4 + h) 32 + wo % 32, so that a warp's loads of
// 32 words are contiguous.  Position of sample i:
__device__ __forceinline__ int64_t v32_at(int64_t i) {
  const int64_t wo = i >> 4;
  const int j = (int)(i & 15);
  const int k = (j & 3) + ((j >> 3) << 2), second = (j >> 2) & 1;
  return (((((wo >> 5) * 4 + (k >> 1)) * 32) + (wo & 31)) << 2) + 2 * (k & 1) + second;
}

// kMarkersA markers per block and C columns per thread: kMarkersA * C accumulator pairs
// (at most 32: 64 registers).  The next step's words are loaded while this one's are used.
template <int C, int kMarkersA>
__global__ void __launch_bounds__(kThreads, C > 4 ? 1 : (C > 1 ? 2 : 3))
    fp32_zt_kernel(const uint32_t* __restrict__ geno, int64_t wpr, const float4* __restrict__ zlut,
                   int64_t m_pad, const float* __restrict__ v32, float* __restrict__ u) {
  __shared__ float2 tab[kMarkersA][16];
  __shared__ float part[kWarps][kMarkersA][C];
  const int64_t m0 = (int64_t)blockIdx.x * kMarkersA;
  for (int e = threadIdx.x; e < kMarkersA * 16; e += kThreads) {
    const int mb = e >> 4, nib = e & 15;
    const float4 z = zlut[m0 + mb];
    tab[mb][nib] = make_float2(zsel(z, nib & 3), zsel(z, nib >> 2));
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2 acc[kMarkersA][C];
#pragma unroll
  for (int mb = 0; mb < kMarkersA; ++mb)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[mb][c] = make_float2(0.f, 0.f);
  const int n_steps = (int)(wpr / 32);
  const int64_t plane = wpr * 4;  // float4 per column
  const uint32_t* rows = geno + m0 * wpr + lane;
  const float4* vp = reinterpret_cast<const float4*>(v32) + lane;
  uint32_t w[kMarkersA], wn[kMarkersA];
#pragma unroll
  for (int mb = 0; mb < kMarkersA; ++mb)
    wn[mb] = warp < n_steps ? __ldg(rows + mb * wpr + warp * 32) : 0u;
  for (int s = warp; s < n_steps; s += kWarps) {
#pragma unroll
    for (int mb = 0; mb < kMarkersA; ++mb) w[mb] = wn[mb];
    if (s + kWarps < n_steps) {
#pragma unroll
      for (int mb = 0; mb < kMarkersA; ++mb) wn[mb] = __ldg(rows + mb * wpr + (s + kWarps) * 32);
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      float4 v[C];
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = __ldg(vp + c * plane + (s * 4 + h) * 32);
#pragma unroll
      for (int mb = 0; mb < kMarkersA; ++mb) {
        const float2 t0 = tab[mb][(w[mb] >> (8 * h)) & 15u];
        const float2 t1 = tab[mb][(w[mb] >> (8 * h + 4)) & 15u];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          acc[mb][c] = __ffma2_rn(t0, make_float2(v[c].x, v[c].y), acc[mb][c]);
          acc[mb][c] = __ffma2_rn(t1, make_float2(v[c].z, v[c].w), acc[mb][c]);
        }
      }
    }
  }
#pragma unroll
  for (int mb = 0; mb < kMarkersA; ++mb)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float t = warp_sum(acc[mb][c].x + acc[mb][c].y);
      if (lane == 0) part[warp][mb][c] = t;
    }
  __syncthreads();
  if (threadIdx.x < kMarkersA * C) {
    const int mb = threadIdx.x / C, c = threadIdx.x % C;
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < kWarps; ++q) s += part[q][mb][c];
    u[c * m_pad + m0 + mb] = s;
  }
}

// kParts threads share a word (each takes 8 / kParts of its nibbles): 1, or 4 where a
// thread per word would leave the SMs short of warps.  One column looks z u up (the
// products of the 16 pairs with u are formed once per marker and block); several look z up
// and multiply by each column's u.
template <int C, int kParts>
__global__ void __launch_bounds__(kThreads, C > 2 ? 2 : 3)
    fp32_z_kernel(const uint32_t* __restrict__ geno, int64_t wpr, const float4* __restrict__ zlut,
                  int64_t m_pad, const float* __restrict__ u, float* __restrict__ ypart,
                  int64_t n_pad, int64_t per_split, int n_splits, float2 neg_zero) {
  constexpr int kNib = 8 / kParts;
  constexpr int kAhead = 8;  // words in flight
  __shared__ float2 tab[kChunkB][16];
  __shared__ float2 us[C > 1 ? kChunkB : 1][C];
  const int64_t ms = (int64_t)blockIdx.y * per_split;
  int64_t me = ms + per_split;
  if (me > m_pad) me = m_pad;
  const int64_t wo = (int64_t)blockIdx.x * (kThreads / kParts) + threadIdx.x / kParts;
  const int k0 = (threadIdx.x % kParts) * kNib;
  const bool active = wo < wpr;
  float2 acc[C][kNib];
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int k = 0; k < kNib; ++k) acc[c][k] = make_float2(0.f, 0.f);
  for (int64_t c0 = ms; c0 < me; c0 += kChunkB) {
    const int cnt = (int)((me - c0) < kChunkB ? (me - c0) : kChunkB);
    const uint32_t* p = geno + c0 * wpr + wo;
    uint32_t wn[kAhead];
    if (active) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) wn[q] = q < cnt ? __ldg(p + (int64_t)q * wpr) : 0u;
    }
    __syncthreads();  // every thread is done with the chunk before
    for (int e = threadIdx.x; e < cnt * 16; e += kThreads) {
      const int mb = e >> 4, nib = e & 15;
      const float4 z = zlut[c0 + mb];
      float2 t = make_float2(zsel(z, nib & 3), zsel(z, nib >> 2));
      if (C == 1) {
        const float um = u[c0 + mb];
        t = make_float2(t.x * um, t.y * um);
      }
      tab[mb][nib] = t;
    }
    if (C > 1)
      for (int e = threadIdx.x; e < cnt * C; e += kThreads) {
        const int c = e / cnt, mb = e - c * cnt;
        const float um = u[c * m_pad + c0 + mb];
        us[mb][c] = make_float2(um, um);
      }
    __syncthreads();
    if (!active) continue;
    auto marker = [&](int mk, uint32_t word) {
      const uint32_t x = kParts > 1 ? word >> (4 * k0) : word;
      float2 uc[C];
      if (C > 1) {
#pragma unroll
        for (int c = 0; c < C; ++c) uc[c] = us[mk][c];
      }
#pragma unroll
      for (int k = 0; k < kNib; ++k) {
        const float2 t = tab[mk][(x >> (4 * k)) & 15u];
        if (C == 1) {
          acc[0][k] = __fadd2_rn(acc[0][k], t);
        } else {
#pragma unroll
          for (int c = 0; c < C; ++c)
            // the rounded product as t u + (-0), with the -0 from the launch: ptxas fuses a
            // packed multiply with the addition that follows, explicit rounding modes and
            // -fmad=false or not
            acc[c][k] = __fadd2_rn(acc[c][k], __ffma2_rn(t, uc[c], neg_zero));
        }
      }
    };
    int mb = 0;
    // whole batches without a branch between markers, so that lookups run ahead
    for (; mb + kAhead <= cnt; mb += kAhead) {
      uint32_t w[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) w[q] = wn[q];
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (mb + kAhead + q < cnt) wn[q] = __ldg(p + (int64_t)(mb + kAhead + q) * wpr);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) marker(mb + q, w[q]);
    }
#pragma unroll
    for (int q = 0; q < kAhead - 1; ++q)
      if (mb + q < cnt) marker(mb + q, wn[q]);
  }
  if (!active) return;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    float* o = ypart + ((int64_t)c * n_splits + blockIdx.y) * n_pad + wo * 16;
    if constexpr (kParts == 1) {
      float4* o4 = reinterpret_cast<float4*>(o);
      o4[0] = make_float4(acc[c][0].x, acc[c][1].x, acc[c][2].x, acc[c][3].x);
      o4[1] = make_float4(acc[c][0].y, acc[c][1].y, acc[c][2].y, acc[c][3].y);
      o4[2] = make_float4(acc[c][4].x, acc[c][5].x, acc[c][6].x, acc[c][7].x);
      o4[3] = make_float4(acc[c][4].y, acc[c][5].y, acc[c][6].y, acc[c][7].y);
    } else {
#pragma unroll
      for (int k = 0; k < kNib; ++k) {
        const int first = k0 + k + (k0 + k >= 4 ? 4 : 0);  // pair k: samples first, first + 4
        o[first] = acc[c][k].x;
        o[first + 4] = acc[c][k].y;
      }
    }
  }
}

__global__ void fp32_finish_kernel(const float* __restrict__ ypart, int n_splits, int64_t n_pad,
                                   int64_t n, float scale, Fp32Cols cols) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* y = ypart + (int64_t)blockIdx.y * n_splits * n_pad + i;
  // added in split order; 32 loads in flight (small cohorts have over a hundred splits)
  float s = 0.f;
  int q = 0;
  for (; q + 32 <= n_splits; q += 32) {
    float t[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) t[k] = __ldg(y + (int64_t)(q + k) * n_pad);
#pragma unroll
    for (int k = 0; k < 32; ++k) s += t[k];
  }
#pragma unroll 8
  for (; q < n_splits; ++q) s += __ldg(y + (int64_t)q * n_pad);
  cols.out[blockIdx.y][i] = (double)(s * scale);
}

__global__ void to_f32_kernel(Fp32Cols cols, int64_t n, int64_t n_pad, float* __restrict__ v32) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_pad)
    v32[blockIdx.y * n_pad + v32_at(i)] = i < n ? (float)cols.v[blockIdx.y][i] : 0.f;
}

}  // namespace

int fp32_z_splits(int64_t n_pad, int64_t m_pad) {
  const int64_t windows = ceil_div(n_pad / 16, kThreads);
  int64_t want = ceil_div(148 * 6, windows);
  const int64_t max_splits = ceil_div(m_pad, kChunkB);
  if (want > max_splits) want = max_splits;
  if (want < 1) want = 1;
  return (int)want;
}

cudaError_t launch_fp32_zt(const uint32_t* geno, int64_t wpr, const float4* zlut, int64_t m_pad,
                           const float* v32, int cols, float* u, cudaStream_t st) {
  auto go = [&](auto kern, int markers) {
    kern<<<(unsigned)(m_pad / markers), kThreads, 0, st>>>(geno, wpr, zlut, m_pad, v32, u);
    count_launches(1);
    return cudaGetLastError();
  };
  switch (cols) {
    case 1: return go(fp32_zt_kernel<1, 16>, 16);
    case 2: return go(fp32_zt_kernel<2, 16>, 16);
    case 3: return go(fp32_zt_kernel<3, 8>, 8);
    case 4: return go(fp32_zt_kernel<4, 8>, 8);
    case 5: return go(fp32_zt_kernel<5, 8>, 8);
    case 6: return go(fp32_zt_kernel<6, 8>, 8);
    case 7: return go(fp32_zt_kernel<7, 8>, 8);
    case 8: return go(fp32_zt_kernel<8, 8>, 8);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_fp32_z(const uint32_t* geno, int64_t wpr, const float4* zlut, int64_t m_pad,
                          const float* u, int cols, float* ypart, int n_splits, cudaStream_t st) {
  const int64_t per_split = round_up(ceil_div(m_pad, n_splits), 4);
  // a thread per word while that gives every SM 16 warps, else four
  const int parts = wpr * n_splits >= 148 * 512 ? 1 : 4;
  const float2 nz = make_float2(-0.0f, -0.0f);
  const dim3 grid((unsigned)ceil_div(wpr * parts, (int64_t)kThreads), (unsigned)n_splits);
  auto go = [&](auto one, auto four) {
    if (parts == 1)
      one<<<grid, kThreads, 0, st>>>(geno, wpr, zlut, m_pad, u, ypart, wpr * 16, per_split,
                                     n_splits, nz);
    else
      four<<<grid, kThreads, 0, st>>>(geno, wpr, zlut, m_pad, u, ypart, wpr * 16, per_split,
                                      n_splits, nz);
    count_launches(1);
    return cudaGetLastError();
  };
  switch (cols) {
    case 1: return go(fp32_z_kernel<1, 1>, fp32_z_kernel<1, 4>);
    case 2: return go(fp32_z_kernel<2, 1>, fp32_z_kernel<2, 4>);
    case 3: return go(fp32_z_kernel<3, 1>, fp32_z_kernel<3, 4>);
    case 4: return go(fp32_z_kernel<4, 1>, fp32_z_kernel<4, 4>);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_fp32_finish(const float* ypart, int n_splits, int64_t n_pad, int64_t n,
                               float scale, const Fp32Cols& cols, int n_cols, cudaStream_t st) {
  fp32_finish_kernel<<<dim3((unsigned)ceil_div(n, 128), (unsigned)n_cols), 128, 0, st>>>(
      ypart, n_splits, n_pad, n, scale, cols);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_to_f32(const Fp32Cols& cols, int n_cols, int64_t n, int64_t n_pad, float* v32,
                          cudaStream_t st) {
  to_f32_kernel<<<dim3((unsigned)ceil_div(n_pad, 256), (unsigned)n_cols), 256, 0, st>>>(cols, n,
                                                                                       n_pad, v32);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace saige
