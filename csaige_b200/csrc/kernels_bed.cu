// K1: gather the sample subset out of raw PLINK .bed rows, repack it into
// 128-byte-aligned 2-bit rows (device word layout, see to_device_layout), and
// count alleles and missing calls exactly.
//
// Replaces PlinkReader::read_marker_raw / read_marker (saige-geno/src/
// plink.rs:182-194, 237-249) and MarkerData::compute_af's sums
// (saige-geno/src/traits.rs:42-54): the counts are integers from popc over
// the code bit planes, so af = alt / (2 n_valid) computed from them on the
// host is bit-identical to the reference's f64 sum of 0/1/2 dosages.
#include "common.cuh"
#include "kernels.cuh"

namespace saige {

namespace {

constexpr int kThreads = 256;
constexpr int64_t kSmemRowMax = 200 * 1024;  // stage raw rows up to this size in shared memory
constexpr int64_t kSmemHalf = 112 * 1024;    // shared memory of one of two blocks on an SM

// Counts over a word of 16 codes; valid = even bits of the real samples.
__device__ __forceinline__ void count_word(uint32_t w, uint32_t valid, long long& alt,
                                           long long& miss) {
  const uint32_t lo = w & 0x55555555u;
  const uint32_t hi = (w >> 1) & 0x55555555u;
  const uint32_t hom_a1 = ~lo & ~hi & valid;  // 00 -> 2 copies of A1
  const uint32_t het = ~lo & hi & valid;      // 10 -> 1 copy
  const uint32_t mis = lo & ~hi & valid;      // 01 -> missing
  alt += 2 * __popc(hom_a1) + __popc(het);
  miss += __popc(mis);
}

// Device layout of a 32-bit word of 16 codes.  PLINK puts sample s at bits
// 2s; the packed rows put sample s = 4j + i at bit 16*(j>>1) + 2*(j&1) + 4i, so
// that each 4-sample group's codes sit in the low bits of four nibbles that one
// mask (or shift + mask) turns into a byte-permute selector.
__device__ __forceinline__ uint32_t nibble_spread16x2(uint32_t x) {
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  return (x | (x << 2)) & 0x33333333u;
}
__device__ __forceinline__ uint32_t to_device_layout(uint32_t plink_word) {
  return nibble_spread16x2(plink_word & 0x00FF00FFu) |
         (nibble_spread16x2((plink_word >> 8) & 0x00FF00FFu) << 2);
}

__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Stages raw row `row` (bpm bytes) in shared memory in 16-byte chunks of its aligned
// span (row byte b at row_s[off + b]); the chunks that reach past either end of the
// row, at most two, are copied byte by byte, so no load leaves the row.  Several
// independent chunk loads per thread are in flight at once.  Returns row_s + off.
// row_s holds round_up(bpm + 16, 16) bytes, 16-byte aligned.
__device__ __forceinline__ const uint8_t* copy_row(const uint8_t* row, int64_t bpm,
                                                   uint8_t* row_s) {
  const int off = (int)(reinterpret_cast<uintptr_t>(row) & 15u);
  const uint4* base = reinterpret_cast<const uint4*>(row - off);
  const int64_t n16 = (off + bpm + 15) / 16;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < n16; i += blockDim.x) {
    const int64_t lo = 16 * i - off;
    if (lo >= 0 && lo + 16 <= bpm) {
      reinterpret_cast<uint4*>(row_s)[i] = __ldg(base + i);
    } else {
      for (int k = 0; k < 16; ++k) {
        const int64_t b = lo + k;
        if (b >= 0 && b < bpm) row_s[16 * i + k] = row[b];
      }
    }
  }
  return row_s + off;
}

// copy_row by the whole block, then the barrier that makes the row readable.
__device__ __forceinline__ const uint8_t* stage_row(const uint8_t* row, int64_t bpm,
                                                    uint8_t* row_s) {
  const uint8_t* p = copy_row(row, bpm, row_s);
  __syncthreads();
  return p;
}

// The codes of samples sidx[0 .. kn) (kn <= 16) of a raw row as one PLINK-order
// word (sample k at bits 2k); vec: sidx is 16-byte aligned and kn == 16, so the
// indices are read as four 16-byte loads.
__device__ __forceinline__ uint32_t gather_word(const uint8_t* src, const int32_t* sidx, int kn,
                                                bool vec) {
  uint32_t word = 0;
  if (vec) {
    const int4* s4 = reinterpret_cast<const int4*>(sidx);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int4 v = __ldg(s4 + g);
      const int32_t ss[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t code = (src[ss[e] >> 2] >> ((ss[e] & 3) * 2)) & 3u;
        word |= code << (2 * (4 * g + e));
      }
    }
  } else {
    for (int k = 0; k < kn; ++k) {
      const int32_t s = sidx[k];
      const uint32_t code = (src[s >> 2] >> ((s & 3) * 2)) & 3u;
      word |= code << (2 * k);
    }
  }
  return word;
}

// A row's counts from its threads' counts: kGroup threads (one warp, or the whole block
// of kThreads) share a row; thread 0 of the group writes.
template <int kGroup>
__device__ __forceinline__ void store_counts(long long alt, long long miss, int64_t* out) {
  alt = warp_sum_ll(alt);
  miss = warp_sum_ll(miss);
  const int lane = threadIdx.x & 31;
  if constexpr (kGroup == 32) {
    if (lane == 0) {
      out[0] = alt;
      out[1] = miss;
    }
  } else {
    __shared__ long long red[2][kGroup / 32];
    const int wid = threadIdx.x >> 5;
    if (lane == 0) {
      red[0][wid] = alt;
      red[1][wid] = miss;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      long long a = 0, mm = 0;
      for (int k = 0; k < kGroup / 32; ++k) {
        a += red[0][k];
        mm += red[1][k];
      }
      out[0] = a;
      out[1] = mm;
    }
  }
}

// All samples in .fam order: word j of a packed row is bytes 4j .. 4j+3 of the raw row,
// whose start (3 + row bpm) is not aligned, so a word is cut out of the two aligned words
// around it.  The aligned word in front starts at most 3 bytes before the row, still inside
// the .bed (the header is 3 bytes); the words near the row's end, whose aligned words
// would reach past it, are read byte by byte.  kGroup threads per row: a warp for short
// rows, the block for long ones.
// Bound: issue, about 20 instructions per 16 samples, three of them population counts
// at half rate, beside DRAM.  The counts come from three sums over the code bits (both
// planes together, the low plane, and their product).  40,000 rows of 200,000 samples:
// counts 1.35 ms with a byte per load, 64-bit counters and every word handled as if it
// were the last; now 0.48 ms with a block per row, 0.39 ms with a warp (5.1 TB/s).
// kMask: the counts of a sample subset without repeats, whose other samples the mask turns
// into 11 (which counts as nothing).
template <int kGroup, bool kOut, bool kCounts, bool kMask = false>
__global__ void __launch_bounds__(kThreads)
    bed_rows_kernel(const uint8_t* __restrict__ bed, int64_t bpm,
                    const int64_t* __restrict__ src_rows, int64_t n_rows, int64_t n,
                    uint32_t* __restrict__ out, int64_t wpr, int64_t* __restrict__ counts,
                    const SubsetMask mask = SubsetMask()) {
  if (kMask && *mask.repeats) return;  // bed_subset_kernel counts
  const int64_t r = (int64_t)blockIdx.x * (kThreads / kGroup) + threadIdx.x / kGroup;
  if (r >= n_rows) return;  // whole warps (kGroup 32) or, never, whole blocks
  const uint8_t* row = bed + 3 + src_rows[r] * bpm;
  const int off = (int)(reinterpret_cast<uintptr_t>(row) & 3u);
  const uint32_t* base = reinterpret_cast<const uint32_t*>(row - off);
  uint32_t* dst = kOut ? out + r * wpr : nullptr;
  // words of 16 samples whose two aligned words end inside the row (n < 2^31: n_words < 2^27)
  const int n_words = (int)(kOut ? wpr : (n + 15) / 16);
  const int64_t safe = bpm + off >= 8 ? (bpm + off - 8) / 4 + 1 : 0;
  const int n_fast = (int)(safe < n / 16 ? safe : n / 16);
  uint32_t both = 0, low = 0, prod = 0;  // over the fast words: set bits, low bits, 11 codes
  int j = threadIdx.x % kGroup;
  const int first = j;
#pragma unroll 8
  for (; j < n_fast; j += kGroup) {
    uint32_t w = __funnelshift_r(__ldg(base + j), __ldg(base + j + 1), 8 * off);
    if (kMask) w |= __ldg(mask.others + j);
    if (kCounts) {
      const uint32_t lo = w & 0x55555555u;
      both += __popc(w);
      low += __popc(lo);
      prod += __popc(lo & (w >> 1));
    }
    if (kOut) dst[j] = to_device_layout(w);
  }
  long long alt = 0, miss = 0;
  if (kCounts) {
    // per code: 00 two alternative alleles, 10 (high bit alone) one, 01 missing
    const int fast = n_fast > first ? (n_fast - first + kGroup - 1) / kGroup : 0;
    const long long high = (long long)both - low;
    alt = 32LL * fast - 2LL * low - high + (long long)prod;
    miss = (long long)low - (long long)prod;
  }
  for (; j < n_words; j += kGroup) {
    // Padding samples are coded 11 (genotype 0, not missing): every vector the
    // products read is zero there, so they contribute nothing to any sum.
    const int64_t left = n - 16 * (int64_t)j;
    uint32_t w = 0xFFFFFFFFu;
    if (left > 0) {
      uint32_t word = 0;
      for (int b = 0; b < 4; ++b) {
        const int64_t bi = 4 * (int64_t)j + b;
        if (bi < bpm) word |= (uint32_t)row[bi] << (8 * b);
      }
      if (kMask) word |= __ldg(mask.others + j);
      const uint32_t keep = left >= 16 ? 0xFFFFFFFFu : ((1u << (2 * (int)left)) - 1u);
      if (kCounts) count_word(word, keep & 0x55555555u, alt, miss);
      w = to_device_layout((word & keep) | ~keep);
    }
    if (kOut) dst[j] = w;
  }
  if (kCounts) store_counts<kGroup>(alt, miss, counts + 2 * r);
}

// A sample subset, kRows raw rows per block staged in shared memory (kRows = 0: one row,
// read from global memory, for rows too long to stage): each thread loads the 16 sample
// indices of a packed word once and gathers that word from every staged row.  Bound: the
// index loads (64 bytes from L2 per 4-byte word and row with a row per block) and the bank
// conflicts of the byte gathers.  39,001 rows of 60,000 of 150,001 samples: 2.10 ms with a
// row per block, 1.59 ms with three.  (Lane = sample with two ballots per 32 samples has no
// bank conflicts but took 2.37 ms: the votes bound it.)
constexpr int kSubsetThreads = 512;

template <int kRows>
__global__ void __launch_bounds__(kSubsetThreads, 2)
    bed_subset_kernel(const uint8_t* __restrict__ bed, int64_t bpm,
                      const int64_t* __restrict__ src_rows, int64_t n_rows,
                      const int32_t* __restrict__ sidx, int64_t n, uint32_t* __restrict__ out,
                      int64_t wpr, int64_t* __restrict__ counts,
                      const unsigned int* __restrict__ only_if) {
  constexpr int R = kRows ? kRows : 1;
  if (only_if && !*only_if) return;  // counted through the mask, or compressed
  extern __shared__ __align__(16) uint8_t row_s[];
  __shared__ int red[2 * R][kSubsetThreads / 32];
  const int64_t r0 = (int64_t)blockIdx.x * R;
  const int nr = n_rows - r0 < R ? (int)(n_rows - r0) : R;
  const int64_t stride = (bpm + 31) / 16 * 16;  // round_up(bpm + 16, 16)
  const uint8_t* src[R];
  const uint8_t* raw[R];
#pragma unroll
  for (int q = 0; q < R; ++q) raw[q] = bed + 3 + src_rows[r0 + (q < nr ? q : 0)] * bpm;
#pragma unroll
  for (int q = 0; q < R; ++q)
    src[q] = kRows ? copy_row(raw[q], bpm, row_s + q * stride) : raw[q];
  if (kRows) __syncthreads();
  const bool vec = (reinterpret_cast<uintptr_t>(sidx) & 15u) == 0;
  const int64_t n_real = (n + 15) / 16;
  const int64_t n_words = out ? wpr : n_real;
  int alt[R], miss[R];
#pragma unroll
  for (int q = 0; q < R; ++q) alt[q] = miss[q] = 0;
  for (int64_t j = threadIdx.x; j < n_words; j += kSubsetThreads) {
    uint32_t w[R];
    if (j < n_real) {
      const int64_t k0 = 16 * j;
      const int kn = n - k0 < 16 ? (int)(n - k0) : 16;
#pragma unroll
      for (int q = 0; q < R; ++q) w[q] = 0u;
      if (vec && kn == 16) {
        const int4* s4 = reinterpret_cast<const int4*>(sidx + k0);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int4 v = __ldg(s4 + g);
          const int32_t ss[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int at = ss[e] >> 2, sh = (ss[e] & 3) * 2;
#pragma unroll
            for (int q = 0; q < R; ++q)
              w[q] |= (((uint32_t)src[q][at] >> sh) & 3u) << (2 * (4 * g + e));
          }
        }
      } else {
        for (int k = 0; k < kn; ++k) {
          const int32_t s = sidx[k0 + k];
#pragma unroll
          for (int q = 0; q < R; ++q)
            w[q] |= (((uint32_t)src[q][s >> 2] >> ((s & 3) * 2)) & 3u) << (2 * k);
        }
      }
      const uint32_t keep = kn >= 16 ? 0xFFFFFFFFu : ((1u << (2 * kn)) - 1u);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        long long a = 0, mm = 0;
        count_word(w[q], keep & 0x55555555u, a, mm);
        alt[q] += (int)a;
        miss[q] += (int)mm;
        w[q] = to_device_layout((w[q] & keep) | ~keep);
      }
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) w[q] = 0xFFFFFFFFu;
    }
    if (out) {
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (q < nr) out[(r0 + q) * wpr + j] = w[q];
    }
  }
  if (!counts) return;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    // a warp's counts (at most n / 8) fit in 32 bits, a row's need not
    const int a = __reduce_add_sync(0xffffffffu, alt[q]);
    const int mm = __reduce_add_sync(0xffffffffu, miss[q]);
    if (lane == 0) {
      red[2 * q][wid] = a;
      red[2 * q + 1][wid] = mm;
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * nr) {
    long long s = 0;
    for (int k = 0; k < kSubsetThreads / 32; ++k) s += red[threadIdx.x][k];
    counts[2 * r0 + threadIdx.x] = s;
  }
}

// Counts of several sample subsets ("cohorts") of the same raw rows in one pass:
// block = marker j0 + blockIdx.x, staged once in shared memory; for cohort c, the
// samples sidx[offs[c] .. offs[c] + n_c) (offs[c] a multiple of 16) are gathered 16 at
// a time and counted as bed_gather_kernel counts them.  counts[(c m_tot + j) 2 + e]:
// e = 0 alt-allele count, 1 missing count.
__global__ void __launch_bounds__(kThreads)
    bed_count_cohorts_kernel(const uint8_t* __restrict__ bed, int64_t bpm, int64_t j0,
                             const int32_t* __restrict__ sidx, const int64_t* __restrict__ offs,
                             const int64_t* __restrict__ ns, int n_cohorts, int64_t m_tot,
                             long long* __restrict__ counts) {
  extern __shared__ __align__(16) uint8_t row_s[];
  __shared__ long long red[2][kThreads / 32];
  const int64_t j = j0 + blockIdx.x;
  const uint8_t* src = stage_row(bed + 3 + j * bpm, bpm, row_s);
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = 0; c < n_cohorts; ++c) {
    const int32_t* sc = sidx + offs[c];
    const int64_t n = ns[c];
    const bool vec = (reinterpret_cast<uintptr_t>(sc) & 15u) == 0;
    long long alt = 0, miss = 0;
    for (int64_t w = threadIdx.x; w < (n + 15) / 16; w += blockDim.x) {
      const int64_t k0 = 16 * w;
      const int kn = (n - k0) < 16 ? (int)(n - k0) : 16;
      const uint32_t word = gather_word(src, sc + k0, kn, vec && kn == 16);
      const uint32_t keep = kn >= 16 ? 0xFFFFFFFFu : ((1u << (2 * kn)) - 1u);
      count_word(word, keep & 0x55555555u, alt, miss);
    }
    alt = warp_sum_ll(alt);
    miss = warp_sum_ll(miss);
    if (lane == 0) {
      red[0][wid] = alt;
      red[1][wid] = miss;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      long long a = 0, mm = 0;
      for (int k = 0; k < kThreads / 32; ++k) {
        a += red[0][k];
        mm += red[1][k];
      }
      counts[2 * ((int64_t)c * m_tot + j)] = a;
      counts[2 * ((int64_t)c * m_tot + j) + 1] = mm;
    }
    __syncthreads();  // red is reused by the next cohort
  }
}

// The packed rows of several sample subsets from one pass over the raw rows: block =
// rpb consecutive raw markers from j0 + blockIdx.x rpb, staged once; for every cohort,
// each thread loads the sample indices of a 16-sample word once and gathers that word
// from each staged row the cohort keeps (row_of[j] >= 0), repacked and written exactly
// as bed_gather_kernel writes it (padding samples coded 11).
constexpr int kGatherRowsMax = 4;
constexpr int kGatherThreads = 1024;  // one block of four staged rows per SM: 32 warps

__global__ void __launch_bounds__(kGatherThreads)
    bed_gather_cohorts_kernel(const uint8_t* __restrict__ bed, int64_t bpm, int64_t j0,
                              int64_t n_rows, int rpb, const int32_t* __restrict__ sidx,
                              const CohortSet set) {
  extern __shared__ __align__(16) uint8_t row_s[];
  const int64_t stride = (bpm + 31) / 16 * 16;  // round_up(bpm + 16, 16)
  const int64_t jb = j0 + (int64_t)blockIdx.x * rpb;
  const int64_t left = j0 + n_rows - jb;
  const int nr = left < rpb ? (int)left : rpb;
  const uint8_t* src[kGatherRowsMax];
#pragma unroll
  for (int q = 0; q < kGatherRowsMax; ++q)
    src[q] = q < nr ? stage_row(bed + 3 + (jb + q) * bpm, bpm, row_s + q * stride) : nullptr;
  for (int c = 0; c < set.n; ++c) {
    const CohortRows& cr = set.c[c];
    int32_t r[kGatherRowsMax];
    bool any = false;
#pragma unroll
    for (int q = 0; q < kGatherRowsMax; ++q) {
      r[q] = q < nr ? cr.row_of[(jb + q) * cr.row_stride] : -1;
      any |= r[q] >= 0;
    }
    if (!any) continue;
    const int32_t* sc = sidx + cr.sidx_off;
    const bool vec = (reinterpret_cast<uintptr_t>(sc) & 15u) == 0;
    const int64_t n_real = (cr.n + 15) / 16;
    for (int64_t w = threadIdx.x; w < cr.wpr; w += blockDim.x) {
      if (w >= n_real) {
#pragma unroll
        for (int q = 0; q < kGatherRowsMax; ++q)
          if (r[q] >= 0) cr.geno[(int64_t)r[q] * cr.wpr + w] = 0xFFFFFFFFu;
        continue;
      }
      const int64_t k0 = 16 * w;
      const int kn = (cr.n - k0) < 16 ? (int)(cr.n - k0) : 16;
      int32_t ss[16];
      if (vec && kn == 16) {
        const int4* s4 = reinterpret_cast<const int4*>(sc + k0);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int4 v = __ldg(s4 + g);
          ss[4 * g] = v.x;
          ss[4 * g + 1] = v.y;
          ss[4 * g + 2] = v.z;
          ss[4 * g + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) ss[e] = e < kn ? sc[k0 + e] : 0;
      }
      const uint32_t keep = kn >= 16 ? 0xFFFFFFFFu : ((1u << (2 * kn)) - 1u);
#pragma unroll
      for (int q = 0; q < kGatherRowsMax; ++q) {
        if (r[q] < 0) continue;
        uint32_t word = 0;
#pragma unroll
        for (int e = 0; e < 16; ++e)
          word |= ((uint32_t)(src[q][ss[e] >> 2] >> ((ss[e] & 3) * 2)) & 3u) << (2 * e);
        cr.geno[(int64_t)r[q] * cr.wpr + w] = to_device_layout((word & keep) | ~keep);
      }
    }
  }
}

}  // namespace

cudaError_t launch_bed_gather_cohorts(const uint8_t* bed, int64_t bpm, int64_t j0, int64_t n_rows,
                                      const int32_t* sidx, const CohortSet& set,
                                      cudaStream_t st) {
  if (n_rows <= 0 || set.n <= 0) return cudaSuccess;
  if (set.n > kCohortsPerLaunch) return cudaErrorInvalidValue;
  if (bpm > kSmemRowMax) return cudaErrorInvalidValue;
  // as many rows per block as 200 KB of shared memory hold (each index load then serves
  // all of them), at most kGatherRowsMax
  const int64_t stride = round_up(bpm + 16, 16);
  const int rpb = (int)std::max<int64_t>(1, std::min<int64_t>(kGatherRowsMax, kSmemRowMax / stride));
  const size_t smem = (size_t)(stride * rpb);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(bed_gather_cohorts_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  bed_gather_cohorts_kernel<<<(unsigned)ceil_div(n_rows, rpb), kGatherThreads, smem, st>>>(
      bed, bpm, j0, n_rows, rpb, sidx, set);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_bed_count_cohorts(const uint8_t* bed, int64_t bpm, int64_t j0, int64_t n_rows,
                                     const int32_t* sidx, const int64_t* offs, const int64_t* ns,
                                     int n_cohorts, int64_t m_tot, long long* counts,
                                     cudaStream_t st) {
  if (n_rows <= 0) return cudaSuccess;
  if (bpm > kSmemRowMax) return cudaErrorInvalidValue;  // rows must fit in shared memory
  const size_t smem = (size_t)round_up(bpm + 16, 16);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(bed_count_cohorts_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  bed_count_cohorts_kernel<<<(unsigned)n_rows, kThreads, smem, st>>>(bed, bpm, j0, sidx, offs, ns,
                                                                    n_cohorts, m_tot, counts);
  count_launches(1);
  return cudaGetLastError();
}

__global__ void subset_mask_kernel(const int32_t* __restrict__ sidx, int64_t n,
                                   uint32_t* __restrict__ others,
                                   unsigned int* __restrict__ repeats,
                                   unsigned int* __restrict__ unsorted) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t s = sidx[i];
  const uint32_t bits = 3u << (2 * (s & 15));
  if (!(atomicAnd(&others[s >> 4], ~bits) & bits)) *repeats = 1u;
  if (i + 1 < n && sidx[i + 1] <= s) *unsorted = 1u;
}

// The even bits 0, 2, .. of x as bits 0, 1, ..; and each of 16 bits as a pair.
__device__ __forceinline__ uint32_t gather_even(uint32_t x) {
  x &= 0x55555555u;
  x = (x | (x >> 1)) & 0x33333333u;
  x = (x | (x >> 2)) & 0x0F0F0F0Fu;
  x = (x | (x >> 4)) & 0x00FF00FFu;
  return (x | (x >> 8)) & 0xFFFFu;
}
__device__ __forceinline__ uint32_t pairs_of(uint32_t m) {
  m = (m | (m << 8)) & 0x00FF00FFu;
  m = (m | (m << 4)) & 0x0F0F0F0Fu;
  m = (m | (m << 2)) & 0x33333333u;
  m = (m | (m << 1)) & 0x55555555u;
  return m | (m << 1);
}

// The compress steps of each word (the parallel-prefix method of Warren, Hacker's Delight,
// 7-4): step e moves by 2^e places the codes whose count of left-out samples below them has
// bit e set.  And how many of the (ascending) subset's samples lie below the word.
__global__ void subset_steps_kernel(const int32_t* __restrict__ sidx, int64_t n,
                                    const uint32_t* __restrict__ others, int64_t n_words,
                                    uint4* __restrict__ steps, int32_t* __restrict__ place) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_words) return;
  uint32_t m = ~gather_even(others[j]) & 0xFFFFu, mk = (~m << 1) & 0xFFFFu;
  uint32_t mv[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    uint32_t mp = mk ^ (mk << 1);
    mp ^= mp << 2;
    mp ^= mp << 4;
    mp ^= mp << 8;
    const uint32_t move = mp & m;
    mv[e] = pairs_of(move & 0xFFFFu);
    m = (m ^ move) | (move >> (1 << e));
    mk &= ~mp;
  }
  steps[j] = make_uint4(mv[0], mv[1], mv[2], mv[3]);
  int64_t lo = 0, hi = n;  // first index with sidx >= 16 j
  while (lo < hi) {
    const int64_t mid = (lo + hi) / 2;
    if (sidx[mid] < 16 * j)
      lo = mid + 1;
    else
      hi = mid;
  }
  place[j] = (int32_t)lo;
}

size_t subset_mask_words(int64_t n_fam, bool steps) {
  const size_t k = (size_t)round_up(ceil_div(n_fam, (int64_t)16), (int64_t)4);
  return k + 4 + (steps ? 5 * k : 0);
}

cudaError_t launch_subset_mask(const int32_t* sidx, int64_t n, int64_t n_fam, bool steps,
                               uint32_t* words, SubsetMask* mask, cudaStream_t st) {
  const int64_t n_words = ceil_div(n_fam, (int64_t)16);
  const size_t k = (size_t)round_up(n_words, (int64_t)4);
  unsigned int* flags = words + k;
  mask->others = words;
  mask->repeats = flags;
  mask->unsorted = flags + 1;
  mask->n_fam = n_fam;
  cudaError_t e = cudaMemsetAsync(words, 0xFF, k * 4, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0, 16, st);
  if (e != cudaSuccess) return e;
  subset_mask_kernel<<<(unsigned)ceil_div(n, (int64_t)256), 256, 0, st>>>(sidx, n, words, flags,
                                                                         flags + 1);
  count_launches(1);
  if (steps) {
    uint4* s4 = reinterpret_cast<uint4*>(flags + 4);
    int32_t* place = reinterpret_cast<int32_t*>(s4 + k);
    subset_steps_kernel<<<(unsigned)ceil_div(n_words, (int64_t)128), 128, 0, st>>>(
        sidx, n, words, n_words, s4, place);
    count_launches(1);
    mask->steps = s4;
    mask->place = place;
  }
  return cudaGetLastError();
}

// The packed rows of an ascending subset, kRows rows per block: each thread compresses a word
// of 16 samples at a time (its steps loaded once for the rows) and ORs the kept codes into the
// rows' packed words in shared memory.  Bound by the latency of a word's loads and by the ORs
// (kCompressThreads 256: 0.83 ms where the packed rows leave room for more blocks, 1.27 at 40 %
// kept; 1,024: 1.33).
constexpr int kCompressThreads = 512;
template <int kRows>
__global__ void __launch_bounds__(kCompressThreads)
    bed_compress_kernel(const uint8_t* __restrict__ bed, int64_t bpm,
                        const int64_t* __restrict__ src_rows, int64_t n_rows,
                        const SubsetMask mask, int64_t n, uint32_t* __restrict__ out,
                        int64_t wpr) {
  extern __shared__ __align__(16) uint32_t packed[];  // kRows x stride
  if (*mask.unsorted) return;  // bed_subset_kernel gathers
  const int64_t r0 = (int64_t)blockIdx.x * kRows;
  const int nr = n_rows - r0 < kRows ? (int)(n_rows - r0) : kRows;
  const int n_real = (int)((n + 15) / 16), stride = n_real + 1;
  for (int i = threadIdx.x; i < kRows * stride; i += kCompressThreads) packed[i] = 0u;
  const uint8_t* row[kRows];
  const uint32_t* base[kRows];
  int off[kRows];
  int n_fast = (int)(mask.n_fam / 16);
#pragma unroll
  for (int q = 0; q < kRows; ++q) {
    row[q] = bed + 3 + src_rows[r0 + (q < nr ? q : 0)] * bpm;
    off[q] = (int)(reinterpret_cast<uintptr_t>(row[q]) & 3u);
    base[q] = reinterpret_cast<const uint32_t*>(row[q] - off[q]);
    // words whose two aligned words end inside the row
    const int64_t safe = bpm + off[q] >= 8 ? (bpm + off[q] - 8) / 4 + 1 : 0;
    if (safe < n_fast) n_fast = (int)safe;
  }
  __syncthreads();
  const int n_src = (int)((mask.n_fam + 15) / 16);
#pragma unroll 2
  for (int j = threadIdx.x; j < n_src; j += kCompressThreads) {
    const uint32_t keep = ~__ldg(mask.others + j);
    if (!keep) continue;
    uint32_t w[kRows];
    if (j < n_fast) {
#pragma unroll
      for (int q = 0; q < kRows; ++q)
        w[q] = __funnelshift_r(__ldg(base[q] + j), __ldg(base[q] + j + 1), 8 * off[q]);
    } else {
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        w[q] = 0u;
        for (int b = 0; b < 4; ++b) {
          const int64_t bi = 4 * (int64_t)j + b;
          if (bi < bpm) w[q] |= (uint32_t)row[q][bi] << (8 * b);
        }
      }
    }
    const uint4 mv = __ldg(mask.steps + j);
    const int at = __ldg(mask.place + j), sh = 2 * (at & 15);
    uint32_t* to = packed + (at >> 4);
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      uint32_t x = w[q] & keep, t;
      t = x & mv.x;
      x = (x ^ t) | (t >> 2);
      t = x & mv.y;
      x = (x ^ t) | (t >> 4);
      t = x & mv.z;
      x = (x ^ t) | (t >> 8);
      t = x & mv.w;
      x = (x ^ t) | (t >> 16);
      const uint32_t lo = x << sh, hi = __funnelshift_l(x, 0u, sh);
      if (lo) atomicOr(to + q * stride, lo);
      if (hi) atomicOr(to + q * stride + 1, hi);  // (at most n codes: the spare word stays 0)
    }
  }
  __syncthreads();
  for (int q = 0; q < nr; ++q)
    for (int64_t j = threadIdx.x; j < wpr; j += kCompressThreads) {
      uint32_t w = 0xFFFFFFFFu;  // padding samples: code 11
      if (j < n_real) {
        const int64_t left = n - 16 * j;
        const uint32_t keep = left >= 16 ? 0xFFFFFFFFu : ((1u << (2 * (int)left)) - 1u);
        w = to_device_layout((packed[q * stride + j] & keep) | ~keep);
      }
      out[(r0 + q) * wpr + j] = w;
    }
}

// 39,001 rows of 150,001 samples, compressed against gathered: 0.99 against 1.08 ms with 17 % of
// the samples kept, 1.03 / 1.26 with 25 %, 1.09 / 1.58 with 40 %, 1.27 / 2.17 with 70 %, 1.52 /
// 2.67 with 95 %.  The gather's time goes with the samples kept, the compress's with all.
bool subset_compress_pays(int64_t n, int64_t n_fam) {
  return 6 * n >= n_fam && (n + 31) / 16 * 4 <= kSmemRowMax;
}

cudaError_t launch_bed_gather(const uint8_t* bed, int64_t bpm, const int64_t* src_rows,
                              int64_t n_rows, const int32_t* sample_idx, int64_t n,
                              uint32_t* geno_out, int64_t words_per_row, int64_t* counts,
                              cudaStream_t st, const SubsetMask* mask) {
  if (n_rows <= 0 || (!geno_out && !counts)) return cudaSuccess;
  // Counts alone need no gather: the whole row is read against the subset's mask, as the
  // gather's staging reads it whole (40,000 rows, 60,013 of 150,001 samples: 1.59 ms gathered,
  // 0.41 ms masked).  A small subset of rows too long to stage is gathered from global
  // memory: it touches at most n of the row's sectors.
  const bool masked = sample_idx && mask && counts && !geno_out &&
                      (bpm <= kSmemRowMax || 32 * n >= bpm);
  if (masked) {
    const int64_t n_fam = mask->n_fam;
    const bool shortrow = bpm <= 2048 || n_rows >= 148 * 16;
    const unsigned grid =
        (unsigned)(shortrow ? ceil_div(n_rows, (int64_t)(kThreads / 32)) : n_rows);
    if (shortrow)
      bed_rows_kernel<32, false, true, true><<<grid, kThreads, 0, st>>>(
          bed, bpm, src_rows, n_rows, n_fam, nullptr, 0, counts, *mask);
    else
      bed_rows_kernel<kThreads, false, true, true><<<grid, kThreads, 0, st>>>(
          bed, bpm, src_rows, n_rows, n_fam, nullptr, 0, counts, *mask);
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  const bool compressed =
      sample_idx && mask && mask->steps && geno_out && !counts && subset_compress_pays(n, mask->n_fam);
  if (compressed) {
    const int64_t per_row = ((n + 15) / 16 + 1) * 4;
    const int rows = 4 * per_row <= kSmemHalf ? 4 : (2 * per_row <= kSmemHalf ? 2 : 1);
    auto go = [&](auto kern) -> cudaError_t {
      const size_t smem = (size_t)(per_row * rows);
      if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
      }
      kern<<<(unsigned)ceil_div(n_rows, (int64_t)rows), kCompressThreads, smem, st>>>(
          bed, bpm, src_rows, n_rows, *mask, n, geno_out, words_per_row);
      return cudaGetLastError();
    };
    count_launches(1);
    cudaError_t e = rows == 4   ? go(bed_compress_kernel<4>)
                    : rows == 2 ? go(bed_compress_kernel<2>)
                                : go(bed_compress_kernel<1>);
    if (e != cudaSuccess) return e;
  }
  if (sample_idx) {
    // as many rows per block as half an SM's shared memory holds (two blocks of 16 warps
    // per SM, so that one stages while the other gathers), at most four; a row beyond
    // that, up to kSmemRowMax, has the SM to itself
    const int64_t stride = round_up(bpm + 16, 16);
    const int64_t fit = kSmemHalf / stride;
    const int rows = bpm > kSmemRowMax ? 0 : (fit >= 4 ? 4 : (fit >= 2 ? (int)fit : 1));
    auto go = [&](auto kern, int per) -> cudaError_t {
      const size_t smem = rows ? (size_t)(stride * rows) : 0;
      if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
      }
      kern<<<(unsigned)ceil_div(n_rows, (int64_t)per), kSubsetThreads, smem, st>>>(
          bed, bpm, src_rows, n_rows, sample_idx, n, geno_out, words_per_row, counts,
          masked ? mask->repeats : (compressed ? mask->unsorted : nullptr));
      return cudaGetLastError();
    };
    cudaError_t e = rows == 4   ? go(bed_subset_kernel<4>, 4)
                    : rows == 3 ? go(bed_subset_kernel<3>, 3)
                    : rows == 2 ? go(bed_subset_kernel<2>, 2)
                    : rows == 1 ? go(bed_subset_kernel<1>, 1)
                                : go(bed_subset_kernel<0>, 1);
    count_launches(1);
    return e;
  }
  // identity subset: a warp per row when the rows are short or enough for the chip, else
  // the block (256 threads on a row of 1,250 words leave a fifth of their steps empty and
  // add a block reduction: 100,000 rows of 20,000 samples 319 us, with warps 126 us; few
  // long rows would leave SMs idle; long rows that are also written: 40,000 rows of 200,000
  // samples 0.69 ms with blocks, 0.78 ms with warps)
  const bool shortrow = bpm <= 2048 || (n_rows >= 148 * 16 && (!geno_out || bpm <= 16 * 1024));
  const unsigned grid = (unsigned)(shortrow ? ceil_div(n_rows, (int64_t)(kThreads / 32)) : n_rows);
  auto go = [&](auto kern) {
    kern<<<grid, kThreads, 0, st>>>(bed, bpm, src_rows, n_rows, n, geno_out, words_per_row, counts,
                                    SubsetMask());
  };
  if (shortrow) {
    if (geno_out && counts) go(bed_rows_kernel<32, true, true>);
    else if (geno_out) go(bed_rows_kernel<32, true, false>);
    else go(bed_rows_kernel<32, false, true>);
  } else {
    if (geno_out && counts) go(bed_rows_kernel<kThreads, true, true>);
    else if (geno_out) go(bed_rows_kernel<kThreads, true, false>);
    else go(bed_rows_kernel<kThreads, false, true>);
  }
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace saige
