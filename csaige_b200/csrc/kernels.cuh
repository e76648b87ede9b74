// Launch wrappers of the library's kernels (all sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace saige {

// ---- K1: .bed gather / repack and per-marker counts ------------------------
// For each selected row r: src marker src_rows[r] of the raw .bed (header at
// bed[0]), samples gathered in sample_idx order (NULL = identity).  When
// geno_out != NULL the 2-bit codes are written to row r of geno_out (pitch
// words_per_row 32-bit words; padding samples coded 11, genotype 0).  counts
// (2 per row, may be NULL) receive {alt-allele count, missing count}.
// With the subset's mask, counts alone are formed without the gather.
struct SubsetMask {
  const uint32_t* others = nullptr;       // both bits of every sample outside the subset
  const unsigned int* repeats = nullptr;  // not 0: the subset names a sample twice
  // for subsets in ascending order: per word of 16 samples, how to move its kept codes
  // together (the four steps of a bit compress) and where they go
  const uint4* steps = nullptr;
  const int32_t* place = nullptr;
  const unsigned int* unsorted = nullptr;  // not 0: the subset is not strictly ascending
  int64_t n_fam = 0;
};
cudaError_t launch_bed_gather(const uint8_t* bed, int64_t bytes_per_marker, const int64_t* src_rows,
                              int64_t n_rows, const int32_t* sample_idx, int64_t n,
                              uint32_t* geno_out, int64_t words_per_row, int64_t* counts,
                              cudaStream_t st, const SubsetMask* mask = nullptr);
// The mask of sidx[0 .. n) among n_fam samples, in `words` (subset_mask_words(n_fam, steps) of
// them, 16-byte aligned), with the steps of an ascending subset when asked for.
size_t subset_mask_words(int64_t n_fam, bool steps);
cudaError_t launch_subset_mask(const int32_t* sidx, int64_t n, int64_t n_fam, bool steps,
                               uint32_t* words, SubsetMask* mask, cudaStream_t st);
// Whether launch_bed_gather takes the steps for rows of n out of n_fam samples.
bool subset_compress_pays(int64_t n, int64_t n_fam);

// Alt-allele and missing counts of rows j0 .. j0 + n_rows of the raw .bed for several
// sample subsets at once: subset c is sidx[offs[c] .. offs[c] + ns[c]) (offs[c] a
// multiple of 16); counts[(c m_tot + j) 2 + {0, 1}].  Rows of more than 200 KB are
// refused (cudaErrorInvalidValue).
cudaError_t launch_bed_count_cohorts(const uint8_t* bed, int64_t bytes_per_marker, int64_t j0,
                                     int64_t n_rows, const int32_t* sidx, const int64_t* offs,
                                     const int64_t* ns, int n_cohorts, int64_t m_tot,
                                     long long* counts, cudaStream_t st);

// One cohort's output of launch_bed_gather_cohorts: raw marker j goes to row
// row_of[j * row_stride] of geno (wpr words per row; -1: not kept), its n samples at
// sidx[sidx_off ..] (sidx_off a multiple of 16).  row_of may be host-mapped memory.
struct CohortRows {
  uint32_t* geno;
  const int32_t* row_of;
  int64_t row_stride;
  int64_t wpr;
  int64_t n;
  int64_t sidx_off;
};
// Up to kCohortsPerLaunch cohorts, passed by value in the launch's parameters (no copy
// to queue behind other transfers).
constexpr int kCohortsPerLaunch = 32;
struct CohortSet {
  CohortRows c[kCohortsPerLaunch];
  int n;
};
// Gathers raw rows j0 .. j0 + n_rows into every cohort of the set that keeps them.  Rows
// of more than 200 KB are refused.
cudaError_t launch_bed_gather_cohorts(const uint8_t* bed, int64_t bytes_per_marker, int64_t j0,
                                      int64_t n_rows, const int32_t* sidx, const CohortSet& set,
                                      cudaStream_t st);

// ---- synthetic cohort ------------------------------------------------------
struct CohortDev;
cudaError_t launch_gen_bed(const void* layout, uint8_t* bed, int64_t bytes_per_marker,
                           int64_t m, cudaStream_t st);

// ---- FP32 GRM product (saige-rs arithmetic) --------------------------------
// One to kFp32Cols columns per call (pass B and the finish: to kFp32ColsB); the planes of v32 (n_pad floats, in the kernels' own
// order), u (m_pad) and ypart (n_splits x n_pad) of column c follow those of column c - 1.
constexpr int kFp32Cols = 8;
constexpr int kFp32ColsB = 4;
struct Fp32Cols {
  const double* v[kFp32Cols];
  double* out[kFp32Cols];
};
// u[m] = sum_i z(code_mi) v32[i]       (pass A, f32)
cudaError_t launch_fp32_zt(const uint32_t* geno, int64_t words_per_row, const float4* zlut,
                           int64_t m_pad, const float* v32, int cols, float* u, cudaStream_t st);
// ypart[s][i] = sum_{m in split s} z(code_mi) u[m]   (pass B, f32)
cudaError_t launch_fp32_z(const uint32_t* geno, int64_t words_per_row, const float4* zlut,
                          int64_t m_pad, const float* u, int cols, float* ypart, int n_splits,
                          cudaStream_t st);
int fp32_z_splits(int64_t n_pad, int64_t m_pad);
// out[i] = (double)((sum_s ypart[s][i]) * scale)  (f32 arithmetic)
cudaError_t launch_fp32_finish(const float* ypart, int n_splits, int64_t n_pad, int64_t n,
                               float scale, const Fp32Cols& cols, int n_cols, cudaStream_t st);
// v32 <- (float)v[i] for i < n, 0 for n <= i < n_pad
cudaError_t launch_to_f32(const Fp32Cols& cols, int n_cols, int64_t n, int64_t n_pad, float* v32,
                          cudaStream_t st);

}  // namespace saige
