// MIXED-precision GRM product on the 5th-generation tensor cores.
//
//   pass A  u[m,r] = (1/s_m) sum_i nm_mi (g_mi - 2p_m) v[i,r]
//   pass B  y[i,r] = (1/M)   sum_m nm_mi (g_mi - 2p_m) u[m,r] / s_m
//
// which is OnTheFlyGrm::mat_vec (saige-core/src/glmm/pcg.rs:128-180) with the
// standardisation of OnTheFlyGrm::new (pcg.rs:101-122) folded into the
// product and missing calls centred to zero, without materialising Z.
//
// Arithmetic.  Each column of v (pass A) and of w = u/s, c = 2p w (pass B) is
// quantised to a signed integer q with |q| <= 127*2^16 (24 bits) and split
// into three signed int8 limbs q = 2^16 l2 + 2^8 l1 + l0.  Genotypes
// g in {0,1,2} and the missing indicator are exact int8 operands.
// tcgen05.mma kind::i8 accumulates exact s32 sums per limb in TMEM; limbs,
// scales and the per-marker 2p, 1/s are combined in FP64 in the epilogue:
//   sum_i nm (g - 2p) v = scale (G - 2p (S - Mi)),  G = sum g q, Mi = sum miss q,
//   S = sum q (exact int64), so the only error is the rounding of v to q.
//
// Genotype tiles.  The tensor-core passes read the packed codes as 4 KB tiles
// (128 rows x 128 K entries, 32 bytes per row) stored contiguously in HBM, so
// that each pipeline stage is one sequential 4 KB burst:
//   tiles_m: rows = markers, K = samples  (pass A)
//   tiles_s: rows = samples, K = markers  (pass B, the transpose)
// Both use the device word layout of the row-major copy (entry 4j+i of a
// 16-entry word at bit 16(j>>1) + 2(j&1) + 4i), built once per GRM.
//
// Pipeline (one persistent CTA per SM; the launch's sub-stages of 128 rows x 128 K entries
// are numbered tile by tile and divided evenly over the CTAs, so a CTA walks a run of
// segments, each a tile or a part of one):
//   warp 0      bulk-copies the sub-stages' code tiles and their vector-limb tile(s)
//               (written beforehand in the 128-byte-swizzled K-major layout)
//               into a shared-memory load ring, running ahead over segments;
//   warps 2-17  four groups of four warps take sub-stages in turn; each thread
//               expands its row's 128 codes into 128 int8 genotypes and 128
//               int8 missing flags with byte permutes and stores them straight
//               into a TMEM operand slot (tcgen05.st): the A operand never
//               touches shared memory;
//   warp 1      issues tcgen05.mma kind::i8 with A from TMEM and B (limbs)
//               from shared memory, and commits each sub-stage to mbarriers;
//   warps 2-17  run the epilogue of each segment from the TMEM accumulators: FP64 and
//               the output for a whole tile; the integer sums of a part of a tile meet
//               in global memory, and the CTA that adds the last part finishes the tile.
// Every mbarrier wait is bounded; a wait that runs out sets an error word the
// host reads back (SAIGE_TIMEOUT).
#include <cuda.h>
#include <math.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <vector>

#include "kernels.cuh"
#include "kernels_tc.cuh"
#include "miss_lists.cuh"
#include "tcgen05.cuh"

namespace saige {

namespace {

using namespace tcx;

constexpr int kRows = 128;                    // MMA M: rows of a CTA tile
constexpr int kKt = 128;                      // K entries per pipeline stage
constexpr uint32_t kTileBytes = kRows * kKt / 4;  // 4 KB of 2-bit codes
constexpr int kGroups = 4;                     // unpack groups of four warps
constexpr int kMaxSA = kGroups;               // TMEM operand slots at most
constexpr int kMaxSL = 24;                    // load-ring stages at most
constexpr int kUnpackThreads = 128 * kGroups;
constexpr int kThreads = 64 + kUnpackThreads;  // producer warp, MMA warp, unpack warps
constexpr size_t kSmemBudget = 227 * 1024;
constexpr uint32_t kTmemCols = 512;           // the whole TMEM (one CTA per SM)
constexpr uint32_t kSlotCols = 64;            // per slot: 32 columns of genotypes + 32 of flags
constexpr int kMaxR = 64;                     // right-hand sides per launch (3*64 = 192 <= 256 MMA N)
constexpr double kQ = 127.0 * 65536.0;

// The product's columns among the caller's (passed by value: no copy to wait for).
struct ColMap {
  int c[kMaxR];
};

struct TcArgs {
  int ng;                   // B tile rows (= MMA N), multiple of 16
  int r;                    // right-hand sides in this launch
  int nk;                   // sub-stages over K of a tile
  // work division (TcWork): whole tiles per CTA, then the sub-stages of the tiles left over
  int whole, extra;         // CTA c takes tiles c + i grid, i < whole (+ 1 for c < extra)
  int tail_tile;            // first tile that CTAs share
  int64_t tail_units;       // sub-stages of the shared tiles
  int sub;                  // 128-entry sub-stages per load stage (1, 2 or 4)
  int sl;                   // load-ring depth in load stages (>= 2)
  int sa;                   // TMEM operand slots, one per sub-stage (2 .. kGroups)
  // sums of tiles that several CTAs share: per slot (TcSplit) 2 x r x 128 int64, and the
  // sub-stages added so far; all zero between launches
  unsigned long long* part;
  unsigned int* part_done;
  const uint8_t* tiles;     // this pass's code tiles, tile t at (t*tile_ld + k)*4 KB
  int64_t tile_ld;          // tiles from one output tile's row of tiles to the next (>= nk)
  const uint8_t* img_g;     // nk x ng x 128 bytes
  const uint8_t* img_m;     // pass B: c image (same shape)
  const double* scale_g;    // [r]
  const double* scale_m;    // [r] pass B
  const long long* sum_q;   // [r] pass A: sum q_v; pass B: sum q_c
  const double* two_p;      // [m_pad]
  const double* inv_s;      // [m_pad]
  double* out;              // pass A: u [r][out_ld]; pass B: kp (column col_map[r])
  int64_t out_ld;
  ColMap col_map;           // pass B
  double out_scale;         // pass B: 1/M
  unsigned int* err;
  unsigned long long* trace;  // optional pipeline trace of CTA 0 (SAIGE_TC_TRACE=1)
  long long wait_cycles;    // budget of each pipeline wait (0: give up unless already done)
};

constexpr int kTraceStages = 64;
constexpr int kTraceSlots = 8;

// Records %globaltimer for CTA 0, sub-stage k, event slot e (kTrace builds of the kernel).
template <bool kTrace>
__device__ __forceinline__ void trace_mark(const TcArgs& a, int k, int e) {
  if (kTrace && blockIdx.x == 0 && k < kTraceStages) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    a.trace[k * kTraceSlots + e] = t;
  }
}

// Instruction descriptor: kind::i8, s32 accumulate, signed A and B, both
// K-major, M = 128.
__host__ __device__ constexpr uint32_t i8_idesc(int n) {
  return (2u << 4)                          // c_format = S32
         | (1u << 7)                        // a_format = signed int8
         | (1u << 10)                       // b_format = signed int8
         | ((uint32_t)(n >> 3) << 17)       // N >> 3
         | ((uint32_t)(kRows >> 4) << 24);  // M >> 4
}

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_i8_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z));
}

constexpr int kEpi = 4;  // columns per step of the epilogue (12 limb columns)
constexpr int kUnpackWarps = kUnpackThreads / 32;

// CTA c's share of the shared tiles' sub-stages: [units c / grid, units (c + 1) / grid).
__host__ __device__ __forceinline__ int64_t unit_begin(int64_t units, int c, int grid) {
  return units * c / grid;
}

// One CTA's run of segments: its whole tiles, then its share of the tiles left over.
struct Segments {
  int64_t u, end;
  int i, n_whole, nk, tail_tile;
  int tile, k0, k1;
  __device__ Segments(const TcArgs& a)
      : u(unit_begin(a.tail_units, blockIdx.x, gridDim.x)),
        end(unit_begin(a.tail_units, blockIdx.x + 1, gridDim.x)),
        i(0),
        n_whole(a.whole + ((int)blockIdx.x < a.extra ? 1 : 0)),
        nk(a.nk),
        tail_tile(a.tail_tile) {}
  // the next segment: sub-stages [k0, k1) of `tile`
  __device__ bool next() {
    if (i < n_whole) {
      tile = (int)(blockIdx.x + (unsigned)i * gridDim.x);
      k0 = 0;
      k1 = nk;
      ++i;
      return true;
    }
    if (u >= end) return false;
    const int q = (int)(u / nk);
    tile = tail_tile + q;
    k0 = (int)(u - (int64_t)q * nk);
    const int64_t left = end - u;
    k1 = left < nk - k0 ? k0 + (int)left : nk;
    u += k1 - k0;
    return true;
  }
};

// Slot of a tile that several CTAs share: the first CTA (>= 1) whose share begins inside it,
// less one.
__device__ __forceinline__ int part_slot(const TcArgs& a, int tile) {
  const int64_t first = (int64_t)(tile - a.tail_tile) * a.nk;
  int c = (int)(first * gridDim.x / a.tail_units);
  while (unit_begin(a.tail_units, c, gridDim.x) <= first) ++c;
  return c - 1;
}

// 16 consecutive TMEM columns of this thread's lane <- v[0..15].
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15])
      : "memory");
}

// Codes 00,01,10,11 -> genotype bytes {2,0,1,0} and missing bytes {0,1,0,0}.
constexpr uint32_t kLutG = 0x00010002u;
constexpr uint32_t kLutM = 0x00000100u;

// Shared-memory plan (1024-byte aligned):
//   load ring  sl x [codes sub x 4 KB | B_g sub x ng*128 | B_m sub x ng*128 (pass B)]
//   barriers   FULL[sl] (load stage landed), LDONE[sl] (its MMAs complete),
//              AFULL[kGroups] (a group's sub-stage is in its operand slot: one arrival per
//              warp), ADONE[kGroups] (its MMAs complete), ACCF (a segment's MMAs complete),
//              AFREE (its accumulators read: one arrival per unpack warp), PSUM and PLAST
//              (the sums of a shared tile: added by every warp, its count taken)
//   misc       TMEM address, abort flag, last-part flag
// Every wait between roles is a bounded wait on an mbarrier: a role that gives up raises the
// abort flag and leaves its loop, the others see the flag in their next wait, and nobody
// waits for an arrival that does not come.
// A load stage carries `sub` consecutive 128-entry sub-stages in one
// transaction-counted mbarrier phase (fewer at the end of a segment).
// TMEM: accumulators G at columns [0, ng), Mi at [ng, 2 ng); operand slots of
// 64 columns (one sub-stage) from column a0 = round_up(2 ng, 32).
struct SmemPlan {
  uint32_t base, l_stage, b_bytes, sub, bars;
  __device__ uint32_t L(int s) const { return base + (uint32_t)s * l_stage; }
  __device__ uint32_t CODES(int s, int t) const { return L(s) + (uint32_t)t * kTileBytes; }
  __device__ uint32_t B_g(int s, int t) const {
    return L(s) + sub * kTileBytes + (uint32_t)t * b_bytes;
  }
  __device__ uint32_t B_m(int s, int t) const {
    return L(s) + sub * (kTileBytes + b_bytes) + (uint32_t)t * b_bytes;
  }
  __device__ uint32_t FULL(int s) const { return bars + 8u * s; }
  __device__ uint32_t LDONE(int s) const { return bars + 8u * (kMaxSL + s); }
  __device__ uint32_t AFULL(int g) const { return bars + 8u * (2 * kMaxSL + g); }
  __device__ uint32_t ADONE(int g) const { return bars + 8u * (2 * kMaxSL + kGroups + g); }
  __device__ uint32_t ACCF() const { return bars + 8u * (2 * kMaxSL + 2 * kGroups); }
  __device__ uint32_t AFREE() const { return ACCF() + 8u; }
  __device__ uint32_t PSUM() const { return ACCF() + 16u; }
  __device__ uint32_t PLAST() const { return ACCF() + 24u; }
  __device__ uint32_t MISC() const { return ACCF() + 32u; }
};

__host__ __device__ constexpr uint32_t round1k(uint32_t x) { return (x + 1023u) & ~1023u; }

// bytes of one sub-stage in the load ring
__host__ __device__ constexpr uint32_t plan_sub_bytes(int ng, bool pass_b) {
  return kTileBytes + (uint32_t)ng * kKt * (pass_b ? 2u : 1u);
}

__host__ __device__ constexpr uint32_t plan_l_stage(int ng, bool pass_b, int sub) {
  return round1k((uint32_t)sub * plan_sub_bytes(ng, pass_b));
}

__host__ __device__ constexpr uint32_t tmem_a0(int ng) { return ((uint32_t)(2 * ng) + 31u) & ~31u; }

// Expands one 16-entry code word into 16 genotype bytes (g[0..3]) and 16
// missing-flag bytes (m[0..3]), entries in order.  PRMT reads only the low
// 16 bits of its selector, so each selector is one nibble group.
__device__ __forceinline__ void expand_word(uint32_t w, uint32_t* g, uint32_t* m) {
  const uint32_t lo = w & 0x33333333u;         // entries 0-3 (bits 0-15), 8-11 (bits 16-31)
  const uint32_t hi = (w >> 2) & 0x33333333u;  // entries 4-7, 12-15
  const uint32_t lo2 = lo >> 16, hi2 = hi >> 16;
  g[0] = __byte_perm(kLutG, 0u, lo);
  g[1] = __byte_perm(kLutG, 0u, hi);
  g[2] = __byte_perm(kLutG, 0u, lo2);
  g[3] = __byte_perm(kLutG, 0u, hi2);
  m[0] = __byte_perm(kLutM, 0u, lo);
  m[1] = __byte_perm(kLutM, 0u, hi);
  m[2] = __byte_perm(kLutM, 0u, lo2);
  m[3] = __byte_perm(kLutM, 0u, hi2);
}

// What bounds it.  The tensor pipe needs 64 cycles for an MMA (M = 128, N = 128, K = 32), 512
// per sub-stage of 128 x 128 entries (4 K-steps x genotype and missing accumulators); at 42
// columns and 200,000 x 150,000 both passes run long enough for the chip's power limit to
// lower the SM clock (1.62-1.77 GHz sampled inside the kernel).  Below that, the MMA warp's own
// instructions (see there), and in pass B shared memory: 36 KB of copies, 32 KB of operand
// reads and 4 KB of codes per sub-stage, against 20 + 32 + 4 KB in pass A.
// 37 columns at 50,000 x 100,000, pass A / pass B in us:
//   1222 / 1182  MMAs issued under a branch on the lane number;
//    945 /  956  by an elected lane, two unpack groups, two sub-stages per handoff, a CTA
//                per tile (five and two waves, the last one partly empty);
//    860 /  845  four unpack groups, a persistent CTA per SM, the tiles left over shared;
//    740 /  852  and the next sub-stage's barrier tested between the halves of this one's MMAs.
// (Two MMA warps, one per accumulator: 785 / 962.  Whole tiles started at different K per CTA:
// no change, so the operand tiles' L2 reads do not bound it.)
template <bool kPassB, bool kTrace>
__global__ void __launch_bounds__(kThreads, 1) tc_grm_kernel(TcArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  SmemPlan P;
  P.base = (raw + 1023u) & ~1023u;
  P.b_bytes = (uint32_t)a.ng * kKt;
  P.sub = (uint32_t)a.sub;
  P.l_stage = plan_l_stage(a.ng, kPassB, a.sub);
  P.bars = P.base + (uint32_t)a.sl * P.l_stage;
  uint8_t* gen = smem_raw + (P.base - raw);  // generic pointer of P.base
  auto gptr = [&](uint32_t saddr) { return gen + (saddr - P.base); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gptr(P.MISC()));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gptr(P.MISC() + 8u));
  volatile int* last_part = reinterpret_cast<volatile int*>(gptr(P.MISC() + 12u));

  // warp: uniform over the warp, and known to be
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.sl; ++s) {
      mbar_init(P.FULL(s), 1);
      mbar_init(P.LDONE(s), 1);
    }
    for (int g = 0; g < kGroups; ++g) {
      mbar_init(P.AFULL(g), kUnpackWarps / kGroups);
      mbar_init(P.ADONE(g), 1);
    }
    mbar_init(P.ACCF(), 1);
    mbar_init(P.AFREE(), kUnpackWarps);
    mbar_init(P.PSUM(), kUnpackWarps);
    mbar_init(P.PLAST(), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_g = tmem, tmem_m = tmem + (uint32_t)a.ng;
  const uint32_t tmem_a = tmem + tmem_a0(a.ng);
  Segments seg(a);

  if (warp == 0) {
    // ---------------- producer: code tiles and limb tiles by bulk copy ----------------
    if (lane == 0) {
      int S = 0, J = 0;  // load slot, load stages so far
      uint32_t ph = 0;   // (J / sl) & 1
      bool live = true;
      while (live && seg.next()) {
        const uint8_t* codes = a.tiles + (size_t)seg.tile * a.tile_ld * kTileBytes;
        for (int k0 = seg.k0; k0 < seg.k1; k0 += a.sub) {
          // the slot is free once the MMAs of load stage J - sl completed
          if (J >= a.sl && !mbar_wait_poll(P.LDONE(S), ph ^ 1u, abort_flag, a.err, a.wait_cycles)) {
            live = false;
            break;
          }
          if (J < kTraceStages) trace_mark<kTrace>(a, J, 0);  // load issued
          const uint32_t cnt = (uint32_t)min(a.sub, seg.k1 - k0);
          mbar_expect_tx(P.FULL(S), cnt * (kTileBytes + P.b_bytes * (kPassB ? 2u : 1u)));
          bulk_load(P.CODES(S, 0), codes + (size_t)k0 * kTileBytes, cnt * kTileBytes, P.FULL(S));
          for (uint32_t t = 0; t < cnt; ++t) {  // limb tiles: one copy per sub-stage (<= 24 KB)
            bulk_load(P.B_g(S, t), a.img_g + (size_t)(k0 + t) * P.b_bytes, P.b_bytes, P.FULL(S));
            if (kPassB)
              bulk_load(P.B_m(S, t), a.img_m + (size_t)(k0 + t) * P.b_bytes, P.b_bytes, P.FULL(S));
          }
          ++J;
          if (++S == a.sl) { S = 0; ph ^= 1u; }
        }
      }
      // Before the CTA exits, every issued copy has landed: load stage j completes
      // phase (j / sl) & 1 of FULL(j % sl), and only the last sl issued stages can
      // still be in flight (stage j was issued after stage j - sl was consumed).  On
      // the normal path these phases completed long ago and the waits return at once.
      for (int j = J > a.sl ? J - a.sl : 0; j < J; ++j)
        mbar_wait_drain(P.FULL(j % a.sl), (uint32_t)((j / a.sl) & 1), a.err);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // All lanes wait for each filled operand slot of the unpack groups and an elected one
    // issues the sub-stage's MMAs.  This warp's instructions set the pace wherever they take
    // longer than the 512 cycles of the tensor pipe (measured per sub-stage, 8 MMAs and
    // their commits, with nothing else running, N = 48 / N = 128):
    //   268 / 512 without a wait: elect.sync, in a branch that is otherwise uniform over the
    //     warp, lets the compiler keep descriptors and addresses in uniform registers, which
    //     tcgen05.mma reads (under a branch on the lane number: 47 cycles per MMA);
    //   325 / 512 with one test of the barrier by all lanes, the polling loop out of line;
    //   399 / 579 with the polling loop inline; 489 / 669 with a lane of its own polling and
    //     a vote.
    // Beside the unpack warps, which share its scheduler, they take longer, and the pipe
    // queues only about two MMAs: so the next sub-stage's barrier is tested while half of
    // this one's are still to be issued.
    // Ring positions advance incrementally: no division in the loop.
    const uint32_t idesc = i8_idesc(a.ng);
    int t = 0, s = 0, ab = 0, grp = 0;  // sub-stage within the load stage, load slot, operand
                                        // slot, unpack group
    uint32_t ph_a = 0;                  // (K / kGroups) & 1
    int K = 0, J = 0, n_seg = 0;        // sub-stages, load stages and segments committed so far
    bool live = true, ready = false;    // ready: the sub-stage's operands are known to be in place
    // all lanes: a bounded wait
    auto wait_for = [&](uint32_t bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait_slow(bar, parity, abort_flag, a.err,
                                                    a.wait_cycles)) != 0;
    };
    while (live && seg.next()) {
      // the accumulators of the segment before have been read
      if (n_seg > 0) live = wait_for(P.AFREE(), (uint32_t)(n_seg - 1) & 1u);
      const int n = __shfl_sync(0xffffffffu, seg.k1 - seg.k0, 0);
      for (int k = 0; live && k < n; ++k) {
        if (kTrace && lane == 0) {
          trace_mark<kTrace>(a, K, 6);  // MMA warp reaches the sub-stage
          if (blockIdx.x == 0 && K < kTraceStages)
            a.trace[K * kTraceSlots + 7] = (unsigned long long)clock64();  // SM clock at the same point
        }
        if (!ready) live = wait_for(P.AFULL(grp), ph_a);
        if (!live) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (kTrace && lane == 0) trace_mark<kTrace>(a, K, 4);  // MMA may issue
        const bool stage_end = t == a.sub - 1 || k == n - 1;
        // genotype and missing-flag MMAs alternate (two independent accumulators)
        const uint64_t bg = sw128_desc(P.B_g(s, t));
        const uint64_t bm = kPassB ? sw128_desc(P.B_m(s, t)) : bg;
        const uint32_t ag = tmem_a + (uint32_t)ab * kSlotCols, am = ag + 32u;
        const uint32_t later = k > 0 ? 1u : 0u;
        // K advance of 32 int8: 8 TMEM columns of A, 32 bytes (2 x 16 B) along a B row
        auto issue = [&](int kk, uint32_t acc) {
          mma_i8_ts(tmem_g, ag + 8u * kk, bg + 2u * kk, idesc, acc);
          mma_i8_ts(tmem_m, am + 8u * kk, bm + 2u * kk, idesc, acc);
        };
        if (elect_one()) {
          issue(0, later);
          issue(1, 1u);
        }
        // between the halves, while MMAs are queued: is the next sub-stage in place?
        ready = __all_sync(0xffffffffu, mbar_test_wait(P.AFULL((grp + 1) % kGroups),
                                                       grp == kGroups - 1 ? ph_a ^ 1u : ph_a));
        if (elect_one()) {
          issue(2, 1u);
          issue(3, 1u);
          mma_commit(P.ADONE(grp));
          if (stage_end) mma_commit(P.LDONE(s));
        }
        ++K;
        ++t;
        if (stage_end) {
          t = 0;
          ++J;
          if (++s == a.sl) s = 0;
        }
        if (++ab == a.sa) ab = 0;
        if (++grp == kGroups) { grp = 0; ph_a ^= 1u; }
        if (kTrace && lane == 0) trace_mark<kTrace>(a, K - 1, 5);  // MMAs issued
      }
      if (live) {
        if (elect_one()) mma_commit(P.ACCF());
        ++n_seg;
      }
    }
    if (lane == 0) {
      // Before the CTA can finish, wait (bounded) for the last committed phase of every
      // barrier: all MMAs are complete then, and no commit's arrival — performed in no set
      // order with the others — can land in the shared memory of the SM's next CTA.
      for (int ls = 0; ls < a.sl && ls < J; ++ls) {
        const int j = J - 1 - (J - 1 - ls) % a.sl;
        mbar_wait_drain(P.LDONE(ls), (uint32_t)((j / a.sl) & 1), a.err);
      }
      for (int g = 0; g < kGroups && g < K; ++g) {
        const int k = K - 1 - (K - 1 - g) % kGroups;
        mbar_wait_drain(P.ADONE(g), (uint32_t)((k / kGroups) & 1), a.err);
      }
      if (n_seg > 0) mbar_wait_drain(P.ACCF(), (uint32_t)(n_seg - 1) & 1u, a.err);
    }
    __syncwarp();
  } else {
    // ---------------- unpack (warps 2-17) ----------------
    // Group g takes the sub-stages K = g, g + 4, ... of the CTA's run;
    // a warp may only address its own TMEM lane group (warp % 4), so thread
    // `lane` of warp w expands row 32 (w % 4) + lane.
    const int grp = (warp - 2) >> 2;
    const int lg = warp & 3;
    const int row = lg * 32 + lane;
    const uint32_t lane_off = (uint32_t)(lg * 32) << 16;
    bool live = true;  // false once a wait gave up (the same for the whole warp)
    const int lsub = a.sub >> 1;  // log2 (sub is 1, 2 or 4)
    int K0 = 0, s0 = 0;           // sub-stages before the segment, load slot at its start
    uint32_t ph0 = 0;             // phase parity of FULL(s0)
    uint32_t ph_acc = 0, ph_part = 0;
    while (live && seg.next()) {
      const int n = seg.k1 - seg.k0;
      // this group's sub-stages i = i0, i0 + 4, ... of the segment (4 is a multiple of sub: the
      // place in the load stage stays)
      int i = (grp - K0) & (kGroups - 1), s = s0 + (i >> lsub), ab = (K0 + i) % a.sa;
      const int t = i & (a.sub - 1);
      uint32_t ph_l = ph0;
      while (s >= a.sl) { s -= a.sl; ph_l ^= 1u; }
      for (; i < n; i += kGroups) {
        const int K = K0 + i;
        // The operand slot is free once the MMAs of its previous use (sub-stage K - sa)
        // completed.  Sub-stage k's completion is phase k / 4 of ADONE(k % 4): a barrier
        // per group, not per slot, so that the phase before (sub-stage K - 4 - sa) is the
        // one this group waited for last and the next one (K + 4 - sa) cannot complete before
        // this sub-stage is unpacked — with fewer slots than groups a slot's barrier could
        // pass two phases between two waits of a group, which a parity cannot tell.
        // This wait comes before the one on the codes: a group sees only every
        // fourth sub-stage, so FULL(s) may still be a phase behind — its previous load in
        // flight — and its parity would then already read as this load's.  Once the MMA
        // warp has taken sub-stage K - sa, every load stage up to it was seen complete, and
        // at a segment's start all loads before it (the epilogue waited for their MMAs), which
        // covers load stage J - sl for every accepted ring shape ((sl - 1) sub + 1 >= sa),
        // so the parity below is unambiguous.
        if (K >= a.sa)
          live = mbar_wait_poll(P.ADONE((K - a.sa) % kGroups),
                                (uint32_t)((K - a.sa) / kGroups) & 1u, abort_flag, a.err,
                                a.wait_cycles);
        if (live) live = mbar_wait_poll(P.FULL(s), ph_l, abort_flag, a.err, a.wait_cycles);
        if (live && row == 0) trace_mark<kTrace>(a, K, 1);  // codes landed
        live = __all_sync(0xffffffffu, live);  // warp-uniform: the barrier calls below must agree
        if (!live) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (row == 0) trace_mark<kTrace>(a, K, 2);  // operand slot free
        const uint32_t crow = P.CODES(s, t) + (uint32_t)row * 32u;
        const uint4 c0 = lds128(crow), c1 = lds128(crow + 16u);
        const uint32_t words[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const uint32_t slot = tmem_a + lane_off + (uint32_t)ab * kSlotCols;
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // in halves: fewer registers live
          uint32_t g[16], m[16];
#pragma unroll
          for (int c = 0; c < 4; ++c) expand_word(words[4 * h + c], g + 4 * c, m + 4 * c);
          tmem_st16(slot + 16u * h, g);
          tmem_st16(slot + 32u + 16u * h, m);
        }
        tmem_wait_st();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (row == 0) trace_mark<kTrace>(a, K, 3);  // unpack done
        __syncwarp();
        if (lane == 0) mbar_arrive_local(P.AFULL(grp));
        s += kGroups >> lsub;
        while (s >= a.sl) { s -= a.sl; ph_l ^= 1u; }
        if (a.sa == 3 && ++ab == 3) ab = 0;  // 4 mod sa: 0 for two and four slots
      }
      K0 += n;
      const int s1 = s0 + ((n + a.sub - 1) >> lsub);
      s0 = s1 % a.sl;
      ph0 ^= (uint32_t)(s1 / a.sl) & 1u;
      // ---------------- epilogue of the segment: four warps per TMEM lane group ----------------
      if (live) live = mbar_wait_poll(P.ACCF(), ph_acc, abort_flag, a.err, a.wait_cycles);
      live = __all_sync(0xffffffffu, live);
      if (!live) break;
      ph_acc ^= 1u;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool whole = seg.k0 == 0 && seg.k1 == a.nk;
      const int64_t grow = (int64_t)seg.tile * kRows + row;  // marker (A) or sample (B)
      const double rowa = kPassB ? 0.0 : a.inv_s[grow], rowb = kPassB ? 0.0 : a.two_p[grow];
      const int slot = whole ? 0 : part_slot(a, seg.tile);
      unsigned long long* part = a.part + (size_t)slot * 2 * a.r * kRows + row;
      // the output of column r from the exact integer sums
      auto finish = [&](int r, long long gi, long long mi) {
        const double G = (double)gi, Mi = (double)mi, S = (double)a.sum_q[r];
        if (!kPassB) {
          // u = (1/s) scale (G - 2p (S - Mi)); explicit roundings (no contraction)
          const double tt = __dsub_rn(G, __dmul_rn(rowb, S - Mi));
          a.out[(int64_t)r * a.out_ld + grow] = __dmul_rn(rowa, __dmul_rn(a.scale_g[r], tt));
        } else {
          // y = (1/M) (sw G - sc (S_c - Mc))
          const double y = __dmul_rn(a.out_scale, __dsub_rn(__dmul_rn(a.scale_g[r], G),
                                                            __dmul_rn(a.scale_m[r], S - Mi)));
          a.out[(int64_t)a.col_map.c[r] * a.out_ld + grow] = y;
        }
      };
      auto free_acc = [&]() {  // this warp has read the accumulators
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_local(P.AFREE());
      };
      if (kEpi * grp >= a.r) free_acc();
      for (int r0 = kEpi * grp; r0 < a.r; r0 += kEpi * kGroups) {
        uint32_t g[3 * kEpi], m[3 * kEpi];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int col = 3 * r0 + 4 * j;
          if (col < a.ng) {
            tmem_ld4(tmem_g + lane_off + (uint32_t)col, g + 4 * j);
            tmem_ld4(tmem_m + lane_off + (uint32_t)col, m + 4 * j);
          }
        }
        tmem_wait_ld();
        if (r0 + kEpi * kGroups >= a.r) free_acc();  // the last read
#pragma unroll
        for (int e = 0; e < kEpi; ++e) {
          const int r = r0 + e;
          if (r >= a.r) break;
          // limbs to the exact integers: below 2^53, so exact in FP64 too
          const long long gi = 65536LL * (int)g[3 * e] + 256LL * (int)g[3 * e + 1] + (int)g[3 * e + 2];
          const long long mi = 65536LL * (int)m[3 * e] + 256LL * (int)m[3 * e + 1] + (int)m[3 * e + 2];
          if (whole) {
            finish(r, gi, mi);
          } else {
            atomicAdd(part + (size_t)r * kRows, (unsigned long long)gi);
            atomicAdd(part + (size_t)(a.r + r) * kRows, (unsigned long long)mi);
          }
        }
      }
      if (!whole) {
        // the part that brings a tile's sub-stages to nk finishes it and leaves zeros
        __threadfence();
        __syncwarp();
        if (lane == 0) mbar_arrive_local(P.PSUM());
        if (threadIdx.x == 64) {  // every warp's sums are added: take the count
          live = mbar_wait_poll(P.PSUM(), ph_part, abort_flag, a.err, a.wait_cycles);
          if (live) {
            __threadfence();
            const unsigned int len = (unsigned int)(seg.k1 - seg.k0);
            const bool last = atomicAdd(a.part_done + slot, len) + len == (unsigned int)a.nk;
            if (last) a.part_done[slot] = 0u;
            *last_part = last ? 1 : 0;
            __threadfence();
            mbar_arrive_local(P.PLAST());
          }
        }
        if (live) live = mbar_wait_poll(P.PLAST(), ph_part, abort_flag, a.err, a.wait_cycles);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        ph_part ^= 1u;
        if (*last_part) {
          __threadfence();
          for (int r0 = kEpi * grp; r0 < a.r; r0 += kEpi * kGroups)
#pragma unroll
            for (int e = 0; e < kEpi; ++e) {
              const int r = r0 + e;
              if (r >= a.r) break;
              unsigned long long* pg = part + (size_t)r * kRows;
              unsigned long long* pm = part + (size_t)(a.r + r) * kRows;
              const long long gi = (long long)__ldcg(pg), mi = (long long)__ldcg(pm);
              *pg = 0ull;
              *pm = 0ull;
              finish(r, gi, mi);
            }
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols));
  }
}

// ---------------------------------------------------------------------------
// genotype tiles
// ---------------------------------------------------------------------------
// Bit offset of entry e (0..15) of a 16-entry word in the device word layout.
__device__ __forceinline__ int entry_bit(int e) {
  const int j = e >> 2, i = e & 3;
  return 16 * (j >> 1) + 2 * (j & 1) + 4 * i;
}

// tiles_m[(mt * n_kt + kt)] row r = row-major row mt*128 + r, words kt*8 .. kt*8+7,
// for the marker tiles mt0 + blockIdx.y.
__global__ void __launch_bounds__(256)
    pack_tiles_kernel(const uint32_t* __restrict__ geno, int64_t wpr, int64_t n_kt, int64_t mt0,
                      uint8_t* __restrict__ tiles) {
  const int64_t kt = blockIdx.x, mt = mt0 + blockIdx.y;
  const int r = threadIdx.x >> 1, half = threadIdx.x & 1;
  const uint4 v = *reinterpret_cast<const uint4*>(geno + (mt * kRows + r) * wpr + kt * 8 + half * 4);
  *reinterpret_cast<uint4*>(tiles + (mt * n_kt + kt) * kTileBytes + r * 32 + half * 16) = v;
}

// tiles_s[(st * s_ld + mt)] row r = sample st*128 + r, word j = markers
// mt*128 + 16j .. +15, read from tiles_m[(mt * n_st + st)], for the marker tiles
// mt0 + blockIdx.x.
__global__ void __launch_bounds__(256)
    transpose_tiles_kernel(const uint8_t* __restrict__ tiles_m, int64_t n_st, int64_t s_ld,
                           int64_t mt0, uint8_t* __restrict__ tiles_s) {
  __shared__ __align__(16) uint32_t src[kTileBytes / 4];
  __shared__ __align__(16) uint32_t dst[kTileBytes / 4];
  const int64_t mt = mt0 + blockIdx.x, st = blockIdx.y;
  const uint4* s4 = reinterpret_cast<const uint4*>(tiles_m + (mt * n_st + st) * kTileBytes);
  reinterpret_cast<uint4*>(src)[threadIdx.x] = s4[threadIdx.x];
  __syncthreads();
  // output word (r, j): thread handles r = idx & 127, j = idx >> 7 for idx = t, t+256, ...
  for (int idx = threadIdx.x; idx < kRows * 8; idx += 256) {
    const int r = idx & 127, j = idx >> 7;
    const int sb = entry_bit(r & 15);
    uint32_t w = 0;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const uint32_t sw = src[(16 * j + e) * 8 + (r >> 4)];  // marker row 16j+e, sample word r/16
      w |= ((sw >> sb) & 3u) << entry_bit(e);
    }
    dst[r * 8 + j] = w;
  }
  __syncthreads();
  reinterpret_cast<uint4*>(tiles_s + (st * s_ld + mt) * kTileBytes)[threadIdx.x] =
      reinterpret_cast<const uint4*>(dst)[threadIdx.x];
}

// ---------------------------------------------------------------------------
// quantisation kernels
// ---------------------------------------------------------------------------
// The maxima that scale a product's operands.  Bound by latency, not by their 8 bytes per
// row.  One atomic per block of kAmaxRows rows, a thread's loads independent: with one per
// warp of 256-row blocks a column's atomics queued at one address (31 columns of 9,001
// samples and 22,003 markers: 4.6 -> 2.2 us for v and 13.0 -> 6.4 us for u).
constexpr int kAmaxRows = 2048;

__device__ __forceinline__ void block_amax(unsigned long long* amax, double m, double* sh) {
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) m = fmax(m, sh[k]);
    if (m > 0.0) atomicMax(amax, (unsigned long long)__double_as_longlong(m));
  }
}

// amax over rows [0, len) of column col_map.c[r] (pass A input v)
__global__ void __launch_bounds__(256)
    amax_v_kernel(const double* __restrict__ v, int64_t ld, int64_t len, ColMap col_map,
                  unsigned long long* amax) {
  __shared__ double sh[8];
  const int r = blockIdx.y;
  const double* c = v + (int64_t)col_map.c[r] * ld;
  const int64_t lo = (int64_t)blockIdx.x * kAmaxRows;
  double m = 0.0;
#pragma unroll
  for (int k = 0; k < kAmaxRows / 256; ++k) {
    const int64_t i = lo + k * 256 + threadIdx.x;
    if (i < len) m = fmax(m, fabs(c[i]));
  }
  block_amax(&amax[r], m, sh);
}

// amax of w = u inv_s and c = w 2p over the markers.  Leave-one-chromosome-out: the rows of u
// of the first m markers with excl set become 0 first (excl may be NULL).
__global__ void __launch_bounds__(256)
    amax_wc_kernel(double* __restrict__ u, int64_t ld, int64_t len,
                   const double* __restrict__ inv_s, const double* __restrict__ two_p,
                   const uint8_t* __restrict__ excl, int64_t m, unsigned long long* amax_w,
                   unsigned long long* amax_c) {
  __shared__ double sh[2][8];
  const int r = blockIdx.y;
  double* c = u + (int64_t)r * ld;
  const int64_t lo = (int64_t)blockIdx.x * kAmaxRows;
  double mw = 0.0, mc = 0.0;
#pragma unroll
  for (int k = 0; k < kAmaxRows / 256; ++k) {
    const int64_t i = lo + k * 256 + threadIdx.x;
    if (i >= len) continue;
    double x = c[i];
    if (excl && i < m && excl[i]) c[i] = x = 0.0;
    const double w = x * inv_s[i];
    mw = fmax(mw, fabs(w));
    mc = fmax(mc, fabs(w * two_p[i]));
  }
  block_amax(&amax_w[r], mw, sh[0]);
  block_amax(&amax_c[r], mc, sh[1]);
}

__device__ __forceinline__ double scale_of(unsigned long long bits) {
  const double amax = __longlong_as_double((long long)bits);
  return amax > 0.0 ? amax / kQ : 1.0;
}

// Split q (|q| <= 127*2^16) into signed limbs q = 2^16 l2 + 2^8 l1 + l0.
__device__ __forceinline__ void limbs(long long q, int& l2, int& l1, int& l0) {
  l0 = (int)(signed char)(q & 0xFF);
  const long long q1 = (q - l0) >> 8;
  l1 = (int)(signed char)(q1 & 0xFF);
  l2 = (int)((q1 - l1) >> 8);
}

// Byte offset of entry pos of limb row `row` in a stage image (K-major, 128-byte swizzle).
__device__ __forceinline__ int image_at(int row, int pos) {
  return row * 128 + (((pos >> 4) ^ (row & 7)) << 4) + (pos & 15);
}

// Limb rows 3r, 3r+1, 3r+2 of a stage image: the limbs of four entries from pos (a multiple
// of 4) as one 32-bit store per row.
__device__ __forceinline__ void put_limbs4(uint8_t* stage_img, int r, int pos,
                                           const long long (&q)[4]) {
  uint32_t w[3] = {0u, 0u, 0u};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    int l2, l1, l0;
    limbs(q[e], l2, l1, l0);
    w[0] |= (uint32_t)(l2 & 0xFF) << (8 * e);
    w[1] |= (uint32_t)(l1 & 0xFF) << (8 * e);
    w[2] |= (uint32_t)(l0 & 0xFF) << (8 * e);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
    *reinterpret_cast<uint32_t*>(stage_img + image_at(3 * r + j, pos)) = w[j];
}

// The image's rows past the last column's limbs (up to the MMA's N): zero.
__device__ __forceinline__ void zero_rows4(uint8_t* stage_img, int first, int ng, int pos) {
  for (int row = first; row < ng; ++row)
    *reinterpret_cast<uint32_t*>(stage_img + image_at(row, pos)) = 0u;
}

__device__ __forceinline__ long long block_sum_ll(long long v, long long* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  long long s = 0;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += sh[k];
  return s;
}

// One warp = one 128-entry stage of one column, four entries per lane: quantise v, write
// the limbs into the swizzled stage image, accumulate sum q.  Four entries per lane make the
// swizzled stores whole words instead of bytes; the last column's blocks zero the image's
// rows past its limbs, so that the image needs no memset before.
__global__ void __launch_bounds__(128)
    quant_v_kernel(const double* __restrict__ v, int64_t ld, int64_t len, int64_t n_stages,
                   ColMap col_map, const unsigned long long* __restrict__ amax,
                   double* __restrict__ scale_out, uint8_t* __restrict__ img, int ng,
                   unsigned long long* __restrict__ sum_q) {
  __shared__ long long sh[4];
  const int r = blockIdx.y;
  const int64_t stage = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int pos = 4 * (threadIdx.x & 31);
  const double sc = scale_of(amax[r]);
  long long sum = 0;
  if (stage < n_stages) {
    const double* c = v + (int64_t)col_map.c[r] * ld + stage * 128 + pos;
    long long q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double x = stage * 128 + pos + e < len ? c[e] : 0.0;
      q[e] = __double2ll_rn(x / sc);
      sum += q[e];
    }
    uint8_t* si = img + stage * (int64_t)ng * 128;
    put_limbs4(si, r, pos, q);
    if (r == (int)gridDim.y - 1) zero_rows4(si, 3 * r + 3, ng, pos);
  }
  const long long s = block_sum_ll(sum, sh);
  if (threadIdx.x == 0) {
    atomicAdd(&sum_q[r], (unsigned long long)s);
    if (blockIdx.x == 0) scale_out[r] = sc;
  }
}

__global__ void __launch_bounds__(128)
    quant_wc_kernel(const double* __restrict__ u, int64_t ld, int64_t n_stages,
                    const double* __restrict__ inv_s, const double* __restrict__ two_p,
                    const unsigned long long* __restrict__ amax_w,
                    const unsigned long long* __restrict__ amax_c, double* __restrict__ scale_w,
                    double* __restrict__ scale_c, uint8_t* __restrict__ img_w,
                    uint8_t* __restrict__ img_c, int ng, unsigned long long* __restrict__ sum_c) {
  __shared__ long long sh[4];
  const int r = blockIdx.y;
  const int64_t stage = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int pos = 4 * (threadIdx.x & 31);
  const double sw = scale_of(amax_w[r]), scc = scale_of(amax_c[r]);
  long long sum = 0;
  if (stage < n_stages) {
    const int64_t m = stage * 128 + pos;
    long long qw[4], qc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double w = u[(int64_t)r * ld + m + e] * inv_s[m + e];
      const double c = w * two_p[m + e];
      qw[e] = __double2ll_rn(w / sw);
      qc[e] = __double2ll_rn(c / scc);
      sum += qc[e];
    }
    uint8_t* siw = img_w + stage * (int64_t)ng * 128;
    uint8_t* sic = img_c + stage * (int64_t)ng * 128;
    put_limbs4(siw, r, pos, qw);
    put_limbs4(sic, r, pos, qc);
    if (r == (int)gridDim.y - 1) {
      zero_rows4(siw, 3 * r + 3, ng, pos);
      zero_rows4(sic, 3 * r + 3, ng, pos);
    }
  }
  const long long s = block_sum_ll(sum, sh);
  if (threadIdx.x == 0) {
    atomicAdd(&sum_c[r], (unsigned long long)s);
    if (blockIdx.x == 0) {
      scale_w[r] = sw;
      scale_c[r] = scc;
    }
  }
}

// ---------------------------------------------------------------------------
// Single-column products.  With one column the tcgen05 passes are bound by their fixed
// per-stage cost (eight MMAs and the unpack of a 4 KB code tile for three limb columns), so
// one column costs nearly what 42 do.  These kernels form the same exact integer sums and
// apply the same FP64 epilogue, so their results are bit-identical to the block path's.
// With the missing-call lists of the handle (miss_lists.cuh) the flag sums give way to int64
// sums over the missing calls, for the same integers.
//
// What bounds it: the unpack (four masks and four byte permutes per 16 entries, and four
// more for the flags), then HBM (7.5 GB of codes at 200,000 x 150,000: 1.15 ms per pass).
// The unpacked bytes stay in registers: they are the A fragments of mma.m16n8k32 over the
// three limb columns of q (one instruction for 16 x 32 entries), which a tcgen05.mma would
// want stored to TMEM or shared memory first.  Formed with dp4a (three per four entries and
// accumulator) the sums took 2.7 and 3.1 ms per pass at 200,000 x 148,979; now 1.83 and 1.80
// (1.31 without the flags).
// ---------------------------------------------------------------------------
// prmt tables of the NEGATED genotype (codes 00, 01, 10, 11 -> -2, 0, -1, 0) and of
// the missing flag (01 -> 1).  A selector nibble holds the code either in its bits
// 0-1 (value c: byte c of x) or in its bits 2-3 (value 4c: byte 0 or byte 4 (y),
// sign-replicated when the code's high bit is set — 10 gives sign(x.byte0), 11
// sign(y.byte0)); both tables give the right byte in both positions, so the
// selectors need masks but no shifts.
constexpr uint32_t kNegGenoX = 0x00FF00FEu, kNegGenoY = 0u;
constexpr uint32_t kMissX = 0x00000100u, kMissY = 0x00000001u;
constexpr int kSrRowsA = 64;     // pass A: markers per block
constexpr int kSrRowsB = 256;    // pass B: samples per block
constexpr int kSrChunkA = 4096;  // pass A: samples per chunk of the missing-call lists
constexpr int kSrChunkB = 1024;  // pass B: markers per chunk
// error word bit of a one-column product: a missing-call list entry out of range (the
// entry is skipped; timeouts of the tensor-core pipeline set other bits)
constexpr unsigned int kSrListErr = 1u << 30;
// Missing-call entries of a segment staged in shared memory (2,621 on average at 1 % missing,
// in both passes); what a segment has beyond them is read from global memory.
constexpr int kSrPiece = 4096;
// dynamic shared memory with the lists: two chunks' values and entries, and two counters
// per row
constexpr size_t sr_list_smem(int chunk, int rows) {
  return 2 * 4 * (size_t)(chunk + kSrPiece + rows);
}
static_assert(kSamplePad % 256 == 0, "pass B of one column takes sample tiles in pairs");

__device__ __forceinline__ uint32_t prmt(uint32_t x, uint32_t y, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(y), "r"(sel));
  return d;
}

// The four 4-entry groups of a packed word (device layout: entry 4j+i at bit
// 16(j>>1) + 2(j&1) + 4i; group g = entries 4g..4g+3) as four bytes each of -g and
// of the missing flag.
__device__ __forceinline__ void sr_expand(uint32_t w, int neg_g[4], int miss[4]) {
  const uint32_t hi = w >> 16;
  const uint32_t sel[4] = {w & 0x3333u, w & 0xCCCCu, hi & 0x3333u, hi & 0xCCCCu};
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    neg_g[g] = (int)prmt(kNegGenoX, kNegGenoY, sel[g]);
    miss[g] = (int)prmt(kMissX, kMissY, sel[g]);
  }
}

// Asynchronous copies global -> shared (cp.async) and the wait for all of this thread's
// committed groups but the latest kLeft.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int kLeft>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// The missing sums of a block's kRows rows over its segments of the lists: chunk c has the
// entries ent[seg[c] .. seg[c + 1]), ascending, each (row in block) << bits | (position in
// chunk), and adds q[c kChunk + position] to the row's sum.  Chunks are staged one ahead of
// the dense steps; 256 threads.
template <int kChunk, int kRows_>
struct SrList {
  const uint32_t* __restrict__ ent;
  const int64_t* __restrict__ seg;
  const int32_t* __restrict__ q;
  int64_t len;  // values (a multiple of 128)
  int bits;
  unsigned int* err;
  uint32_t* smem;
  long long sum = 0;  // thread t < kRows_: the sum of row t

  __device__ uint32_t* piece(int64_t c) const { return smem + (c & 1) * kSrPiece; }
  __device__ int32_t* values(int64_t c) const {
    return reinterpret_cast<int32_t*>(smem + 2 * kSrPiece) + (c & 1) * kChunk;
  }
  __device__ int* counters() const {
    return reinterpret_cast<int*>(smem + 2 * (kSrPiece + kChunk));
  }
  __device__ int positions(int64_t c) const {
    return (int)(len - c * kChunk < kChunk ? len - c * kChunk : kChunk);
  }
  // before the first add (a barrier in between)
  __device__ void init() const {
    for (int i = threadIdx.x; i < 2 * kRows_; i += 256) counters()[i] = 0;
  }
  __device__ void stage(int64_t c) const {
    const int n = positions(c);
    int32_t* v = values(c);
    for (int i = threadIdx.x; 4 * i < n; i += 256) cp_async16(v + 4 * i, q + c * kChunk + 4 * i);
    const int64_t e0 = __ldg(seg + c), left = __ldg(seg + c + 1) - e0;
    const int k = (int)(left < kSrPiece ? left : kSrPiece);
    uint32_t* e = piece(c);
    for (int i = threadIdx.x; i < k; i += 256) cp_async4(e + i, ent + e0 + i);
  }
  // k <= kSrPiece consecutive entries.  A thread takes a contiguous slice (of odd length:
  // no bank conflicts), whose entries mostly share a row, and adds each run of one row with
  // two 32-bit atomics: at most 17 values of 24 bits, split at bit 12, so that the counters
  // of one chunk stay in range.  An entry out of range sets kSrListErr and is skipped.
  __device__ void add_piece(const uint32_t* e, int k, const int32_t* v, int n) const {
    const int slice = ((k + 255) >> 8) | 1;
    const int lo = threadIdx.x * slice, hi = lo + slice < k ? lo + slice : k;
    const uint32_t pmask = (1u << bits) - 1u;
    int* cnt = counters();
    int row = -1, acc = 0;
    for (int i = lo; i < hi; i += 4) {
      uint32_t x[4];
      int val[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = i + j < hi ? e[i + j] : 0xFFFFFFFFu;
#pragma unroll
      for (int j = 0; j < 4; ++j) val[j] = (int)(x[j] & pmask) < n ? v[x[j] & pmask] : 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i + j >= hi) break;
        const uint32_t g = x[j] >> bits;
        if (g >= (uint32_t)kRows_ || (int)(x[j] & pmask) >= n) {
          report_error(err, kSrListErr);
          continue;
        }
        if ((int)g != row) {
          if (row >= 0) {
            atomicAdd(&cnt[row], acc >> 12);
            atomicAdd(&cnt[kRows_ + row], acc & 4095);
          }
          row = (int)g;
          acc = 0;
        }
        acc += val[j];
      }
    }
    if (row >= 0) {
      atomicAdd(&cnt[row], acc >> 12);
      atomicAdd(&cnt[kRows_ + row], acc & 4095);
    }
  }
  // chunk c, staged and waited for; a barrier before and after it
  __device__ void add(int64_t c) {
    const int64_t e0 = __ldg(seg + c), left = __ldg(seg + c + 1) - e0;
    const int n = positions(c);
    add_piece(piece(c), (int)(left < kSrPiece ? left : kSrPiece), values(c), n);
    for (int64_t done = kSrPiece; done < left; done += kSrPiece)
      add_piece(ent + e0 + done, (int)(left - done < kSrPiece ? left - done : kSrPiece), values(c),
                n);
    __syncthreads();
    int* cnt = counters();
    if (threadIdx.x < kRows_) {
      sum += 4096LL * cnt[threadIdx.x] + cnt[kRows_ + threadIdx.x];
      cnt[threadIdx.x] = 0;
      cnt[kRows_ + threadIdx.x] = 0;
    }
  }
};

// The same groups as bytes of -g only (the missing sums come from the lists).
__device__ __forceinline__ void sr_expand_g(uint32_t w, int neg_g[4]) {
  const uint32_t hi = w >> 16;
  const uint32_t sel[4] = {w & 0x3333u, w & 0xCCCCu, hi & 0x3333u, hi & 0xCCCCu};
#pragma unroll
  for (int g = 0; g < 4; ++g) neg_g[g] = (int)prmt(kNegGenoX, kNegGenoY, sel[g]);
}

// d += a b: a 16 x 32 int8 (row-major fragment), b 32 x 8 int8 (column-major), d int32.
__device__ __forceinline__ void mma_s8(int (&d)[4], int a0, int a1, int a2, int a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A warp's share of one step: kSrTiles row tiles of 16 rows of one 4 KB code tile (128 rows
// of 32 bytes) against the limb planes.  Lane (g = lane / 4, t = lane % 4) holds words 2t
// and 2t + 1 of rows g and g + 8 of each row tile, and of plane g (the last plane from there
// on: columns nobody reads) the 32 limbs of these words' entries.  The fragments' K order is
// then a permutation of the tile's entries, the same for both operands.
constexpr int kSrTiles = 4;
constexpr int kSrWarpRows = 16 * kSrTiles;
struct SrStep {
  uint2 a[kSrTiles][2];
  uint4 b[2];
};

__device__ __forceinline__ void sr_load(SrStep& s, const uint8_t* __restrict__ rows,
                                        const int8_t* __restrict__ plane) {
#pragma unroll
  for (int k = 0; k < kSrTiles; ++k)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      s.a[k][h] = __ldg(reinterpret_cast<const uint2*>(rows + (16 * k + 8 * h) * 32));
  s.b[0] = __ldg(reinterpret_cast<const uint4*>(plane));
  s.b[1] = __ldg(reinterpret_cast<const uint4*>(plane) + 1);
}

// The step's sums: dg with the bytes of -g, dm (kMiss) with the missing flags.
template <bool kMiss>
__device__ __forceinline__ void sr_step(const SrStep& s, int (&dg)[kSrTiles][4],
                                        int (&dm)[kSrTiles][4]) {
  const uint32_t b[2][4] = {{s.b[0].x, s.b[0].y, s.b[0].z, s.b[0].w},
                            {s.b[1].x, s.b[1].y, s.b[1].z, s.b[1].w}};
#pragma unroll
  for (int k = 0; k < kSrTiles; ++k)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t w0 = i ? s.a[k][0].y : s.a[k][0].x, w1 = i ? s.a[k][1].y : s.a[k][1].x;
      int g0[4], g1[4];
      if constexpr (kMiss) {
        int m0[4], m1[4];
        sr_expand(w0, g0, m0);
        sr_expand(w1, g1, m1);
        mma_s8(dm[k], m0[0], m1[0], m0[1], m1[1], b[i][0], b[i][1]);
        mma_s8(dm[k], m0[2], m1[2], m0[3], m1[3], b[i][2], b[i][3]);
      } else {
        sr_expand_g(w0, g0);
        sr_expand_g(w1, g1);
      }
      mma_s8(dg[k], g0[0], g1[0], g0[1], g1[1], b[i][0], b[i][1]);
      mma_s8(dg[k], g0[2], g1[2], g0[3], g1[3], b[i][2], b[i][3]);
    }
}

// Adds a warp's sums to red[row][column]: columns c0 .. c0 + 2 of d to columns at .. at + 2.
__device__ __forceinline__ void sr_add(int (*red)[6], int row0, const int (&d)[kSrTiles][4],
                                       int c0, int at) {
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
  for (int k = 0; k < kSrTiles; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = row0 + 16 * k + 8 * (e >> 1) + g, c = 2 * t + (e & 1) - c0;
      if (c >= 0 && c < 3) atomicAdd(&red[row][at + c], d[k][e]);
    }
}

// q = rint(x / scale) as in quant_v_kernel, into three int8 planes (l2, l1, l0) of
// length n_pad (zero past len) and, when q32 is given, as int32 (|q| <= 127 * 2^16); and
// sum q.
__global__ void __launch_bounds__(256)
    sr_quant_v_kernel(const double* __restrict__ v, int64_t len, int64_t n_pad,
                      const unsigned long long* __restrict__ amax, double* __restrict__ scale_out,
                      int8_t* __restrict__ planes, int32_t* __restrict__ q32,
                      unsigned long long* __restrict__ sum_q) {
  __shared__ long long sh[8];
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const double sc = scale_of(amax[0]);
  long long q = 0;
  if (i < n_pad) {
    const double x = i < len ? v[i] : 0.0;
    q = __double2ll_rn(x / sc);
    int l2, l1, l0;
    limbs(q, l2, l1, l0);
    planes[i] = (int8_t)l2;
    planes[n_pad + i] = (int8_t)l1;
    planes[2 * n_pad + i] = (int8_t)l0;
    if (q32) q32[i] = (int32_t)q;
  }
  long long t = q;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long s = 0;
    for (int k = 0; k < 8; ++k) s += sh[k];
    atomicAdd(sum_q, (unsigned long long)s);
    if (blockIdx.x == 0) scale_out[0] = sc;
  }
}

// w = u inv_s, c = w 2p quantised as in quant_wc_kernel into planes (w: l2 l1 l0,
// c: l2 l1 l0; length m_pad each) and, when qc32 is given, qc as int32 (|qc| <= 127 *
// 2^16); and sum qc.
__global__ void __launch_bounds__(256)
    sr_quant_wc_kernel(const double* __restrict__ u, int64_t m_pad,
                       const double* __restrict__ inv_s, const double* __restrict__ two_p,
                       const unsigned long long* __restrict__ amax_w,
                       const unsigned long long* __restrict__ amax_c, double* __restrict__ scale_w,
                       double* __restrict__ scale_c, int8_t* __restrict__ planes,
                       int32_t* __restrict__ qc32, unsigned long long* __restrict__ sum_c) {
  __shared__ long long sh[8];
  const int64_t m = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const double sw = scale_of(amax_w[0]), scc = scale_of(amax_c[0]);
  long long qc = 0;
  if (m < m_pad) {
    const double w = u[m] * inv_s[m];
    const double c = w * two_p[m];
    const long long qw = __double2ll_rn(w / sw);
    qc = __double2ll_rn(c / scc);
    int l2, l1, l0;
    limbs(qw, l2, l1, l0);
    planes[m] = (int8_t)l2;
    planes[m_pad + m] = (int8_t)l1;
    planes[2 * m_pad + m] = (int8_t)l0;
    limbs(qc, l2, l1, l0);
    planes[3 * m_pad + m] = (int8_t)l2;
    planes[4 * m_pad + m] = (int8_t)l1;
    planes[5 * m_pad + m] = (int8_t)l0;
    if (qc32) qc32[m] = (int32_t)qc;
  }
  long long t = qc;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long s = 0;
    for (int k = 0; k < 8; ++k) s += sh[k];
    atomicAdd(sum_c, (unsigned long long)s);
    if (blockIdx.x == 0) {
      scale_w[0] = sw;
      scale_c[0] = scc;
    }
  }
}

// How a one-column pass divides the columns of its code tiles: `tiles` per block, `blocks`
// blocks per row block, chosen for the shortest sum of waves x (tiles + ends), plus `meet` where
// partial sums meet; ends is what a block's first loads and last sums cost, in tiles.  A cohort's
// row blocks alone neither fill the SMs (n = 9,001: 36 in pass B) nor come in whole waves.
// `resident`, blocks that an SM takes in the time of one: in pass A two take as long as one after
// the other, since the eight warps of one block keep the integer pipe busy; in pass B, where a
// warp has every second column tile, two take less.  Fitted to every division of 30 sizes from
// 1,000 x 108 to 200,000 x 19,022: within 0.4 % (A, 3 % at most) and 0.9 % (B, 7.5 % at most) of the
// best division on average, against 2.5 % and 3.8 % (31 % and 68 % at most) with waves of two blocks per
// SM in both passes and nothing for the meeting.  us undivided / that rule / this one:
//                        pass A              pass B
//   100,000 x 49,000   352 / 326 / 327     343 / 309 / 309
//    20,000 x 48,995  77.3 / 77.4 / 77.4   122 / 72.3 / 70.5
//     9,001 x 21,010  20.4 / 20.6 / 20.6  53.9 / 18.3 / 18.5
//     5,000 x  7,053   6.1 /  8.3 /  6.3  20.0 /  7.5 /  7.5
//    30,000 x  2,138  21.4 / 10.2 / 10.1   8.3 / 10.8 /  8.4
//     3,000 x    750   4.6 /  5.6 /  4.7   4.5 /  5.1 /  4.6
//     2,000 x  4,081   4.0 /  4.0 /  4.0  12.4 /  5.9 /  5.9
struct SrSplit {
  int64_t tiles;
  unsigned blocks;
};

struct SrCost {
  int resident;
  int64_t ends, ends_divided, meet;
};
constexpr SrCost kSrCostA{1, 2, 10, 16}, kSrCostB{2, 4, 4, 8};

SrSplit sr_split(int64_t row_blocks, int64_t n_kt, int sms, const SrCost& cost) {
  const int64_t slots = (int64_t)cost.resident * sms;
  SrSplit best{n_kt, 1};
  int64_t least = ceil_div(row_blocks, slots) * (n_kt + cost.ends);
  for (int64_t b = 2; b <= std::min<int64_t>(n_kt, 64); ++b) {
    const int64_t tiles = ceil_div(n_kt, b), blocks = ceil_div(n_kt, tiles);
    const int64_t c =
        ceil_div(row_blocks * blocks, slots) * (tiles + cost.ends_divided) + cost.meet;
    if (c < least) {
      least = c;
      best = SrSplit{tiles, (unsigned)blocks};
    }
  }
  return best;
}

struct SrArgs {
  const uint8_t* tiles;   // A: tiles_m; B: tiles_s
  int64_t ld;             // tiles from one row of tiles to the next
  int64_t n_kt;           // column tiles
  const int8_t* planes;   // A: three limb planes of v; B: of w, then of c
  SrSplit split;
  // with the missing-call lists
  const int32_t* q32;     // A: the quantised v; B: c
  const uint32_t* ent;
  const int64_t* seg;
  int64_t nch;
  int bits;
  unsigned int* err;
  // per row, and tickets per row block (when a pass is divided): zero between launches
  unsigned long long *sums_g, *sums_m;
  unsigned int* tickets;
  const unsigned long long* sum_q;  // A: sum q_v; B: sum q_c
  const double *scale_g, *scale_m;  // A: scale of v (scale_m unused); B: of w and of c
  const double *two_p, *inv_s;      // A
  double out_scale;                 // B: 1 / M
  double* out;                      // A: u; B: the product's column
};

// One pass of a one-column product: block = kSrRowsA markers (pass A) or kSrRowsB samples
// (pass B; two tiles) x a range of column tiles.  A warp has 64 rows; the warps of the same
// rows take the column tiles in turn, the next step's loads in flight, and their sums meet in
// shared memory.  Without kLists the flag sums are a second set of accumulators over the same
// limbs; in pass B, whose flags go with c, the planes of w and of c are the six columns of one
// B fragment: the genotype sums are its first three, the flag sums its last three.  With
// kLists the missing sums come from the handle's lists, a chunk falling to the block that has
// its first tile: the same integers the flags give.
//
// The sums are integers, so the partial sums of the blocks of one row block meet in sums_g /
// sums_m (int64 per row, atomics) in any order with the same result; the block that takes the
// last ticket runs the epilogue and leaves the sums and the ticket at zero for the next pass.
template <bool kPassB, bool kLists>
__global__ void __launch_bounds__(256, 2) sr_pass_kernel(SrArgs a) {
  constexpr int kRowsBlk = kPassB ? kSrRowsB : kSrRowsA;
  constexpr int kRowGroups = kRowsBlk / kSrWarpRows, kColGroups = 8 / kRowGroups;
  constexpr int kChunk = kPassB ? kSrChunkB : kSrChunkA;
  constexpr int64_t kChunkTiles = kChunk / kKt;
  extern __shared__ uint4 sr_dyn[];
  __shared__ int red[kRowsBlk][6];
  const int r = threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = r; i < kRowsBlk * 6; i += 256) (&red[0][0])[i] = 0;
  const int64_t t0 = (int64_t)blockIdx.y * a.split.tiles;
  const int64_t t1 = min(t0 + a.split.tiles, a.n_kt), k_len = a.n_kt * kKt;
  const int64_t c0 = (t0 + kChunkTiles - 1) / kChunkTiles, c1 = (t1 + kChunkTiles - 1) / kChunkTiles;
  SrList<kChunk, kRowsBlk> list{a.ent, a.seg + (int64_t)blockIdx.x * a.nch, a.q32, k_len, a.bits,
                                a.err, reinterpret_cast<uint32_t*>(sr_dyn)};
  if constexpr (kLists) {
    list.init();
    if (c0 < c1) list.stage(c0);
    cp_async_commit();
  }
  const int row0 = (warp % kRowGroups) * kSrWarpRows;
  const int64_t grow = (int64_t)blockIdx.x * kRowsBlk + row0;
  const uint8_t* rows = a.tiles + grow / kRows * a.ld * kTileBytes +
                        (grow % kRows + (lane >> 2)) * 32 + (lane & 3) * 8;
  const int8_t* plane = a.planes + min(lane >> 2, kPassB && !kLists ? 5 : 2) * k_len +
                        (lane & 3) * 32;
  int dg[kSrTiles][4] = {}, dm[kSrTiles][4] = {};
  SrStep cur, next;
  int64_t kt = t0 + warp / kRowGroups;
  if (kt < t1) sr_load(cur, rows + kt * kTileBytes, plane + kt * kKt);
  auto dense = [&](int64_t end) {
    for (; kt < end; kt += kColGroups) {
      const int64_t to = kt + kColGroups;
      if (to < t1) sr_load(next, rows + to * kTileBytes, plane + to * kKt);
      sr_step<!kLists>(cur, dg, dm);
      cur = next;
    }
  };
  if constexpr (kLists) {
    for (int64_t c = c0; c < c1; ++c) {
      if (c + 1 < c1) list.stage(c + 1);
      cp_async_commit();
      dense(min(t1, (c + 1) * kChunkTiles));
      cp_async_wait<1>();
      __syncthreads();
      list.add(c);
    }
  }
  dense(t1);
  __syncthreads();  // red is zero
  sr_add(red, row0, dg, 0, 0);
  if constexpr (!kLists) sr_add(red, row0, dm, kPassB ? 3 : 0, 3);
  __syncthreads();
  // this block's integer sums of row r: G (formed with -g) and Mi
  const int64_t i = (int64_t)blockIdx.x * kRowsBlk + r;
  const bool mine = r < kRowsBlk;
  long long g = 0, mi = 0;
  if (mine) {
    const int* d = red[r];
    g = 65536LL * d[0] + 256LL * d[1] + (long long)d[2];
    if constexpr (kLists)
      mi = list.sum;
    else
      mi = 65536LL * d[3] + 256LL * d[4] + (long long)d[5];
  }
  if (gridDim.y > 1) {
    __shared__ int last_s;
    if (mine) {
      atomicAdd(&a.sums_g[i], (unsigned long long)g);
      atomicAdd(&a.sums_m[i], (unsigned long long)mi);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const bool last = atomicAdd(&a.tickets[blockIdx.x], 1u) == gridDim.y - 1;
      if (last) a.tickets[blockIdx.x] = 0u;
      last_s = last ? 1 : 0;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    if (mine) {
      g = (long long)__ldcg(&a.sums_g[i]);
      mi = (long long)__ldcg(&a.sums_m[i]);
      a.sums_g[i] = 0ull;
      a.sums_m[i] = 0ull;
    }
  }
  if (!mine) return;
  // both integers are below 2^53: exact in FP64, as the limb sums of the block path's
  // epilogue are
  const double S = (double)(long long)a.sum_q[0];
  const double G = -(double)g, Mi = (double)mi;
  if constexpr (kPassB) {
    a.out[i] = __dmul_rn(a.out_scale, __dsub_rn(__dmul_rn(a.scale_g[0], G),
                                                __dmul_rn(a.scale_m[0], S - Mi)));
  } else {
    const double tt = __dsub_rn(G, __dmul_rn(a.two_p[i], S - Mi));
    a.out[i] = __dmul_rn(a.inv_s[i], __dmul_rn(a.scale_g[0], tt));
  }
}

size_t tc_fixed_bytes() { return 1024 + 8 * (2 * kMaxSL + 2 * kGroups + 4) + 16; }

struct Rings {
  int sub, sl, sa;
};

// Operand slots that a ring of sl load stages of sub sub-stages accepts: at most
// (sl - 1) sub + 1, so that the slot-reuse wait of an unpack group implies its load slot's
// previous load landed; at most what the accumulators leave of the TMEM.
int slots_for_ring(int ng, int sl, int sub) {
  const int room = std::min<int>(kMaxSA, (int)((kTmemCols - tmem_a0(ng)) / kSlotCols));
  return std::min(room, (sl - 1) * sub + 1);
}

Rings ring_of(int ng, bool pass_b, int sub) {
  const size_t room = kSmemBudget - tc_fixed_bytes();
  Rings g;
  g.sub = sub;
  g.sl = (int)std::min<size_t>(kMaxSL, room / plan_l_stage(ng, pass_b, sub));
  g.sa = slots_for_ring(ng, g.sl, sub);
  return g;
}

// Ring shape of a launch: the most sub-stages per load stage (a copy's fixed cost is shared)
// that leave a ring of at least three load stages; as many load stages as fit; as many
// operand slots as the accumulators leave.
Rings tc_rings(int ng, bool pass_b) {
  for (int sub : {4, 2}) {
    const Rings g = ring_of(ng, pass_b, sub);
    if (g.sl >= 3) return g;
  }
  return ring_of(ng, pass_b, 1);
}

// Division of a launch's tiles over CTAs (one per SM).  Full waves of whole tiles first; the
// tiles left over, fewer than CTAs, are shared out by sub-stages when that saves at least
// kMinSaved of them per CTA, else one CTA takes each.  A part of a tile costs its atomics and the
// last part's second pass (a few us together).
struct TcWork {
  int grid, whole, extra, tail_tile;
  int64_t tail_units;
};
constexpr int64_t kMinSaved = 24;

TcWork tc_work(int64_t tiles, int64_t nk, int sms, bool share_tiles) {
  TcWork w;
  w.grid = sms;
  w.whole = (int)(tiles / sms);
  w.tail_tile = w.whole * sms;
  const int64_t rest = tiles - w.tail_tile, share = ceil_div(rest * nk, (int64_t)sms);
  w.extra = 0;
  w.tail_units = 0;
  if (share_tiles && rest > 0 && nk - share >= kMinSaved) {
    w.tail_units = rest * nk;
  } else {
    w.extra = (int)rest;
    if (w.whole == 0) w.grid = (int)rest;
  }
  return w;
}

}  // namespace

struct TcPlan {
  DevBuf tiles_m, tiles_s, img_a, img_w, img_c, u, scal, trace;
  DevBuf part;  // counts and sums of the tiles that CTAs share: zero between launches
  int sms = 0;
  int64_t s_ld = 0;  // tiles_s: marker tiles per sample tile (>= m_pad / 128)
  bool tracing = false;
  MissLists miss;  // one-column products: the missing-call lists
  DevBuf sr_q32;   // with them: the quantised v (n_pad) and c (m_pad) as int32
  DevBuf sr_sums;  // the divided passes' sums and tickets: zero between launches
};

// Bytes of the counts of the tiles that CTAs share.
static size_t part_counts(const TcPlan* p) { return (size_t)round_up((int64_t)p->sms * 4, 256); }

// When a handle lists its missing calls.  The lists take about two products' time to build (four
// passes over the codes) and 8 bytes per missing call, and the products with them are not the
// faster ones.  us per pass, A + B, with the flags / with the lists of that many missing calls:
//                        flags          0.1 %          1 %
//   200,000 x 148,988  1831 + 1802   2157 + 2111   2634 + 2672
//    50,000 x  98,979   325 +  312    385 +  367
//     9,001 x  21,010  20.7 + 18.5   25.9 + 20.9   32.9 + 25.1
//     3,000 x   3,105   4.7 +  5.9    5.1 +  6.2
//     3,000 x     750   4.7 +  4.6    5.2 +  4.9    6.0 +  6.0
// (with no call missing at all 1978 + 1920 at the first size: the staging of the values and the
// barriers around it.)  So large handles keep the flags.  Small ones, where a product loses at
// most 3 us, list their calls from the second AI-REML fit on, at its first one-column product, as
// they always have and as their statistics say (saige_grm_stats: missing_listed).
// SAIGE_SR_LISTS: 0 keeps the flag sums, 2 builds the lists at a handle's first one-column
// product (up to kMissListMaxFrac missing), otherwise (default) by this rule.
constexpr int64_t kSrListSmall = (int64_t)1 << 22;  // entries: up to kMissListMaxFrac missing
constexpr int64_t kSrListMost = (int64_t)1 << 24;   // up to kSrListFrac; above, none
constexpr double kSrListFrac = 0.003;

// The largest fraction of missing calls that the default lists (0: none).
static double sr_list_frac(const saige_grm* h) {
  const int64_t entries = h->m_pad * h->n_pad;
  return entries <= kSrListSmall ? kMissListMaxFrac : (entries <= kSrListMost ? kSrListFrac : 0.0);
}

static int sr_lists_mode() {
  const char* e = getenv("SAIGE_SR_LISTS");
  if (!e || !e[0]) return 1;
  return e[0] == '0' ? 0 : (e[0] == '2' ? 2 : 1);
}

// Pipeline trace: with SAIGE_TC_TRACE=1 each tensor-core launch records, for
// CTA 0 and its first stages, when loads were issued and landed, when the
// operand slot was free and filled, and when MMAs issued; the per-stage
// offsets (ns from the first load) are printed to stderr.
static Status trace_dump(TcPlan* p, const char* what, cudaStream_t st) {
  std::vector<unsigned long long> t((size_t)kTraceStages * kTraceSlots);
  SG_CUDA(cudaMemcpyAsync(t.data(), p->trace.ptr, t.size() * 8, cudaMemcpyDeviceToHost, st));
  SG_CUDA(cudaStreamSynchronize(st));
  const unsigned long long t0 = t[0];
  fprintf(stderr, "[tc trace] %s: stage load landed free filled may-issue issued reach (ns) | SM clock (MHz)\n", what);
  for (int k = 0; k < kTraceStages; k += (k < 8 ? 1 : 8)) {
    fprintf(stderr, "[tc trace] %3d", k);
    for (int e = 0; e < 7; ++e) {
      const unsigned long long v = t[(size_t)k * kTraceSlots + e];
      fprintf(stderr, " %9lld", v ? (long long)(v - t0) : -1LL);
    }
    // effective SM clock between the MMA warp's arrivals at stage 0 and stage k
    const unsigned long long c0 = t[7], ck = t[(size_t)k * kTraceSlots + 7];
    const unsigned long long g0 = t[6], gk = t[(size_t)k * kTraceSlots + 6];
    fprintf(stderr, " | %6.0f", (k > 0 && gk > g0) ? (double)(ck - c0) * 1e3 / (double)(gk - g0) : 0.0);
    fprintf(stderr, "\n");
  }
  SG_CUDA(cudaMemsetAsync(p->trace.ptr, 0, t.size() * 8, st));
  return Status();
}

// Builds the two tile copies of the packed genotypes (marker-major for pass A,
// sample-major for pass B) from the row-major copy, on the handle's stream.
// Tiles of the marker tiles [mt0, mt1) from the row-major rows, on stream st.
static Status tiles_range(saige_grm* h, TcPlan* p, int64_t mt0, int64_t mt1, cudaStream_t st) {
  if (mt1 <= mt0) return Status();
  const int64_t n_st = h->n_pad / kKt;
  pack_tiles_kernel<<<dim3((unsigned)n_st, (unsigned)(mt1 - mt0)), 256, 0, st>>>(
      h->geno, h->wpr, n_st, mt0, p->tiles_m.as<uint8_t>());
  SG_CHECK_LAUNCH();
  transpose_tiles_kernel<<<dim3((unsigned)(mt1 - mt0), (unsigned)n_st), 256, 0, st>>>(
      p->tiles_m.as<uint8_t>(), n_st, p->s_ld, mt0, p->tiles_s.as<uint8_t>());
  SG_CHECK_LAUNCH();
  count_launches(2);
  return Status();
}

static Status reserve_tiles(saige_grm* h, TcPlan* p, int64_t n_mt) {
  const size_t bytes = (size_t)n_mt * (size_t)(h->n_pad / kKt) * kTileBytes;
  SG_TRY(p->tiles_m.reserve(bytes));
  SG_TRY(p->tiles_s.reserve(bytes));
  p->s_ld = n_mt;
  return Status();
}

// A new plan with the kernels' attributes set and, when asked for, the trace buffer;
// the tiles are the caller's.
static Status tc_plan_new(TcPlan** out) {
  TcPlan* p = new TcPlan();
  auto bail = [&](Status s) {
    delete p;
    return s;
  };
  {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return bail(fail(SAIGE_ECUDA, "device: %s", cudaGetErrorString(e)));
  }
  for (auto kern : {tc_grm_kernel<false, false>, tc_grm_kernel<true, false>,
                    tc_grm_kernel<false, true>, tc_grm_kernel<true, true>}) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSmemBudget);
    if (e != cudaSuccess)
      return bail(fail(SAIGE_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e)));
  }
  {
    cudaError_t e = cudaFuncSetAttribute(sr_pass_kernel<false, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sr_list_smem(kSrChunkA, kSrRowsA));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(sr_pass_kernel<true, true>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sr_list_smem(kSrChunkB, kSrRowsB));
    if (e != cudaSuccess)
      return bail(fail(SAIGE_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e)));
  }
  const char* tr = getenv("SAIGE_TC_TRACE");
  p->tracing = tr && tr[0] == '1';
  if (p->tracing) {
    Status ts = p->trace.reserve((size_t)kTraceStages * kTraceSlots * 8);
    if (!ts.ok()) return bail(ts);
    // (tracing only) cleared on the legacy stream and waited for, since the handle's
    // non-blocking stream would not order itself after it
    cudaError_t e = cudaMemset(p->trace.ptr, 0, (size_t)kTraceStages * kTraceSlots * 8);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return bail(fail(SAIGE_ECUDA, "cudaMemset: %s", cudaGetErrorString(e)));
  }
  *out = p;
  return Status();
}

static Status tc_init(saige_grm* h) {
  if (h->tc) return Status();
  TcPlan* p = nullptr;
  SG_TRY(tc_plan_new(&p));
  PhaseTimer tm;
  Status bs = reserve_tiles(h, p, h->m_pad / kRows);
  if (bs.ok()) bs = tiles_range(h, p, 0, h->m_pad / kRows, h->stream);
  if (!bs.ok()) {
    delete p;
    return bs;
  }
  tm.mark(" tc tiles");
  h->tc = p;
  return Status();
}

Status tc_stream_begin(saige_grm* h, int64_t rows_cap) {
  if (h->tc) return fail(SAIGE_EINVAL, "tensor-core tiles already built");
  TcPlan* p = nullptr;
  SG_TRY(tc_plan_new(&p));
  Status s = reserve_tiles(h, p, ceil_div(rows_cap, (int64_t)kRows));
  if (!s.ok()) {
    delete p;
    return s;
  }
  h->tc = p;
  return Status();
}

Status tc_stream_tiles(saige_grm* h, int64_t mt0, int64_t mt1, cudaStream_t st) {
  if (!h->tc || mt1 > h->tc->s_ld) return fail(SAIGE_EINVAL, "tile range beyond the reserved tiles");
  return tiles_range(h, h->tc, mt0, mt1, st);
}

void tc_destroy(saige_grm* h) {
  if (!h || !h->tc) return;
  delete h->tc;
  h->tc = nullptr;
}

// Scalar block layout (device): per launch of R <= kMaxR columns.
struct Scal {
  unsigned long long* amax_v;  // R
  unsigned long long* amax_w;
  unsigned long long* amax_c;
  unsigned long long* sum_v;
  unsigned long long* sum_c;
  double* scale_v;
  double* scale_w;
  double* scale_c;
  unsigned int* err;
};

static Scal carve(TcPlan* p) {
  char* b = p->scal.as<char>();
  Scal s;
  s.amax_v = reinterpret_cast<unsigned long long*>(b);
  s.amax_w = s.amax_v + kMaxR;
  s.amax_c = s.amax_w + kMaxR;
  s.sum_v = s.amax_c + kMaxR;
  s.sum_c = s.sum_v + kMaxR;
  s.scale_v = reinterpret_cast<double*>(s.sum_c + kMaxR);
  s.scale_w = s.scale_v + kMaxR;
  s.scale_c = s.scale_w + kMaxR;
  s.err = reinterpret_cast<unsigned int*>(s.scale_c + kMaxR);
  return s;
}

// Budget of each pipeline wait in SM cycles; saige_tc_set_wait_budget changes it.
std::atomic<long long> g_tc_wait_cycles{kWaitCycles};

template <bool kPassB>
static cudaError_t launch_tc(unsigned grid, const TcArgs& args, cudaStream_t st) {
  TcArgs a = args;
  a.wait_cycles = g_tc_wait_cycles.load(std::memory_order_relaxed);
  if (a.sa < 2 || a.sa > kMaxSA || a.sl < 2 || a.sl > kMaxSL || a.sub < 1 || a.sub > 4)
    return cudaErrorInvalidValue;
  // an unpack group may wait on a load slot's codes only once the slot's previous load
  // is known to have landed (see the unpack loop): (sl - 1) sub + 1 >= sa
  if ((a.sl - 1) * a.sub + 1 < a.sa) return cudaErrorInvalidValue;
  const size_t smem = tc_fixed_bytes() + (size_t)a.sl * plan_l_stage(a.ng, kPassB, a.sub);
  if (smem > kSmemBudget) return cudaErrorInvalidValue;
  if (a.trace)
    tc_grm_kernel<kPassB, true><<<grid, kThreads, smem, st>>>(a);
  else
    tc_grm_kernel<kPassB, false><<<grid, kThreads, smem, st>>>(a);
  count_launches(1);
  return cudaGetLastError();
}

// ---- ring-shape autotuner ----------------------------------------------------
// The ring shape (sub-stages per load stage, load-ring depth, TMEM operand slots)
// does not change a product's result — the sums are exact integers and the epilogue
// is per element — only its speed.  So the tuning needs no launches of its own: the
// first launches of each key — pass, ng and the launch's size class (log2 of its 4 KB
// stages) — in the process each run the real product with the next candidate shape
// (sub 4, 2, 1 with the deepest ring the shared memory holds; tc_rings' choice first),
// timed with CUDA events
// that are read at the key's next launch; once every candidate has run, the fastest is
// kept for the later launches.  Launches of fewer than kTuneMinStages stages keep the
// fixed choice of tc_rings, as does SAIGE_TC_AUTOTUNE=0 (=2 tunes every size).
// SAIGE_TIMING=1 logs each timed candidate.
namespace {

struct TuneKey {
  int dev, pass_b, ng, size_class;
  bool operator<(const TuneKey& o) const {
    if (dev != o.dev) return dev < o.dev;
    if (pass_b != o.pass_b) return pass_b < o.pass_b;
    if (ng != o.ng) return ng < o.ng;
    return size_class < o.size_class;
  }
};

constexpr double kTuneMinStages = 1 << 20;  // ~4 GB of code tiles per launch

int size_class(double stages) {
  int c = 0;
  while (stages >= 2.0) {
    stages *= 0.5;
    ++c;
  }
  return c;
}

struct TuneState {
  std::vector<Rings> cand;
  std::vector<float> ms;               // per candidate; < 0: not timed (launch refused)
  size_t next = 0;                     // next candidate to run
  int pending = -1;                    // candidate whose events wait to be read
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  bool done = false;
  Rings best{};
};

std::mutex g_tune_mu;
std::map<TuneKey, TuneState> g_tune;
std::atomic<int64_t> g_tune_trials{0};

// SAIGE_TC_AUTOTUNE: 0 off, 2 every launch size, otherwise (default) launches of at
// least kTuneMinStages stages.
int autotune_level() {
  const char* e = getenv("SAIGE_TC_AUTOTUNE");
  if (!e || !e[0]) return 1;
  return e[0] == '0' ? 0 : (e[0] == '2' ? 2 : 1);
}

std::vector<Rings> tc_candidates(int ng, bool pass_b) {
  std::vector<Rings> out = {tc_rings(ng, pass_b)};  // the fixed choice first
  for (int sub : {4, 2, 1}) {
    const Rings g = ring_of(ng, pass_b, sub);
    if (sub != out[0].sub && g.sl >= 2 && g.sa >= 2) out.push_back(g);
  }
  return out;
}

}  // namespace

// Launches pass kPassB with the tuned ring shape of its key, tuning it first when the
// key is new.  a carries everything but the ring shape.
template <bool kPassB>
static Status launch_tc_tuned(int dev, unsigned grid, TcArgs a, cudaStream_t st) {
  const Rings fixed = tc_rings(a.ng, kPassB);
  const double stages = ((double)a.whole * grid + a.extra) * a.nk + (double)a.tail_units;
  const int level = autotune_level();
  if (level == 0 || (level == 1 && stages < kTuneMinStages)) {
    a.sub = fixed.sub;
    a.sl = fixed.sl;
    a.sa = fixed.sa;
    SG_CUDA(launch_tc<kPassB>(grid, a, st));
    return Status();
  }
  const TuneKey key{dev, kPassB ? 1 : 0, a.ng, size_class(stages)};
  auto use = [&](const Rings& g) {
    a.sub = g.sub;
    a.sl = g.sl;
    a.sa = g.sa;
  };
  // the state is held under the lock through the (asynchronous) launch, so that one
  // key's candidates and events are used by one launch at a time
  std::lock_guard<std::mutex> lk(g_tune_mu);
  TuneState& ts = g_tune[key];
  if (ts.done) {
    use(ts.best);
    SG_CUDA(launch_tc<kPassB>(grid, a, st));
    return Status();
  }
  if (ts.cand.empty()) {
    ts.cand = tc_candidates(a.ng, kPassB);
    ts.ms.assign(ts.cand.size(), -1.f);
    SG_CUDA(cudaEventCreate(&ts.e0));
    SG_CUDA(cudaEventCreate(&ts.e1));
  }
  const char* tlog = getenv("SAIGE_TIMING");
  const bool log = tlog && tlog[0] == '1';
  if (ts.pending >= 0) {  // the previous candidate's launch of this key has long been queued
    SG_CUDA(cudaEventSynchronize(ts.e1));
    float ms = 0.f;
    SG_CUDA(cudaEventElapsedTime(&ms, ts.e0, ts.e1));
    ts.ms[(size_t)ts.pending] = ms;
    const Rings& g = ts.cand[(size_t)ts.pending];
    if (log)
      fprintf(stderr, "[saige tune] pass %c ng %d grid %u nk %d: sub %d sl %d sa %d -> %.3f ms\n",
              kPassB ? 'B' : 'A', a.ng, grid, a.nk, g.sub, g.sl, g.sa, ms);
    ts.pending = -1;
  }
  while (ts.next < ts.cand.size()) {
    const size_t c = ts.next++;
    use(ts.cand[c]);
    SG_CUDA(cudaEventRecord(ts.e0, st));
    const cudaError_t le = launch_tc<kPassB>(grid, a, st);
    if (le != cudaSuccess) {  // a shape the launch refuses: next candidate
      (void)cudaGetLastError();
      continue;
    }
    SG_CUDA(cudaEventRecord(ts.e1, st));
    ts.pending = (int)c;
    g_tune_trials += 1;
    return Status();
  }
  // every candidate has run: keep the fastest
  int bi = -1;
  for (size_t c = 0; c < ts.cand.size(); ++c)
    if (ts.ms[c] >= 0.f && (bi < 0 || ts.ms[c] < ts.ms[(size_t)bi])) bi = (int)c;
  ts.best = bi >= 0 ? ts.cand[(size_t)bi] : fixed;
  ts.done = true;
  use(ts.best);
  SG_CUDA(launch_tc<kPassB>(grid, a, st));
  return Status();
}

int64_t tc_autotune_trials() { return g_tune_trials.load(); }

int64_t tc_missing_listed(const saige_grm* h) {
  return h->tc && h->tc->miss.state == 1 ? h->tc->miss.total : -1;
}

void tc_set_wait_budget(long long cycles) {
  g_tc_wait_cycles.store(cycles < 0 ? kWaitCycles : cycles, std::memory_order_relaxed);
}

// Sets the work division of a launch over `tiles` tiles, which CTAs share only when there is room
// for the sums (`share`); returns its grid.
static unsigned set_work(TcArgs* a, int64_t tiles, const TcPlan* p, bool share) {
  const TcWork w = tc_work(tiles, a->nk, p->sms, share);
  a->whole = w.whole;
  a->extra = w.extra;
  a->tail_tile = w.tail_tile;
  a->tail_units = w.tail_units;
  // the counts come first: their place does not depend on the columns
  a->part_done = p->part.as<unsigned int>();
  a->part = reinterpret_cast<unsigned long long*>(p->part.as<char>() + part_counts(p));
  return (unsigned)w.grid;
}

// Room, all zero, for the sums and counts of tiles that CTAs share when r columns are in a
// launch: a slot per CTA (see TcWork).
static Status part_reserve(TcPlan* p, int r, cudaStream_t st) {
  const size_t want = part_counts(p) + (size_t)p->sms * 2 * r * kRows * 8;
  if (want <= p->part.bytes) return Status();
  SG_TRY(p->part.reserve(want));
  SG_CUDA(cudaMemsetAsync(p->part.ptr, 0, p->part.bytes, st));
  return Status();
}

Status tc_product_failed(saige_grm* h, unsigned int err, cudaStream_t st) {
  if (err & kSrListErr)
    return fail(SAIGE_ECUDA, "one-column GRM product: a missing-call list entry out of range");
  // shared tiles may be left half summed
  TcPlan* p = h->tc;
  if (p->part.ptr) SG_CUDA(cudaMemsetAsync(p->part.ptr, 0, p->part.bytes, st));
  SG_CUDA(cudaStreamSynchronize(st));
  return fail(SAIGE_TIMEOUT, "tensor-core GRM product: a pipeline wait timed out");
}

Status tc_product(saige_grm* h, const double* v, double* kp, int q, const int32_t* active,
                  cudaStream_t st, unsigned int* later) {
  SG_TRY(tc_init(h));
  TcPlan* p = h->tc;
  std::vector<int> cols;
  for (int c = 0; c < q; ++c)
    if (!active || active[c] == kColActive) cols.push_back(c);
  if (cols.empty()) return Status();
  if (st != h->stream) {
    // the tiles were built on the handle's stream
    cudaEvent_t built;
    SG_CUDA(cudaEventCreateWithFlags(&built, cudaEventDisableTiming));
    SG_CUDA(cudaEventRecord(built, h->stream));
    SG_CUDA(cudaStreamWaitEvent(st, built, 0));
    cudaEventDestroy(built);
  }
  const int64_t n_stages_a = h->n_pad / kKt;  // samples
  const int64_t n_stages_b = h->m_pad / kKt;  // markers
  const int rmax = (int)std::min<size_t>(cols.size(), (size_t)kMaxR);
  const int ng_max = (int)round_up(3 * rmax, 16);
  SG_TRY(p->img_a.reserve((size_t)h->n_pad * ng_max));
  SG_TRY(p->img_w.reserve((size_t)h->m_pad * ng_max));
  SG_TRY(p->img_c.reserve((size_t)h->m_pad * ng_max));
  SG_TRY(p->u.reserve((size_t)h->m_pad * rmax * sizeof(double)));
  const size_t scal_bytes = 9 * kMaxR * 8 + 64;
  SG_TRY(p->scal.reserve(scal_bytes));
  const uint8_t* excl = h->masked ? h->excl.as<uint8_t>() : nullptr;
  Scal sc = carve(p);
  // The kernels write the error word where the host reads it: `later`, or a word of the handle's
  // page-locked block (idle here: every product's word is read after a wait), or, without one,
  // device memory.
  if (h->profiling || p->tracing) later = nullptr;
  unsigned int* word = later;
  if (!word)
    if (char* pin = static_cast<char*>(h->pin.get()))
      word = reinterpret_cast<unsigned int*>(pin + kPinBytes - kPinWord);
  if (word) {
    *word = 0u;
    sc.err = word;
  }
  // per-pass CUDA-event timing when profiling is on (events on the launching stream)
  std::vector<cudaEvent_t> ev;
  auto mark = [&](cudaEvent_t* e) -> Status {
    if (!h->profiling) return Status();
    SG_CUDA(cudaEventCreate(e));
    ev.push_back(*e);
    SG_CUDA(cudaEventRecord(*e, st));
    return Status();
  };
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_a, ev_b, ev_s;
  const char* sc_env = getenv("SAIGE_SC");
  const bool single = cols.size() == 1 && !(sc_env && sc_env[0] == '0');
  if (single) {
    // one column: both passes by sr_pass_kernel (same integer sums, same epilogue)
    int8_t* planes_a = p->img_a.as<int8_t>();  // 3 x n_pad limb planes of q
    int8_t* planes_b = p->img_w.as<int8_t>();  // 6 x m_pad limb planes of qw, qc
    double* u = p->u.as<double>();
    const int lmode = sr_lists_mode();
    const double frac = lmode == 2 ? kMissListMaxFrac : (lmode == 1 ? sr_list_frac(h) : 0.0);
    if ((p->miss.state == 0 && (lmode == 2 || (frac > 0.0 && h->n_fits >= 2))) ||
        (p->miss.state == kMissListsLeft && lmode == 2))
      SG_TRY(miss_lists_build(
          h, p->tiles_s.as<uint8_t>(), p->s_ld,
          MissShape{kSrRowsA, kSrChunkA / 16, kSrRowsB, kSrChunkB}, frac, &p->miss, st));
    const bool lists = p->miss.state == 1 && lmode != 0;
    int32_t *qv32 = nullptr, *qc32 = nullptr;
    if (lists) {
      SG_TRY(p->sr_q32.reserve((size_t)(h->n_pad + h->m_pad) * sizeof(int32_t)));
      qv32 = p->sr_q32.as<int32_t>();
      qc32 = qv32 + h->n_pad;
    }
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    SG_TRY(mark(&t0));
    SG_CUDA(cudaMemsetAsync(p->scal.ptr, 0, scal_bytes, st));  // maxima, sums, error word
    ColMap cm{};
    cm.c[0] = cols[0];
    amax_v_kernel<<<(unsigned)ceil_div(h->n, kAmaxRows), 256, 0, st>>>(v, h->n_pad, h->n, cm,
                                                                       sc.amax_v);
    sr_quant_v_kernel<<<(unsigned)ceil_div(h->n_pad, 256), 256, 0, st>>>(
        v + (int64_t)cols[0] * h->n_pad, h->n, h->n_pad, sc.amax_v, sc.scale_v, planes_a, qv32,
        sc.sum_v);
    const unsigned blocks_a = (unsigned)(h->m_pad / kSrRowsA);
    const unsigned blocks_b = (unsigned)(h->n_pad / kSrRowsB);  // (n_pad: a multiple of 512)
    SrArgs a{};
    a.split = sr_split(blocks_a, n_stages_a, p->sms, kSrCostA);
    SrArgs b{};
    b.split = sr_split(blocks_b, n_stages_b, p->sms, kSrCostB);
    if ((a.split.blocks > 1 || b.split.blocks > 1) && !p->sr_sums.ptr) {
      const size_t bytes = (size_t)std::max(h->n_pad, h->m_pad) * 16 +
                           (size_t)std::max(blocks_a, blocks_b) * 4;
      const Status ss = p->sr_sums.reserve(bytes);
      if (ss.ok()) {
        SG_CUDA(cudaMemsetAsync(p->sr_sums.ptr, 0, bytes, st));
      } else if (ss.code == SAIGE_ENOMEM) {  // undivided, for the same sums
        set_error("");
        a.split = SrSplit{n_stages_a, 1};
        b.split = SrSplit{n_stages_b, 1};
      } else {
        return ss;
      }
    }
    a.sums_g = p->sr_sums.as<unsigned long long>();
    a.sums_m = a.sums_g + std::max(h->n_pad, h->m_pad);
    a.tickets = reinterpret_cast<unsigned int*>(a.sums_m + std::max(h->n_pad, h->m_pad));
    b.sums_g = a.sums_g;
    b.sums_m = a.sums_m;
    b.tickets = a.tickets;
    a.tiles = p->tiles_m.as<uint8_t>();
    a.ld = n_stages_a;
    a.n_kt = n_stages_a;
    a.planes = planes_a;
    a.q32 = qv32;
    a.ent = p->miss.a_ent.as<uint32_t>();
    a.seg = p->miss.a_seg.as<int64_t>();
    a.nch = p->miss.a_nch;
    a.bits = p->miss.a_bits;
    a.err = sc.err;
    a.sum_q = sc.sum_v;
    a.scale_g = sc.scale_v;
    a.two_p = h->two_p;
    a.inv_s = h->inv_s;
    a.out = u;
    const dim3 grid_a(blocks_a, a.split.blocks);
    if (lists)
      sr_pass_kernel<false, true><<<grid_a, 256, sr_list_smem(kSrChunkA, kSrRowsA), st>>>(a);
    else
      sr_pass_kernel<false, false><<<grid_a, 256, 0, st>>>(a);
    SG_CHECK_LAUNCH();
    amax_wc_kernel<<<(unsigned)ceil_div(h->m_pad, kAmaxRows), 256, 0, st>>>(
        u, h->m_pad, h->m_pad, h->inv_s, h->two_p, excl, h->m, sc.amax_w, sc.amax_c);
    sr_quant_wc_kernel<<<(unsigned)ceil_div(h->m_pad, 256), 256, 0, st>>>(
        u, h->m_pad, h->inv_s, h->two_p, sc.amax_w, sc.amax_c, sc.scale_w, sc.scale_c, planes_b,
        qc32, sc.sum_c);
    b.tiles = p->tiles_s.as<uint8_t>();
    b.ld = p->s_ld;
    b.n_kt = n_stages_b;
    b.planes = planes_b;
    b.q32 = qc32;
    b.ent = p->miss.b_ent.as<uint32_t>();
    b.seg = p->miss.b_seg.as<int64_t>();
    b.nch = p->miss.b_nch;
    b.bits = p->miss.b_bits;
    b.err = sc.err;
    b.sum_q = sc.sum_c;
    b.scale_g = sc.scale_w;
    b.scale_m = sc.scale_c;
    b.out_scale = 1.0 / (double)(h->masked ? h->m_active : h->m_eff);
    b.out = kp + (int64_t)cols[0] * h->n_pad;
    const dim3 grid_b(blocks_b, b.split.blocks);
    if (lists)
      sr_pass_kernel<true, true><<<grid_b, 256, sr_list_smem(kSrChunkB, kSrRowsB), st>>>(b);
    else
      sr_pass_kernel<true, false><<<grid_b, 256, 0, st>>>(b);
    SG_CHECK_LAUNCH();
    count_launches(6);
    SG_TRY(mark(&t1));
    if (h->profiling) ev_s.emplace_back(t0, t1);
    h->stats.sc_launches += 1;
    h->stats.sc_list_launches += lists ? 1 : 0;
    h->n_kv += 1;
  }
  bool share = false;
  if (!single) {
    // short of memory: no tile is shared, for the same sums
    const Status ps = part_reserve(p, rmax, st);
    if (!ps.ok() && ps.code != SAIGE_ENOMEM) return ps;
    if (!ps.ok()) set_error("");
    share = ps.ok();
  }
  for (size_t c0 = 0; c0 < (single ? 0 : cols.size()); c0 += kMaxR) {
    const int r = (int)std::min<size_t>(kMaxR, cols.size() - c0);
    const int ng = (int)round_up(3 * r, 16);
    ColMap cm{};
    for (int k = 0; k < r; ++k) cm.c[k] = cols[c0 + (size_t)k];
    // maxima and sums (the error word is zeroed before the first group only)
    SG_CUDA(cudaMemsetAsync(p->scal.ptr, 0, c0 == 0 ? scal_bytes : 5 * kMaxR * 8, st));
    // ---- pass A operand ----
    {
      dim3 g1((unsigned)ceil_div(h->n, kAmaxRows), (unsigned)r);
      amax_v_kernel<<<g1, 256, 0, st>>>(v, h->n_pad, h->n, cm, sc.amax_v);
      count_launches(2);
      dim3 g2((unsigned)ceil_div(n_stages_a, (int64_t)4), (unsigned)r);
      quant_v_kernel<<<g2, 128, 0, st>>>(v, h->n_pad, h->n, n_stages_a, cm, sc.amax_v, sc.scale_v,
                                         p->img_a.as<uint8_t>(), ng, sc.sum_v);
      SG_CHECK_LAUNCH();
    }
    // ---- pass A: u = Z' v ----
    {
      TcArgs a{};
      a.ng = ng;
      a.r = r;
      a.nk = (int)n_stages_a;
      a.tiles = p->tiles_m.as<uint8_t>();
      a.tile_ld = n_stages_a;
      a.img_g = p->img_a.as<uint8_t>();
      a.scale_g = sc.scale_v;
      a.sum_q = reinterpret_cast<const long long*>(sc.sum_v);
      a.two_p = h->two_p;
      a.inv_s = h->inv_s;
      a.out = p->u.as<double>();
      a.out_ld = h->m_pad;
      a.err = sc.err;
      a.trace = p->tracing ? p->trace.as<unsigned long long>() : nullptr;
      const unsigned grid = set_work(&a, h->m_pad / kRows, p, share);
      cudaEvent_t t0 = nullptr, t1 = nullptr;
      SG_TRY(mark(&t0));
      SG_TRY(launch_tc_tuned<false>(h->device, grid, a, st));
      SG_TRY(mark(&t1));
      if (h->profiling) ev_a.emplace_back(t0, t1);
      h->stats.tc_pass_a_launches += 1;
      if (p->tracing) SG_TRY(trace_dump(p, "pass A", st));
    }
    // ---- pass B operands ----
    {
      dim3 g1((unsigned)ceil_div(h->m_pad, kAmaxRows), (unsigned)r);
      count_launches(2);
      amax_wc_kernel<<<g1, 256, 0, st>>>(p->u.as<double>(), h->m_pad, h->m_pad, h->inv_s,
                                         h->two_p, excl, h->m, sc.amax_w, sc.amax_c);
      dim3 g2((unsigned)ceil_div(n_stages_b, (int64_t)4), (unsigned)r);
      quant_wc_kernel<<<g2, 128, 0, st>>>(p->u.as<double>(), h->m_pad, n_stages_b, h->inv_s,
                                          h->two_p, sc.amax_w, sc.amax_c, sc.scale_w, sc.scale_c,
                                          p->img_w.as<uint8_t>(), p->img_c.as<uint8_t>(), ng,
                                          sc.sum_c);
      SG_CHECK_LAUNCH();
    }
    // ---- pass B: y = Z w / M ----
    {
      TcArgs a{};
      a.ng = ng;
      a.r = r;
      a.nk = (int)n_stages_b;
      a.tiles = p->tiles_s.as<uint8_t>();
      a.tile_ld = p->s_ld;
      a.img_g = p->img_w.as<uint8_t>();
      a.img_m = p->img_c.as<uint8_t>();
      a.scale_g = sc.scale_w;
      a.scale_m = sc.scale_c;
      a.sum_q = reinterpret_cast<const long long*>(sc.sum_c);
      a.out = kp;
      a.out_ld = h->n_pad;
      a.col_map = cm;
      a.out_scale = 1.0 / (double)(h->masked ? h->m_active : h->m_eff);
      a.err = sc.err;
      a.trace = p->tracing ? p->trace.as<unsigned long long>() : nullptr;
      const unsigned grid = set_work(&a, h->n_pad / kRows, p, share);
      cudaEvent_t t0 = nullptr, t1 = nullptr;
      SG_TRY(mark(&t0));
      SG_TRY(launch_tc_tuned<true>(h->device, grid, a, st));
      SG_TRY(mark(&t1));
      if (h->profiling) ev_b.emplace_back(t0, t1);
      h->stats.tc_pass_b_launches += 1;
      if (p->tracing) SG_TRY(trace_dump(p, "pass B", st));
    }
    h->n_kv += r;
  }
  h->n_kv_launches += 1;
  if (later) return Status();
  unsigned int err = 0;
  if (word) {
    SG_CUDA(cudaStreamSynchronize(st));
    err = *word;
  } else {
    SG_TRY(read_back(h, &err, sc.err, sizeof(err), st));
  }
  for (auto& pr : ev_a) {
    float ms = 0.f;
    SG_CUDA(cudaEventElapsedTime(&ms, pr.first, pr.second));
    h->stats.tc_pass_a_ms += ms;
  }
  for (auto& pr : ev_b) {
    float ms = 0.f;
    SG_CUDA(cudaEventElapsedTime(&ms, pr.first, pr.second));
    h->stats.tc_pass_b_ms += ms;
  }
  for (auto& pr : ev_s) {
    float ms = 0.f;
    SG_CUDA(cudaEventElapsedTime(&ms, pr.first, pr.second));
    h->stats.sc_ms += ms;
  }
  for (cudaEvent_t e : ev) cudaEventDestroy(e);
  return err ? tc_product_failed(h, err, st) : Status();
}

}  // namespace saige
