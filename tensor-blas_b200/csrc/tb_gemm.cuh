// Persistent warp-specialised tcgen05 GEMM engine (sm_100a).
//
//   C[m0+i, n0+j] = alpha * sum_k A(m0+i, k) * B(n0+j, k) + beta * C[...]
//
// over a host-built list of 128 x BN output tiles, each with its own K-block
// range. This single kernel serves every contraction of the library: the
// flattened recursion levels of SYRK/SYR2K (lower-triangle tile lists), the
// off-diagonal updates and leaf products of TRSM, and TRMM/SYMM.
//
// Roles (384 threads, one CTA per SM):
//   warp 0       TMA producer: 64-wide K slabs of A and B into a smem ring.
//   warp 1       TMEM allocator + single-thread UMMA issuer.
//   warp 2       C loader: streams 128 x 16 chunks of C into the epilogue's
//                shared-memory slots ahead of their use.
//   warps 4..11  epilogue, two groups of four warps, one half of the tile's
//                columns each: TMEM -> registers -> alpha/beta -> C.
// The fp32 accumulators are double-buffered in TMEM so the epilogue of tile t
// overlaps the MMAs of tile t+1.
//
// Operands are fp16 in global memory, either MN-major (column-major storage
// with the M/N index contiguous, the layout the reference's FP32->FP16
// conversion produces) or K-major. Both map onto 128B-swizzled UMMA canonical
// layouts:
//   MN-major: TMA box {64 (MN), 64 (K)} -> 8 KB atoms; LBO = 8 KB between
//             64-wide MN atoms, SBO = 1 KB between 8-row K groups; a K step of
//             16 advances the descriptor by 2 KB.
//   K-major : TMA box {64 (K), R rows} -> R x 128 B; SBO = 1 KB between
//             8-row groups; a K step of 16 advances the descriptor by 32 B.
//
// Output: each 128 x 16 chunk of the tile is staged in shared memory
// (column-major, 512 B per column) and written with one TMA tensor store, so
// HBM sees 512-byte runs instead of one 128-byte piece per warp and column.
// When beta != 0 the chunk of C is first brought in with a TMA load and
// combined in shared memory (masked elements keep their old value). A plain
// per-element path serves C that TMA cannot address (unaligned base or
// leading dimension) and masked tiles with beta = 0.
//
// Split ("3-product") mode holds hi and lo copies of both operands and runs
//   acc0 += Ahi*Bhi ; acc1 += Ahi*Blo + Alo*Bhi
// with the correction in its own TMEM accumulator (Ootomo & Yokota 2022,
// the error-corrected FP16 scheme cuMpSGEMM's FP16TCEC mode uses). Every
// `kchunk` K-blocks the epilogue adds acc0 to FP32 registers with
// round-to-nearest adds: the tensor core's own FP32 accumulation truncates,
// which would cost ~K/16 ulps. The correction, 2^-11 of the result, stays in
// its accumulator for kCorrRounds such folds, so that most of them read half
// the TMEM columns and round half as often.
#pragma once
#include "tb_internal.h"
#include "tb_ptx.cuh"

namespace tb {

struct GemmArgs {
  CUtensorMap mapA[2];  // [0] hi, [1] lo (split mode only)
  CUtensorMap mapB[2];
  CUtensorMap mapC;     // fp32 C, box {128, 16} (TMA epilogue only)
  const int4* tiles;    // {m0, n0, kb_begin, kb_end}; m0/n0 relative to C
  int num_tiles;
  int a_off;  // row offset of the A operand in mapA's row coordinate
  int b_off;  // row offset of the B operand in mapB's row coordinate
  int k_off;  // K offset (elements) applied to both operands
  int M, N;   // extent of C (predication)
  float* C;
  long long ldc;
  float alpha, beta;
  int tri;   // 1: write only (i - j) >= diag (lower triangle); 2: only (j - i) >= diag (upper)
  int diag;
  float corr_scale;  // weight of the correction accumulator
  int kchunk;        // split mode: K-blocks per round-to-nearest fold
  int tma_c;         // 1: C through mapC (TMA epilogue)
  // Optional fused fp16 copies of the written result (column-major, ld_out):
  //   out_hi = fp16(v), out_lo = fp16((v - out_hi) * out_lo_scale)
  __half* out_hi;
  __half* out_lo;
  long long ld_out;
  float out_lo_scale;
  int out_m, out_n;  // side copies only for rows < out_m and columns < out_n
  int* err;
  // FP8: per-(128-row block, 128-deep K block) scales of the A and B
  // operands, row-block-major with scale_ld K blocks per row block.
  const float* scale_a;
  const float* scale_b;
  int scale_ld;
  // Grouped launches: per-tile problem index into a device array of
  // GemmArgs (64-byte aligned; their tensor maps are read from global memory).
  const struct GemmArgs* problems;
  const int* tile_prob;
  // Device-side tile scheduler: nullptr = static assignment; otherwise a
  // zeroed counter from which the CTAs' producers claim tiles one at a time.
  int* sched;
  // Static assignment: nullptr = striding (CTA b takes tiles b, b + grid,
  // ...); otherwise CTA (or CTA pair) b takes tiles [ranges[b], ranges[b+1])
  // of a list the host balanced by simulating greedy claiming.
  const int* ranges;
};

// First / next tile of CTA (or CTA pair) `b` of `nb` under the static
// assignment; -1 when there is none.
__device__ __forceinline__ int static_first(const GemmArgs& a, int b) {
  if (a.ranges) return a.ranges[b] < a.ranges[b + 1] ? a.ranges[b] : -1;
  return b < a.num_tiles ? b : -1;
}
__device__ __forceinline__ int static_next(const GemmArgs& a, int b, int nb, int t) {
  if (a.ranges) return t + 1 < a.ranges[b + 1] ? t + 1 : -1;
  return t + nb < a.num_tiles ? t + nb : -1;
}

// Tile hand-off inside a CTA under the device-side scheduler: the producer
// claims a tile and queues its index (or -1, the end) in a kTileQ-deep ring;
// the MMA issuer, the eight epilogue warps and the C loader each take the
// indices in order and release the slot.
constexpr int kTileQ = 4;

// Split mode: main folds for which the correction stays in its accumulator (a
// stretch; 128 K-blocks, K = 8192, with the default fold interval). The sum in
// TMEM truncates about twice per 16-deep step, so a stretch loses at most
// 2^-22 * 512 / 2 = 6e-5 of a correction that is at most 2^-11 of the sum of
// the products' magnitudes: half an FP32 unit roundoff of that sum, whatever
// K is. Over the whole K range the loss grows with K: with lo parts of one
// sign the correction was off by 1.1e-4 at K = 16384, 2.1e-4 at 32768 and
// 8.6e-4 at 131072, now 5e-5 at each. Each stretch end adds one rounding per
// element; folded every 16 rounds or every 8 the error of U[-1, 1] operands
// at K = 16384 rose from 3.72e-7 to 3.73e-7 or 3.76e-7, and folding every
// round (two roundings a fold) made it 3.98e-7. Time: within the runs' spread
// (SGEMM 4096 x 4096 x 32768 on pairs 2.62 to 2.69 ms before and after).
constexpr int kCorrRounds = 32;

// The next tile of a consumer role: static striding, or the producer's
// queue (q/ph: the role's ring position). EPI: called by the 128 threads of
// an epilogue group together, which then agree on the result (named barrier
// `bar`).
template <bool EPI>
__device__ __forceinline__ int next_tile(const GemmArgs& args, int t, const volatile int* tq_idx, uint64_t* tq_full,
                                         uint64_t* tq_empty, int& q, uint32_t& ph, volatile int* abort_flag,
                                         int code, int bar = 1) {
  if (!args.sched) return t < 0 ? static_first(args, blockIdx.x) : static_next(args, blockIdx.x, gridDim.x, t);
  const bool got = mbar_wait(&tq_full[q], ph, abort_flag, args.err, code);
  int v = got ? tq_idx[q] : -1;
  if constexpr (EPI) {
    if (named_bar_any(bar, 128, !got)) v = -1;
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(&tq_empty[q]);
  } else {
    mbar_arrive(&tq_empty[q]);
  }
  if (++q == kTileQ) {
    q = 0;
    ph ^= 1u;
  }
  return v;
}

// The problem a tile belongs to: the launch's own arguments, or (grouped
// launches) one of the descriptors in global memory.
template <bool GROUPED>
__device__ __forceinline__ const GemmArgs& tile_problem(const GemmArgs& args, int t) {
  if constexpr (GROUPED) {
    return args.problems[args.tile_prob[t]];
  } else {
    return args;
  }
}

// Epilogue: two groups of four warps, each with one half of the tile's
// columns, its own C slots and its own named barrier, in rolled loops over
// chunks of 16 columns. What bounded the short launches was neither the MMAs
// nor memory but instruction fetch: with four warps and the fold's 128
// register sums handed to four unrolled 32-column copies of the store code, a
// launch of four 128 x 128 tiles with 4 K-blocks took 22 us, of which the MMAs
// were 2, and a TRSM leaf product of 512 x 16384 42.6 us. A group now runs one
// short copy of the chunk code on 16 columns at a time, read back from TMEM
// (split: the folded tile replaces its correction there) or picked out of the
// fold's registers (pick16): 15 and 35 us. C (TMA slots) or the old values
// (per-element path) are on their way before the accumulator is: a leaf
// product of 6003 x 512 with an odd leading dimension went from 73 to 30 us,
// the 512-instance batch from 6.5 to 5.1 ms.
constexpr int kEpiGroups = 2;
constexpr int kEpiWarp0 = 4;  // first epilogue warp
constexpr int kGemmThreads = 32 * (kEpiWarp0 + 4 * kEpiGroups);

// Shared memory left beside the operand stages goes to the C slots: a group's
// loader ring runs that many 8 KB chunks ahead of its epilogue.
// PF variants (plain, 128 x 128) serve launches whose tiles have few K-blocks:
// there C, not the MMA, bounds the tile, so they trade operand stages for C
// slots. A split tile's three stages leave room for two slots a group at any K.
// FP8 variant: e4m3 K-major operands scaled per 128 x 128 block; the
// accumulator is folded into fp32 registers after every 128-deep K block
// with the product of the two blocks' scales.
// BN = 64 variants serve launches that leave more than half of the SMs idle
// with wider tiles (the small solves): twice the CTAs, half the epilogue.
template <int BN_, int NSPLIT_, bool A_MN_, bool B_MN_, bool PF_ = false, bool FP8_ = false>
struct GemmCfg {
  static constexpr bool PF = PF_;
  static constexpr bool FP8 = FP8_;
  static_assert(!PF || (BN_ == 128 && NSPLIT_ == 1 && !FP8), "PF: plain 128 x 128 tiles");
  static constexpr int ELEM = FP8 ? 1 : 2;       // operand bytes per element
  static constexpr int BM = 128, BN = BN_, BK = 128 / ELEM;  // one 128-byte swizzle row of K per stage
  static constexpr int KSTEPS = 4;               // MMAs per stage (K = 16 fp16 / 32 fp8 each)
  static constexpr int NSPLIT = NSPLIT_;
  static constexpr bool A_MN = A_MN_, B_MN = B_MN_;
  static constexpr bool SPLIT = NSPLIT > 1;
  static constexpr bool FOLD = SPLIT || FP8;  // accumulate in registers across TMEM rounds
  static constexpr int NOPS = SPLIT ? 2 : 1;  // copies per operand (hi[, lo])
  static constexpr int A_BYTES = BM * BK * ELEM;
  static constexpr int B_BYTES = BN * BK * ELEM;
  static constexpr int STAGE_BYTES = NOPS * (A_BYTES + B_BYTES);
  static constexpr int STAGES = SPLIT ? (BN == 64 ? 4 : 3) : (PF || BN == 256) ? 4 : 6;
  // TMEM: two main accumulators (alternating by round), then two corrections
  // (alternating by stretch)
  static constexpr int CORR_COL = 2 * BN;
  static constexpr int TMEM_COLS = (SPLIT ? 4 : 2) * BN;
  static_assert(TMEM_COLS <= 512, "TMEM budget");
  static constexpr int GC = BN / kEpiGroups;              // columns of one epilogue group
  static constexpr int CHUNK_BYTES = 128 * kEpiCols * 4;  // one staged 128 x 16 fp32 chunk
  static constexpr int C_SLOTS = PF ? 6 : 2;              // per group (BN = 64: all its chunks)
  static constexpr int GROUP_BYTES = C_SLOTS * CHUNK_BYTES;
  static constexpr int EPI_BYTES = kEpiGroups * GROUP_BYTES;
  static constexpr int BAR_BYTES = 512;
  static_assert(8 * (2 * STAGES + 7 + 2 * kEpiGroups * C_SLOTS + 2 * kTileQ) + 4 * kTileQ + 8 <= BAR_BYTES,
                "barrier space");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 + BAR_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  static constexpr uint32_t IDESC = idesc_f16(BM, BN, false, A_MN, B_MN);
};

template <bool MN, int ROWS>
__device__ __forceinline__ void load_operand(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row0, int k) {
  if constexpr (MN) {
#pragma unroll
    for (int j = 0; j < ROWS / 64; ++j) tma_load_2d(dst + j * 8192, map, bar, row0 + 64 * j, k);
  } else {
    tma_load_2d(dst, map, bar, k, row0);
  }
}

template <bool MN>
__device__ __forceinline__ uint64_t operand_desc(uint32_t base, int kk) {
  if constexpr (MN) {
    return sdesc_sw128(base + kk * 2048, 8192, 1024);
  } else {
    return sdesc_sw128(base + kk * 32, 16, 1024);
  }
}

// Output triangle mask: tri 1 writes only (i - j) >= diag (lower), tri 2
// only (j - i) >= diag (upper); masked elements keep their old value.
// Whether a BM x BN tile at (m0, n0) reaches into the masked region.
__device__ __forceinline__ bool tile_reaches_mask(const GemmArgs& a, long long m0, long long n0, int bm, int bn) {
  return a.tri == 1 ? (m0 - (n0 + bn - 1)) < a.diag : (a.tri == 2 ? (n0 - (m0 + bm - 1)) < a.diag : false);
}

// Epilogue scalars, read into registers once per tile. The epilogue's
// stores go through generic pointers (shared-memory slots, C, side copies)
// that the compiler cannot tell apart from the kernel's parameter memory (or
// a grouped launch's descriptor in global memory), so GemmArgs fields read
// inside a store loop may be reloaded after every store.
struct EpiK {
  float alpha, beta, lo_scale;
  int tri, diag;
  __device__ __forceinline__ explicit EpiK(const GemmArgs& a)
      : alpha(a.alpha), beta(a.beta), lo_scale(a.out_lo_scale), tri(a.tri), diag(a.diag) {}
  // some element of the 128 x W chunk at (m0, n0) is masked
  template <int W>
  __device__ __forceinline__ bool chunk_masked(long long m0, long long n0) const {
    return tri == 1 ? (m0 - (n0 + W - 1)) < diag : (tri == 2 ? (n0 - (m0 + 127)) < diag : false);
  }
  // The columns gj0 + [lo, hi) of row gi, out of the W from gj0 and below
  // `ncols` (a bound on gj), that the mask keeps: one range per row, so the
  // element loops compare small ints instead of testing every element's
  // 64-bit (i, j) against the triangle (which cost more than the stores).
  template <int W>
  __device__ __forceinline__ void keep_range(long long gi, long long gj0, long long ncols, int& lo, int& hi) const {
    long long h = ncols - gj0, l = 0;
    if (tri == 1) h = min(h, gi - diag + 1 - gj0);  // keep gj <= gi - diag
    if (tri == 2) l = gi + diag - gj0;              // keep gj >= gi + diag
    hi = (int)max(0LL, min((long long)W, h));
    lo = (int)max(0LL, min((long long)W, l));
  }
};

// New values of one row's W staged C elements: alpha v + beta old where
// unmasked (old kept where masked), written back in place.
template <int W>
__device__ __forceinline__ void combine(const EpiK& k, float* S, int row, const float* v, long long gi, long long gj0,
                                        bool any_masked, float* r) {
  if (any_masked) {
    int lo, hi;
    k.keep_range<W>(gi, gj0, gj0 + W, lo, hi);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const float old = S[j * 128 + row];
      r[j] = (j >= lo && j < hi) ? fmaf(k.beta, old, k.alpha * v[j]) : old;
    }
  } else {
#pragma unroll
    for (int j = 0; j < W; ++j) r[j] = fmaf(k.beta, S[j * 128 + row], k.alpha * v[j]);
  }
#pragma unroll
  for (int j = 0; j < W; ++j) S[j * 128 + row] = r[j];
}

// Scalars of the per-element store path for one tile (EpiK's fields plus C,
// bounds and the side-copy fields).
struct StoreK : EpiK {
  float* C;
  long long ldc, ld_out;
  int N, out_m, out_n;
  __half* out_hi;
  __half* out_lo;
  __device__ __forceinline__ explicit StoreK(const GemmArgs& a)
      : EpiK(a), C(a.C), ldc(a.ldc), ld_out(a.ld_out), N(a.N), out_m(a.out_m), out_n(a.out_n), out_hi(a.out_hi),
        out_lo(a.out_lo) {}
  // the side copies take 8-byte stores at rows that are multiples of 4
  __device__ __forceinline__ bool side_vec() const {
    return tri == 0 && ((reinterpret_cast<uintptr_t>(out_hi) | reinterpret_cast<uintptr_t>(out_lo)) & 7) == 0 &&
           (ld_out & 3) == 0;
  }
};

// Side copies of a staged 128 x 16 chunk S (fp32, column-major) at (m0, gj),
// written by the 128 threads of a group (t) after its values are in place:
// eight threads take 32 rows of a column, four rows each, so the copies leave
// as 8-byte stores. From the registers that hold a row of the chunk each value
// would be a 2-byte store of its own, 256 a thread and tile, with its address;
// that was most of a TRSM leaf product's epilogue.
__device__ __forceinline__ void copy_side16(const StoreK& k, const float* S, int t, int m0, int gj) {
  const int j = t >> 3, r0 = 4 * (t & 7);
  if (gj + j >= k.out_n) return;
  const long long at = (long long)m0 + r0 + (long long)(gj + j) * k.ld_out;
  __half* hi = k.out_hi + at;
  __half* lo = k.out_lo + at;  // used only when out_lo is set
  const bool has_lo = k.out_lo != nullptr;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = r0 + 32 * q;
    const float4 x = *reinterpret_cast<const float4*>(S + j * 128 + r);
    const __half2 a = __floats2half2_rn(x.x, x.y), b = __floats2half2_rn(x.z, x.w);
    const float2 fa = __half22float2(a), fb = __half22float2(b);
    const __half2 c = __floats2half2_rn((x.x - fa.x) * k.lo_scale, (x.y - fa.y) * k.lo_scale);
    const __half2 d = __floats2half2_rn((x.z - fb.x) * k.lo_scale, (x.w - fb.y) * k.lo_scale);
    if (m0 + r + 4 <= k.out_m) {
      *reinterpret_cast<uint2*>(hi + 32 * q) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
      if (has_lo)
        *reinterpret_cast<uint2*>(lo + 32 * q) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&c), *reinterpret_cast<const uint32_t*>(&d));
    } else {
      const __half h[4] = {__low2half(a), __high2half(a), __low2half(b), __high2half(b)};
      const __half l[4] = {__low2half(c), __high2half(c), __low2half(d), __high2half(d)};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (m0 + r + i < k.out_m) {
          hi[32 * q + i] = h[i];
          if (has_lo) lo[32 * q + i] = l[i];
        }
    }
  }
}

// Fused fp16 hi[/lo] copies of W result values of one row.
template <int W>
__device__ __forceinline__ void store_fp16_copies(const StoreK& s, const float* r, long long gi, long long gj0) {
  const long long ld = s.ld_out;
  __half* hrow = s.out_hi + gi + gj0 * ld;
  __half* lrow = s.out_lo ? s.out_lo + gi + gj0 * ld : nullptr;
  int lo, hi;
  s.keep_range<W>(gi, gj0, s.out_n, lo, hi);
#pragma unroll
  for (int j = 0; j < W; ++j) {
    if (j < lo || j >= hi) continue;
    const __half h = __float2half_rn(r[j]);
    hrow[(long long)j * ld] = h;
    if (lrow) lrow[(long long)j * ld] = __float2half_rn((r[j] - __half2float(h)) * s.lo_scale);
  }
}

// The old C values the per-element path needs for W consecutive columns of
// one row (zeros where nothing is read), all loads in flight together.
template <int W>
__device__ __forceinline__ void load_old(const StoreK& s, float* old, bool row_ok, long long gi, long long gj0) {
  int lo = 0, hi = 0;
  if (row_ok) s.keep_range<W>(gi, gj0, s.N, lo, hi);
  const float* crow = s.C + gi + gj0 * s.ldc;
#pragma unroll
  for (int j = 0; j < W; ++j) old[j] = (j >= lo && j < hi) ? __ldcg(crow + (long long)j * s.ldc) : 0.f;
}

// Per-element path: alpha/beta update of W consecutive columns of one row,
// with the triangle mask and bounds; old: load_old's values (read only when
// beta != 0); r: the new values.
template <int W>
__device__ __forceinline__ void epilogue_store(const StoreK& s, const float* v, const float* old, bool row_ok,
                                               long long gi, long long gj0, float* r) {
  const long long ldc = s.ldc;
  float* crow = s.C + gi + gj0 * ldc;
  int lo = 0, hi = 0;
  if (row_ok) s.keep_range<W>(gi, gj0, s.N, lo, hi);
  const bool has_beta = s.beta != 0.0f;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const float av = s.alpha * v[j];
    r[j] = has_beta ? fmaf(s.beta, old[j], av) : av;
  }
#pragma unroll
  for (int j = 0; j < W; ++j)
    if (j >= lo && j < hi) crow[(long long)j * ldc] = r[j];
}

// Columns [16 c, 16 c + 16) of a thread's register sums: registers cannot be
// indexed at run time, so one copy per chunk position (behind a branch: the
// asm keeps the compiler from turning all of them into predicated moves)
// keeps a single copy of the chunk code instead of one per chunk.
template <int N>
__device__ __forceinline__ void pick16(const float (&acc)[N], int c, float* v) {
#pragma unroll
  for (int q = 0; q < N / 16; ++q)
    if (c == q) {
#pragma unroll
      for (int j = 0; j < 16; ++j) asm volatile("mov.f32 %0, %1;" : "=f"(v[j]) : "f"(acc[16 * q + j]));
    }
}

// Whether a tile's chunks go through the C slots (TMA); the others are
// stored per element. Masked tiles with beta == 0 store their unmasked
// elements directly: the slots would first have to load C to keep the masked
// ones. TMA stores clip at 16 bytes, not at the element: the last row tile of
// a C whose M is no multiple of 4 is stored per element, or up to three rows
// past M would be overwritten.
__device__ __forceinline__ bool tile_staged(const GemmArgs& P, bool masked, int m0) {
  return P.tma_c && !(masked && P.beta == 0.0f) && ((P.M & 3) == 0 || m0 + 128 <= P.M);
}

// Whether a tile's chunks pass through the C slots at all: also per-element
// tiles that make side copies, which build them from the slot.
__device__ __forceinline__ bool tile_slots(const GemmArgs& P, bool masked, int m0) {
  return tile_staged(P, masked, m0) || (P.out_hi && !masked);
}

// The C loader's walk (one thread): the CTA's tiles in the epilogue's chunk
// order, the groups in turn; a group's chunk n goes to slot n % SLOTS of its
// ring once the epilogue has given back the slot's previous chunk
// (n - SLOTS). Chunks that are not loaded (beta == 0, per-element tiles) only
// pass the slot's barrier.
template <int SLOTS, int STRIDE>
struct CLoader {
  float* stage;  // group g's slots start at stage + g * STRIDE
  uint64_t *cfull, *cfree;
  int slot[kEpiGroups];
  uint32_t ph[kEpiGroups];
  uint32_t armed, armed_phase;  // per slot: a load was armed / its phase

  __device__ __forceinline__ CLoader(float* stage_, uint64_t* cfull_, uint64_t* cfree_)
      : stage(stage_), cfull(cfull_), cfree(cfree_), armed(0), armed_phase(0) {
    for (int g = 0; g < kEpiGroups; ++g) slot[g] = 0, ph[g] = 0;
  }
  // chunks of the tile at (m0, n0) with gc columns per group; false when a wait gave up
  __device__ __forceinline__ bool tile(const GemmArgs& P, int m0, int n0, int gc, bool masked,
                                       volatile int* abort_flag) {
    if (!tile_slots(P, masked, m0)) return true;
    const bool need = P.beta != 0.0f && tile_staged(P, masked, m0);
    for (int c0 = 0; c0 < gc; c0 += kEpiCols) {
#pragma unroll
      for (int g = 0; g < kEpiGroups; ++g) {
        const int gj = n0 + g * gc + c0;
        if (gj >= P.N) continue;
        const int s = g * SLOTS + slot[g];
        if (!mbar_wait(&cfree[s], ph[g] ^ 1u, abort_flag, P.err, kDevErrTimeoutProducer)) return false;
        if (need) {
          mbar_arrive_expect_tx(&cfull[s], 128 * kEpiCols * 4);
          tma_load_2d(stage + g * STRIDE + slot[g] * (128 * kEpiCols), &P.mapC, &cfull[s], m0, gj);
          armed |= 1u << s;
          armed_phase = (armed_phase & ~(1u << s)) | (ph[g] << s);
        } else {
          // the slot's earlier load was consumed before the slot came back
          armed &= ~(1u << s);
          mbar_arrive(&cfull[s]);
        }
        if (++slot[g] == SLOTS) {
          slot[g] = 0;
          ph[g] ^= 1u;
        }
      }
    }
    return true;
  }
  // every armed load lands before the CTA exits (immediate unless the
  // epilogue left early)
  __device__ __forceinline__ void drain(int* err) {
    for (int i = 0; i < kEpiGroups * SLOTS; ++i) {
      if (!((armed >> i) & 1u)) continue;
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(&cfull[i], (armed_phase >> i) & 1u))
        if (globaltimer_ns() - t0 > 1000000000ull) {
          if (err) atomicCAS(err, 0, kDevErrTimeoutTeardown);
          break;
        }
    }
  }
};

// One epilogue group of four warps (128 threads, named barrier `bar`).
template <int SLOTS>
struct EpiGroup {
  static constexpr bool kSlots = SLOTS > 0;
  float* slots;               // the group's ring of 128 x 16 chunks
  uint64_t *cfull, *cfree;    // per slot: chunk (or its hand-over) arrived / slot given back
  int bar, row;               // row: this thread's row of the tile
  bool issuer;
  int slot = 0;        // next ring slot
  uint32_t phase = 0;  // its barrier's phase (flips when the ring wraps)
  int prev = -1;       // slot of the previous chunk, still to be released (-1: none)

  // One 128 x 16 chunk at (m0, gj) through the next slot. Staged (TMA): the
  // slot holds this chunk of C when beta != 0; the result is combined in place
  // and stored from the slot. Otherwise (per-element C, old: its old values)
  // the result is stored from registers and left in the slot for the side
  // copies. The FP16 side copies are made from the slot after the barrier
  // that completes the chunk; the slot goes back to the loader at the next
  // chunk's barrier, when every thread has read it and its store has, too.
  // All 128 threads call it together; false, in every thread alike, when the
  // slot's wait gave up.
  __device__ __forceinline__ bool chunk_slot(const GemmArgs& P, const StoreK& k, bool staged, bool side_vec,
                                             bool row_ok, const float* v, const float* old, int m0, int gj,
                                             volatile int* abort_flag) {
    constexpr int W = kEpiCols;
    float* S = slots + slot * (128 * W);
    const bool got = mbar_wait(&cfull[slot], phase, abort_flag, P.err, kDevErrTimeoutEpilogue);
    const long long gi = (long long)m0 + row;
    float r[W];
    if (staged && k.beta != 0.0f) {
      combine<W>(k, S, row, v, gi, gj, k.chunk_masked<W>(m0, gj), r);
    } else {
      if (staged) {
#pragma unroll
        for (int j = 0; j < W; ++j) r[j] = k.alpha * v[j];
      } else {
        epilogue_store<W>(k, v, old, row_ok, gi, gj, r);
      }
#pragma unroll
      for (int j = 0; j < W; ++j) S[j * 128 + row] = r[j];
    }
    fence_proxy_async_smem();
    if (named_bar_any(bar, 128, !got)) return false;
    if (issuer) {
      bulk_wait_read<0>();  // the previous chunk's store has read its slot, and every thread is past it
      if (prev >= 0) mbar_arrive(&cfree[prev]);
      if (staged) {
        tma_store_2d(&P.mapC, S, m0, gj);
        bulk_commit();
      }
    }
    prev = slot;
    if (++slot == SLOTS) {
      slot = 0;
      phase ^= 1u;
    }
    if (k.out_hi && m0 < k.out_m && gj < k.out_n) {
      if (side_vec)
        copy_side16(k, S, threadIdx.x & 127, m0, gj);
      else if (gi < k.out_m)
        store_fp16_copies<W>(k, r, gi, gj);
    }
    return true;
  }
};

// The per-tile part of the epilogue. acc.begin() makes the group's
// accumulators ready (waits for the MMAs, folds) and returns false when a
// wait gave up; acc.chunk(c, v) gives columns [16 c, 16 c + 16) of the
// group's GC. (m0, gy): the group's first row and column of C. False when
// the epilogue has to stop.
template <int GC, class Group, class Acc>
__device__ __forceinline__ bool epilogue_tile(const GemmArgs& P, Group& g, Acc& acc, int m0, int gy, bool masked,
                                              volatile int* abort_flag) {
  const StoreK sk(P);
  const long long gi = (long long)m0 + g.row;
  const bool row_ok = gi < P.M;
  const int nval = min(max((sk.N - gy + kEpiCols - 1) / kEpiCols, 0), GC / kEpiCols);  // chunks inside C
  const bool side_vec = sk.side_vec();
  // kSlots false: no ring (launches that read no C and make no side copies)
  const bool staged = Group::kSlots && m0 < P.M && tile_staged(P, masked, m0);
  const bool through = Group::kSlots && m0 < P.M && tile_slots(P, masked, m0);
  // per-element path: C's old values are loaded one chunk ahead, the first
  // before the accumulator wait (where the fold leaves registers for it)
  float old[kEpiCols];
  const bool read_old = !staged && sk.beta != 0.0f;
  if (Acc::kEarlyLoad && read_old) load_old<kEpiCols>(sk, old, row_ok, gi, gy);
  if (named_bar_any(g.bar, 128, !acc.begin())) return false;
  if (!Acc::kEarlyLoad && read_old) load_old<kEpiCols>(sk, old, row_ok, gi, gy);
#pragma unroll 1
  for (int c = 0; c < GC / kEpiCols; ++c) {
    float v[kEpiCols];
    acc.chunk(c, v);
    if (c >= nval) continue;
    const int gj = gy + c * kEpiCols;
    if (through) {
      if (!g.chunk_slot(P, sk, staged, side_vec, row_ok, v, old, m0, gj, abort_flag)) return false;
    } else {
      float r[kEpiCols];
      epilogue_store<kEpiCols>(sk, v, old, row_ok, gi, gj, r);
      if (sk.out_hi && row_ok && gi < sk.out_m) store_fp16_copies<kEpiCols>(sk, r, gi, gj);
    }
    if (!staged) {
      if (read_old && c + 1 < nval) load_old<kEpiCols>(sk, old, row_ok, gi, gj + kEpiCols);
    }
  }
  return true;
}

// FP8: the block scales of a tile's rounds, one round ahead of their use (a
// load per round in the fold's path cost more than the round's MMAs).
struct Fp8Scales {
  const float *pa, *pb;
  float na = 0.f, nb = 0.f;
  // the scale rows of the 128-row block of A at C row m0 and of B at C column
  // n0; blocks wholly outside C take the last one (their products are not stored)
  __device__ __forceinline__ Fp8Scales(const GemmArgs& P, int m0, int n0, int kb0, int kb1) {
    const int ra = (P.a_off + min(m0, P.M - 1)) >> 7, rb = (P.b_off + min(n0, P.N - 1)) >> 7;
    pa = P.scale_a + (long long)ra * P.scale_ld + (P.k_off >> 7);
    pb = P.scale_b + (long long)rb * P.scale_ld + (P.k_off >> 7);
    if (kb0 < kb1) {
      na = __ldg(pa + kb0);
      nb = __ldg(pb + kb0);
    }
  }
  __device__ __forceinline__ float next(int kb, int kb1) {
    const float s = na * nb;
    if (kb + 1 < kb1) {
      na = __ldg(pa + kb + 1);
      nb = __ldg(pb + kb + 1);
    }
    return s;
  }
};

// Accumulators of one tile in the single-CTA kernel, as an epilogue group's
// warp sees them (tmem: base + lane quarter + the group's first column).
template <class Cfg>
struct TileAcc {
  static constexpr bool kEarlyLoad = true;
  const GemmArgs& args;
  const GemmArgs& P;
  int4 tile;
  int gc0;
  uint32_t tmem;
  uint64_t *tfull, *tempty, *xempty;
  int &it, &nt;
  volatile int* abort_flag;
  float acc[Cfg::FOLD ? Cfg::GC : 16];
  int buf = 0;
  uint32_t folded = 0;  // split: TMEM columns of the folded tile

  __device__ __forceinline__ void release(uint64_t* bar) {
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
  }
  __device__ __forceinline__ bool round() {
    buf = it & 1;
    const uint32_t ph = (uint32_t)(it >> 1) & 1u;
    ++it;
    const bool got = mbar_wait(&tfull[buf], ph, abort_flag, args.err, kDevErrTimeoutEpilogue);
    tc_fence_after();
    return __all_sync(0xffffffffu, got);  // one decision per warp: TMEM loads follow
  }
  __device__ __forceinline__ bool begin() {
    if constexpr (!Cfg::FOLD) {
      return round();
    } else {
#pragma unroll
      for (int j = 0; j < Cfg::GC; ++j) acc[j] = 0.f;
      if constexpr (Cfg::FP8) {
        Fp8Scales sc(P, tile.x, tile.y + gc0, tile.z, tile.w);
        for (int kb = tile.z; kb < tile.w; ++kb) {  // kchunk = 1
          const float s = sc.next(kb, tile.w);
          if (!round()) return false;
          const uint32_t ta = tmem + (uint32_t)(buf * Cfg::BN);
          tmem_for32<Cfg::GC>(ta, [&](int c0, const float* v) {
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c0 + j] = fmaf(s, v[j], acc[c0 + j]);
          });
          release(&tempty[buf]);
        }
      } else {
        // one round's main sums
        auto fold_round = [&]() {
          if (!round()) return false;
          tmem_for32<Cfg::GC>(tmem + (uint32_t)(buf * Cfg::BN), [&](int c0, const float* v) {
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c0 + j] += v[j];
          });
          release(&tempty[buf]);
          return true;
        };
        // the correction (the last round's commit covers its MMAs) with the
        // main sums, in its place
        auto fold_stretch = [&]() {
          const uint32_t tc = tmem + (uint32_t)(Cfg::CORR_COL + (nt & 1) * Cfg::BN);
#pragma unroll
          for (int c0 = 0; c0 < Cfg::GC; c0 += 32) {
            float w[32];
            tmem_ld32(tc + c0, w);
#pragma unroll
            for (int j = 0; j < 32; ++j) w[j] = fmaf(args.corr_scale, w[j], acc[c0 + j]);
            tmem_st32(tc + c0, w);
          }
          tmem_st_wait();
          folded = tc;
        };
        // Stretches before the last. On 64-column tiles, whose short launches
        // are bound by fetching their code, the same fold serves them and its
        // sums are read back (TRSM 4096 x 256 0.5 to 2 % faster than with a
        // copy of it); the wider tiles' registers do not allow that.
        if constexpr (Cfg::GC == 32) {
          for (int c0k = tile.z; c0k < tile.w;) {
            const int cend = min(tile.w, c0k + kCorrRounds * args.kchunk);
            for (; c0k < cend; c0k += args.kchunk)
              if (!fold_round()) return false;
            fold_stretch();
            if (c0k < tile.w) {
              tmem_ld32(folded, acc);
              release(&xempty[nt & 1]);
              ++nt;
            }
          }
        } else {
          int left = kCorrRounds;
          for (int c0k = tile.z; c0k < tile.w; c0k += args.kchunk) {
            if (!fold_round()) return false;
            if (--left == 0 && tile.w - c0k > args.kchunk) {
              tmem_for32<Cfg::GC>(tmem + (uint32_t)(Cfg::CORR_COL + (nt & 1) * Cfg::BN), [&](int c0, const float* w) {
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[c0 + j] = fmaf(args.corr_scale, w[j], acc[c0 + j]);
              });
              release(&xempty[nt & 1]);
              ++nt;
              left = kCorrRounds;
            }
          }
          if (tile.z < tile.w) fold_stretch();
        }
      }
      return true;
    }
  }
  __device__ __forceinline__ void chunk(int c, float* v) {
    if constexpr (Cfg::FP8) {
      pick16(acc, c, v);
    } else if constexpr (Cfg::SPLIT) {
      if (tile.z < tile.w) {
        tmem_ld16(folded + (uint32_t)(c * kEpiCols), v);
        if (c == Cfg::GC / kEpiCols - 1) {
          release(&xempty[nt & 1]);
          ++nt;
        }
      } else {
#pragma unroll
        for (int j = 0; j < kEpiCols; ++j) v[j] = 0.f;
      }
    } else {
      tmem_ld16(tmem + (uint32_t)(buf * Cfg::BN + c * kEpiCols), v);
      if (c == Cfg::GC / kEpiCols - 1) release(&tempty[buf]);  // fully read: hand it back to the MMA warp
    }
  }
};

template <class Cfg, bool GROUPED>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_kernel(const __grid_constant__ GemmArgs args) {
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, STAGES = Cfg::STAGES;
  constexpr int kSlots = kEpiGroups * Cfg::C_SLOTS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* stage_c = reinterpret_cast<float*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES + Cfg::EPI_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;    // [2] main accumulator rounds
  uint64_t* tempty = tfull + 2;        // [2]
  uint64_t* xempty = tempty + 2;       // [2] correction accumulators given back
  uint64_t* drain = xempty + 2;        // [1] teardown barrier for the MMA issuer
  uint64_t* cfull = drain + 1;         // [group][C_SLOTS] C chunks of the loader's ring
  uint64_t* cfree = cfull + kSlots;    // [group][C_SLOTS] ring slots the epilogue gave back
  uint64_t* tq_full = cfree + kSlots;  // [kTileQ] tile hand-off (device-side scheduler)
  uint64_t* tq_empty = tq_full + kTileQ;     // [kTileQ]
  int* tq_idx = reinterpret_cast<int*>(tq_empty + kTileQ);  // [kTileQ]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tq_idx + kTileQ);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 4 * kEpiGroups);
      mbar_init(&xempty[b], 4 * kEpiGroups);
    }
    for (int b = 0; b < kSlots; ++b) {
      mbar_init(&cfull[b], 1);
      mbar_init(&cfree[b], 1);
    }
    for (int b = 0; b < kTileQ; ++b) {
      mbar_init(&tq_full[b], 1);
      mbar_init(&tq_empty[b], 2 + 4 * kEpiGroups);  // MMA issuer, C loader, epilogue warps
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (!GROUPED && warp == 0 && lane == 0) {
    tma_prefetch_map(&args.mapA[0]);
    tma_prefetch_map(&args.mapB[0]);
    if (Cfg::NSPLIT > 1) {
      tma_prefetch_map(&args.mapA[1]);
      tma_prefetch_map(&args.mapB[1]);
    }
    if (args.tma_c) tma_prefetch_map(&args.mapC);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // the set-up above touches no global memory and may overlap the previous
  // launch's last tiles (programmatic dependent launch)
  grid_dep_wait();
  grid_dep_launch();

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      uint32_t issued_mask = 0, phase_mask = 0;  // per-stage: copy issued / its phase
      bool ok = true;
      const bool dyn = args.sched != nullptr;
      int tq = 0;
      uint32_t tq_ph = 0;
      int t = dyn ? atomicAdd(args.sched, 1) : static_first(args, blockIdx.x);
      while (ok) {
        if (t >= args.num_tiles) t = -1;
        if (dyn) {
          // hand the tile (or the end mark) to the other roles
          if (!mbar_wait(&tq_empty[tq], tq_ph ^ 1u, abort_flag, args.err, kDevErrTimeoutProducer)) {
            ok = false;
            break;
          }
          tq_idx[tq] = t;
          mbar_arrive(&tq_full[tq]);
          if (++tq == kTileQ) {
            tq = 0;
            tq_ph ^= 1u;
          }
        }
        if (t < 0) break;
        if (debug_stall_tile(args.err, t)) break;  // test hook: this tile's loads never come
        // the next claim is issued early so its latency hides
        const int t_next = dyn ? atomicAdd(args.sched, 1) : static_next(args, blockIdx.x, gridDim.x, t);
        const int4 tile = args.tiles[t];
        for (int kb = tile.z; kb < tile.w; ++kb) {
          if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag, args.err, kDevErrTimeoutProducer)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&full[s], Cfg::STAGE_BYTES);
          uint8_t* st = smem + s * Cfg::STAGE_BYTES;
          const GemmArgs& P = tile_problem<GROUPED>(args, t);
          const int k = P.k_off + kb * BK;
#pragma unroll
          for (int h = 0; h < Cfg::NOPS; ++h) {
            load_operand<Cfg::A_MN, BM>(st + h * Cfg::A_BYTES, &P.mapA[h], &full[s], P.a_off + tile.x, k);
            load_operand<Cfg::B_MN, BN>(st + Cfg::NOPS * Cfg::A_BYTES + h * Cfg::B_BYTES, &P.mapB[h], &full[s],
                                        P.b_off + tile.y, k);
          }
          issued_mask |= 1u << s;
          phase_mask = (phase_mask & ~(1u << s)) | (ph << s);
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
        t = t_next;
      }
      if (!ok) {
        // Abort path: let every copy in flight land before the CTA exits.
        for (int i = 0; i < STAGES; ++i) {
          if (!((issued_mask >> i) & 1u)) continue;
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(&full[i], (phase_mask >> i) & 1u)) {
            if (globaltimer_ns() - t0 > 1000000000ull) {
              if (args.err) atomicCAS(args.err, 0, kDevErrTimeoutTeardown);
              break;
            }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // Main accumulation in rounds, one TMEM buffer each: plain mode runs a
    // tile's whole K range in one round; split mode closes a round every
    // `kchunk` K-blocks and FP8 every K-block. Split mode's correction
    // products go to an accumulator of their own for kCorrRounds rounds.
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int it = 0;  // round counter (selects the main buffer and its phase)
      int nt = 0;  // stretch counter (selects the correction buffer and its phase)
      bool ok = true;
      bool any = false;
      const int kc = Cfg::FOLD ? args.kchunk : (1 << 30);
      int tq = 0;
      uint32_t tq_ph = 0;
      for (int t = next_tile<false>(args, -1, tq_idx, tq_full, tq_empty, tq, tq_ph, abort_flag, kDevErrTimeoutMma);
           t >= 0 && ok;
           t = next_tile<false>(args, t, tq_idx, tq_full, tq_empty, tq, tq_ph, abort_flag, kDevErrTimeoutMma)) {
        const int4 tile = args.tiles[t];
        uint32_t x0 = 0;
        int xkb = 0, left = 0;  // the correction's stretch: first K-block, rounds left
        for (int c0 = tile.z; c0 < tile.w && ok; c0 += kc, ++it) {
          const int c1 = (tile.w - c0 > kc) ? c0 + kc : tile.w;
          if (Cfg::SPLIT && --left < 0) {
            if (!mbar_wait(&xempty[nt & 1], ((uint32_t)(nt >> 1) & 1u) ^ 1u, abort_flag, args.err,
                           kDevErrTimeoutMma)) {
              ok = false;
              break;
            }
            x0 = tmem_base + (uint32_t)(Cfg::CORR_COL + (nt & 1) * BN);
            xkb = c0;
            left = kCorrRounds - 1;
            ++nt;
          }
          const int buf = it & 1;
          const uint32_t tph = (uint32_t)(it >> 1) & 1u;
          if (!mbar_wait(&tempty[buf], tph ^ 1u, abort_flag, args.err, kDevErrTimeoutMma)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d0 = tmem_base + (uint32_t)(buf * BN);
          for (int kb = c0; kb < c1; ++kb) {
            if (!mbar_wait(&full[s], ph, abort_flag, args.err, kDevErrTimeoutMma)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t st = smem_u32(smem + s * Cfg::STAGE_BYTES);
            const uint32_t a_hi = st, b_hi = st + Cfg::NOPS * Cfg::A_BYTES;
#pragma unroll
            for (int kk = 0; kk < Cfg::KSTEPS; ++kk) {
              const uint32_t acc = (kb > c0 || kk > 0) ? 1u : 0u;
              const uint64_t da = operand_desc<Cfg::A_MN>(a_hi, kk);
              const uint64_t db = operand_desc<Cfg::B_MN>(b_hi, kk);
              if constexpr (Cfg::FP8)
                umma_f8(d0, da, db, Cfg::IDESC, acc);
              else
                umma_f16(d0, da, db, Cfg::IDESC, acc);
              if constexpr (Cfg::SPLIT) {
                const uint64_t da_lo = operand_desc<Cfg::A_MN>(a_hi + Cfg::A_BYTES, kk);
                const uint64_t db_lo = operand_desc<Cfg::B_MN>(b_hi + Cfg::B_BYTES, kk);
                umma_f16(x0, da, db_lo, Cfg::IDESC, (kb > xkb || kk > 0) ? 1u : 0u);
                umma_f16(x0, da_lo, db, Cfg::IDESC, 1u);
              }
            }
            any = true;
            tc_commit(&empty[s]);
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
          if (!ok) break;
          tc_commit(&tfull[buf]);
        }
      }
      if (!ok && any) {
        // Abort path: wait (bounded) until every issued MMA has retired.
        tc_commit(drain);
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(drain, 0)) {
          if (globaltimer_ns() - t0 > 1000000000ull) {
            if (args.err) atomicCAS(args.err, 0, kDevErrTimeoutTeardown);
            break;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------ C loader
    if (lane == 0) {
      CLoader<Cfg::C_SLOTS, Cfg::GROUP_BYTES / 4> ld(stage_c, cfull, cfree);
      bool ok = true;
      int tq = 0;
      uint32_t tq_ph = 0;
      for (int t = next_tile<false>(args, -1, tq_idx, tq_full, tq_empty, tq, tq_ph, abort_flag,
                                    kDevErrTimeoutProducer);
           t >= 0 && ok;
           t = next_tile<false>(args, t, tq_idx, tq_full, tq_empty, tq, tq_ph, abort_flag, kDevErrTimeoutProducer)) {
        const int4 tile = args.tiles[t];
        const GemmArgs& P = tile_problem<GROUPED>(args, t);
        ok = ld.tile(P, tile.x, tile.y, Cfg::GC, tile_reaches_mask(P, tile.x, tile.y, BM, BN), abort_flag);
      }
      ld.drain(args.err);
    }
    __syncwarp();
  } else if (warp >= kEpiWarp0) {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3;  // TMEM lane quarter this warp may access
    const int group = (warp - kEpiWarp0) >> 2, gc0 = group * Cfg::GC;
    const uint32_t tmem = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)gc0;
    EpiGroup<Cfg::C_SLOTS> g{stage_c + group * (Cfg::GROUP_BYTES / 4), cfull + group * Cfg::C_SLOTS,
                             cfree + group * Cfg::C_SLOTS, 1 + group, quarter * 32 + lane,
                             quarter == 0 && lane == 0};
    int it = 0, nt = 0;
    int tq = 0;
    uint32_t tq_ph = 0;
    for (int t = next_tile<true>(args, -1, tq_idx, tq_full, tq_empty, tq, tq_ph, abort_flag, kDevErrTimeoutEpilogue,
                                 g.bar);
         t >= 0; t = next_tile<true>(args, t, tq_idx, tq_full, tq_empty, tq, tq_ph, abort_flag,
                                     kDevErrTimeoutEpilogue, g.bar)) {
      const int4 tile = args.tiles[t];
      const GemmArgs& P = tile_problem<GROUPED>(args, t);
      TileAcc<Cfg> acc{args, P, tile, gc0, tmem, tfull, tempty, xempty, it, nt, abort_flag};
      if (!epilogue_tile<Cfg::GC>(P, g, acc, tile.x, tile.y + gc0, tile_reaches_mask(P, tile.x, tile.y, BM, BN),
                                  abort_flag))
        break;
    }
    if (g.issuer) bulk_wait<0>();  // all TMA stores complete before the CTA retires
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

// ---------------------------------------------------------------------------
// Pair variant: a cluster of two CTAs computes 256 x 256 output tiles with
// tcgen05.mma.cta_group::2. CTA r of the pair loads rows [m0 + 128r, +128) of
// A and rows [n0 + 128r, +128) of B (half of the tile's columns) into its own
// shared memory; the leader (r = 0) issues the 256-row MMA, which reads both
// CTAs' halves, and each CTA's TMEM receives its 128 accumulator rows. Per SM,
// one 64-deep K slab moves 32 KB from L2 instead of the single-CTA tile's
// 48 KB for the same MMA work.
//   full[s]   leader only: both CTAs' loads complete_tx on it, the leader's
//             producer arms it with both CTAs' bytes;
//   empty[s]  both CTAs: the leader's commit multicasts to the pair;
//   tfull[b]  both CTAs: the leader's commit multicasts to the pair;
//   tempty[b] leader only: the 16 epilogue warps of the pair arrive remotely.
// Every wait is bounded like the single-CTA kernel's; a cluster barrier
// before TMEM is freed keeps either CTA from leaving while the pair's MMAs
// or remote arrivals may still touch it.
//
// kDirect: launches that read no C and write no side copies (beta = 0, e.g.
// SYRK) store each thread's row of a chunk straight from registers (a warp's
// 32 rows of one column are one 128-byte line), which frees the C slots for
// more operand stages. kStaged: the others, with a ring of C slots.
// kSplit: hi/lo operands, three products (64 KB a stage). Main and correction
// accumulators take all 512 TMEM columns, so nothing is double-buffered;
// instead each K-block runs its four main MMAs before its eight correction
// MMAs: while a round's last correction MMAs run (1024 cycles per SM), the
// epilogue reads the main accumulator, and the next round's main MMAs find it
// free. Buffer 0 is the main accumulator (one phase a round), buffer 1 the
// correction (one phase a stretch of kCorrRounds). Per 64-deep K block and SM the 256 x 256 tile
// moves 64 KB into shared memory and 96 KB out of it for 1536 MMA cycles,
// where 256 x 128 tiles (which left room to double-buffer) moved 96 + 144 KB.
// The tensor pipe is 93 % busy while the SM is active against 65 %: SYR2K n =
// 16384, k = 4096 went from 6.0 to 5.3 ms.
// kFp8: e4m3 operands, one 128-deep K block a round (512 MMA cycles per SM),
// the accumulators double-buffered and folded with the blocks' scales. The
// path of a round's signals (commit, fold, release, next MMAs) bounds it: a
// round takes about 1350 cycles, the tensor pipe is 38 % busy. Single-CTA 128 x
// 128 tiles have 256 MMA cycles a round and nearly as long a path for a quarter
// of the work a pair does: SYMM 16384 went from 8.8 to 6.6 ms.
// The fold modes keep 128 sums per epilogue thread: the first four warps give
// registers to the epilogue's eight (setmaxnreg: 128 x 72 + 256 x 216 = 384 x
// 168, the launch's allocation).
enum class PairMode { kStaged, kDirect, kSplit, kFp8 };

template <bool A_MN_, bool B_MN_, PairMode MODE_>
struct PairCfg {
  static constexpr PairMode MODE = MODE_;
  static constexpr bool SPLIT = MODE == PairMode::kSplit, FP8 = MODE == PairMode::kFp8;
  static constexpr bool FOLD = SPLIT || FP8, DIRECT = MODE == PairMode::kDirect;
  static constexpr int NOPS = SPLIT ? 2 : 1;  // copies per operand (hi[, lo])
  static constexpr int ELEM = FP8 ? 1 : 2;
  static constexpr int BM = 128, BN = 256, BK = 128 / ELEM;  // BM: rows per CTA; BN: the pair tile's columns
  static constexpr bool A_MN = A_MN_, B_MN = B_MN_;
  static constexpr int A_BYTES = BM * BK * ELEM;
  static constexpr int B_BYTES = (BN / 2) * BK * ELEM;
  static constexpr int STAGE_BYTES = NOPS * (A_BYTES + B_BYTES);
  static constexpr int STAGES = SPLIT ? 3 : (FP8 ? 6 : (DIRECT ? 7 : 5));
  static constexpr int TMEM_COLS = 512;
  static constexpr int GC = BN / kEpiGroups;
  static constexpr int CHUNK_BYTES = 128 * kEpiCols * 4;
  static constexpr int C_SLOTS = DIRECT ? 0 : (FOLD ? 2 : 4);  // per group
  static constexpr int GROUP_BYTES = C_SLOTS * CHUNK_BYTES;
  static constexpr int EPI_BYTES = kEpiGroups * GROUP_BYTES;
  static constexpr int BAR_BYTES = 320;
  static_assert(8 * (2 * STAGES + 5 + 2 * kEpiGroups * C_SLOTS) + 8 <= BAR_BYTES, "barrier space");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 + BAR_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  static constexpr uint32_t IDESC = idesc_f16(2 * BM, BN, false, A_MN, B_MN);
};

template <bool MN, int ROWS>
__device__ __forceinline__ void load_operand_pair(uint8_t* dst, const CUtensorMap* map, uint32_t leader_bar, int row0,
                                                  int k) {
  if constexpr (MN) {
#pragma unroll
    for (int j = 0; j < ROWS / 64; ++j) tma_load_2d_pair(dst + j * 8192, map, leader_bar, row0 + 64 * j, k);
  } else {
    tma_load_2d_pair(dst, map, leader_bar, k, row0);
  }
}

// Accumulators of one pair tile, as an epilogue warp of CTA `rank` sees them.
template <class Cfg>
struct PairAcc {
  static constexpr bool kEarlyLoad = !Cfg::FOLD;
  const GemmArgs& args;
  int4 tile;
  int m0, gc0;
  uint32_t tmem;
  uint64_t* tfull;
  uint32_t tempty_leader;
  int &it, &nt;
  volatile int* abort_flag;
  float acc[Cfg::FOLD ? Cfg::GC : 16];
  int buf = 0;

  __device__ __forceinline__ bool wait(int b, uint32_t ph) {
    const bool got = mbar_wait(&tfull[b], ph, abort_flag, args.err, kDevErrTimeoutEpilogue);
    tc_fence_after();
    return __all_sync(0xffffffffu, got);  // one decision per warp: TMEM loads follow
  }
  // this CTA's warp has read its part of buffer b: tell the leader
  __device__ __forceinline__ void release(int b) {
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive_cluster(tempty_leader + 8u * (uint32_t)b);
  }
  __device__ __forceinline__ bool begin() {
    if constexpr (!Cfg::FOLD) {
      buf = it & 1;
      const uint32_t ph = (uint32_t)(it >> 1) & 1u;
      ++it;
      return wait(buf, ph);
    } else {
#pragma unroll
      for (int j = 0; j < Cfg::GC; ++j) acc[j] = 0.f;
      if constexpr (Cfg::FP8) {
        Fp8Scales sc(args, m0, tile.y + gc0, tile.z, tile.w);
        for (int kb = tile.z; kb < tile.w; ++kb, ++it) {
          const float s = sc.next(kb, tile.w);
          const int b = it & 1;
          if (!wait(b, (uint32_t)(it >> 1) & 1u)) return false;
          const uint32_t ta = tmem + (uint32_t)(b * Cfg::BN);
          if (!(s < 0.f))  // negative: a block outside a triangle, all zeros
            tmem_for32<Cfg::GC>(ta, [&](int c0, const float* v) {
#pragma unroll
              for (int j = 0; j < 32; ++j) acc[c0 + j] = fmaf(s, v[j], acc[c0 + j]);
            });
          release(b);
        }
      } else {
        int left = kCorrRounds;  // rounds up to the end of the correction's stretch
        for (int c0k = tile.z; c0k < tile.w; c0k += args.kchunk, ++it) {
          if (!wait(0, (uint32_t)it & 1u)) return false;
          tmem_for32<Cfg::GC>(tmem, [&](int c0, const float* v) {
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c0 + j] += v[j];
          });
          release(0);
          if (--left == 0 || tile.w - c0k <= args.kchunk) {
            if (!wait(1, (uint32_t)nt & 1u)) return false;
            tmem_for32<Cfg::GC>(tmem + Cfg::BN, [&](int c0, const float* w) {
#pragma unroll
              for (int j = 0; j < 32; ++j) acc[c0 + j] = fmaf(args.corr_scale, w[j], acc[c0 + j]);
            });
            release(1);
            ++nt;
            left = kCorrRounds;
          }
        }
      }
      return true;
    }
  }
  __device__ __forceinline__ void chunk(int c, float* v) {
    if constexpr (Cfg::FOLD) {
      pick16(acc, c, v);
    } else {
      tmem_ld16(tmem + (uint32_t)(buf * Cfg::BN + c * kEpiCols), v);
      if (c == Cfg::GC / kEpiCols - 1) release(buf);
    }
  }
};

template <class Cfg>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
    gemm_pair_kernel(const __grid_constant__ GemmArgs args) {
  constexpr int BN = Cfg::BN, BK = Cfg::BK, STAGES = Cfg::STAGES;
  constexpr int kSlots = kEpiGroups * Cfg::C_SLOTS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* stage_c = reinterpret_cast<float*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES + Cfg::EPI_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;  // [2]
  uint64_t* tempty = tfull + 2;      // [2]
  uint64_t* drain = tempty + 2;      // [1]
  uint64_t* cfull = drain + 1;       // [group][C_SLOTS]
  uint64_t* cfree = cfull + kSlots;  // [group][C_SLOTS]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cfree + kSlots);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 2 * 4 * kEpiGroups);
    }
    for (int b = 0; b < kSlots; ++b) {
      mbar_init(&cfull[b], 1);
      mbar_init(&cfree[b], 1);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_map(&args.mapA[0]);
    tma_prefetch_map(&args.mapB[0]);
    if (Cfg::NOPS > 1) {
      tma_prefetch_map(&args.mapA[1]);
      tma_prefetch_map(&args.mapB[1]);
    }
    if (args.tma_c) tma_prefetch_map(&args.mapC);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before any remote arrival
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_wait();  // as in gemm_kernel
  grid_dep_launch();
  const uint32_t full_leader = mapa_shared(smem_u32(full), 0);
  const uint32_t tempty_leader = mapa_shared(smem_u32(tempty), 0);

  if (warp < kEpiWarp0) {
    if constexpr (Cfg::FOLD) setmaxnreg_dec<72>();
    if (warp == 0) {
      // ---------------------------------------------------------- producers (both CTAs)
      if (lane == 0) {
        int s = 0;
        uint32_t ph = 0;
        uint32_t issued_mask = 0, phase_mask = 0;
        bool ok = true;
        for (int t = static_first(args, pair); t >= 0 && ok; t = static_next(args, pair, npairs, t)) {
          if (debug_stall_tile(args.err, t)) break;  // test hook: this tile's loads never come
          const int4 tile = args.tiles[t];
          for (int kb = tile.z; kb < tile.w; ++kb) {
            if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag, args.err, kDevErrTimeoutProducer)) {
              ok = false;
              break;
            }
            if (leader) mbar_arrive_expect_tx(&full[s], 2 * Cfg::STAGE_BYTES);
            uint8_t* st = smem + s * Cfg::STAGE_BYTES;
            const int k = args.k_off + kb * BK;
            const uint32_t bar = full_leader + 8u * (uint32_t)s;
#pragma unroll
            for (int h = 0; h < Cfg::NOPS; ++h) {
              load_operand_pair<Cfg::A_MN, 128>(st + h * Cfg::A_BYTES, &args.mapA[h], bar,
                                                args.a_off + tile.x + 128 * (int)rank, k);
              load_operand_pair<Cfg::B_MN, BN / 2>(st + Cfg::NOPS * Cfg::A_BYTES + h * Cfg::B_BYTES, &args.mapB[h],
                                                   bar, args.b_off + tile.y + (BN / 2) * (int)rank, k);
            }
            issued_mask |= 1u << s;
            phase_mask = (phase_mask & ~(1u << s)) | (ph << s);
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        if (!ok) {
          // Abort path: the leader sees its loads land on its own barriers; the
          // peer's loads report to the leader, so the peer waits a bounded time.
          if (leader) {
            for (int i = 0; i < STAGES; ++i) {
              if (!((issued_mask >> i) & 1u)) continue;
              const uint64_t t0 = globaltimer_ns();
              while (!mbar_try_wait(&full[i], (phase_mask >> i) & 1u))
                if (globaltimer_ns() - t0 > 1000000000ull) break;
            }
          } else {
            const uint64_t t0 = globaltimer_ns();
            while (globaltimer_ns() - t0 < 2000000ull) {
            }
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------------------------------------------------- MMA issuer (leader)
      if (leader && lane == 0) {
        int s = 0;
        uint32_t ph = 0;
        int it = 0, nt = 0;  // rounds and (split) stretches: buffers and phases, as in gemm_kernel
        bool ok = true, any = false;
        const int kc = Cfg::FOLD ? args.kchunk : (1 << 30);
        for (int t = static_first(args, pair); t >= 0 && ok; t = static_next(args, pair, npairs, t)) {
          const int4 tile = args.tiles[t];
          int xkb = tile.z, left = kCorrRounds;  // split: the correction's stretch, as in gemm_kernel
          for (int c0 = tile.z; c0 < tile.w && ok; c0 += kc, ++it) {
            const int c1 = (tile.w - c0 > kc) ? c0 + kc : tile.w;
            const int buf = Cfg::SPLIT ? 0 : (it & 1);
            const uint32_t tph = (uint32_t)(Cfg::SPLIT ? it : (it >> 1)) & 1u;
            if (!mbar_wait(&tempty[buf], tph ^ 1u, abort_flag, args.err, kDevErrTimeoutMma)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t d0 = tmem_base + (uint32_t)(buf * BN);
            for (int kb = c0; kb < c1; ++kb) {
              if (!mbar_wait(&full[s], ph, abort_flag, args.err, kDevErrTimeoutMma)) {
                ok = false;
                break;
              }
              tc_fence_after();
              const uint32_t a = smem_u32(smem + s * Cfg::STAGE_BYTES), b = a + Cfg::NOPS * Cfg::A_BYTES;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                const uint32_t acc = (kb > c0 || kk > 0) ? 1u : 0u;
                const uint64_t da = operand_desc<Cfg::A_MN>(a, kk), db = operand_desc<Cfg::B_MN>(b, kk);
                if constexpr (Cfg::FP8)
                  umma_f8_pair(d0, da, db, Cfg::IDESC, acc);
                else
                  umma_f16_pair(d0, da, db, Cfg::IDESC, acc);
              }
              any = true;
              if constexpr (Cfg::SPLIT) {
                if (kb == c1 - 1) tc_commit_pair(&tfull[0], 3);  // the round's main products are issued
                if (kb == xkb) {
                  if (!mbar_wait(&tempty[1], ((uint32_t)nt & 1u) ^ 1u, abort_flag, args.err, kDevErrTimeoutMma)) {
                    ok = false;
                    break;
                  }
                  tc_fence_after();
                }
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                  const uint64_t da = operand_desc<Cfg::A_MN>(a, kk), db = operand_desc<Cfg::B_MN>(b, kk);
                  umma_f16_pair(d0 + BN, da, operand_desc<Cfg::B_MN>(b + Cfg::B_BYTES, kk), Cfg::IDESC,
                                (kb > xkb || kk > 0) ? 1u : 0u);
                  umma_f16_pair(d0 + BN, operand_desc<Cfg::A_MN>(a + Cfg::A_BYTES, kk), db, Cfg::IDESC, 1u);
                }
              }
              tc_commit_pair(&empty[s], 3);
              if (++s == STAGES) {
                s = 0;
                ph ^= 1u;
              }
            }
            if (!ok) break;
            if constexpr (Cfg::SPLIT) {
              if (--left == 0 || c1 == tile.w) {
                tc_commit_pair(&tfull[1], 3);  // the stretch's correction products are issued
                ++nt;
                xkb = c1;
                left = kCorrRounds;
              }
            } else {
              tc_commit_pair(&tfull[buf], 3);
            }
          }
        }
        if (!ok && any) {
          tc_commit_pair(drain, 1);
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(drain, 0)) {
            if (globaltimer_ns() - t0 > 1000000000ull) {
              if (args.err) atomicCAS(args.err, 0, kDevErrTimeoutTeardown);
              break;
            }
          }
        }
      }
      __syncwarp();
    } else if (!Cfg::DIRECT && warp == 2) {
      // ---------------------------------------------------------- C loader (both CTAs)
      if constexpr (!Cfg::DIRECT) {
        if (lane == 0) {
          CLoader<Cfg::C_SLOTS, Cfg::GROUP_BYTES / 4> ld(stage_c, cfull, cfree);
          bool ok = true;
          for (int t = static_first(args, pair); t >= 0 && ok; t = static_next(args, pair, npairs, t)) {
            const int4 tile = args.tiles[t];
            const int m0 = tile.x + 128 * (int)rank;
            if (m0 < args.M)  // rows wholly outside C are stored by no one
              ok = ld.tile(args, m0, tile.y, Cfg::GC, tile_reaches_mask(args, m0, tile.y, 128, BN), abort_flag);
          }
          ld.drain(args.err);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs)
    if constexpr (Cfg::FOLD) setmaxnreg_inc<216>();
    const int quarter = warp & 3;
    const int group = (warp - kEpiWarp0) >> 2, gc0 = group * Cfg::GC;
    const uint32_t tmem = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)gc0;
    EpiGroup<Cfg::C_SLOTS> g{stage_c + group * (Cfg::GROUP_BYTES / 4), cfull + group * Cfg::C_SLOTS,
                             cfree + group * Cfg::C_SLOTS, 1 + group, quarter * 32 + lane,
                             quarter == 0 && lane == 0};
    int it = 0, nt = 0;
    for (int t = static_first(args, pair); t >= 0; t = static_next(args, pair, npairs, t)) {
      const int4 tile = args.tiles[t];
      const int m0 = tile.x + 128 * (int)rank;
      PairAcc<Cfg> acc{args, tile, m0, gc0, tmem, tfull, tempty_leader, it, nt, abort_flag};
      if (!epilogue_tile<Cfg::GC>(args, g, acc, m0, tile.y + gc0, tile_reaches_mask(args, m0, tile.y, 128, BN),
                                  abort_flag))
        break;
    }
    if (g.issuer) bulk_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the pair's MMAs, remote arrivals and TMEM reads are over
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
}

}  // namespace tb
