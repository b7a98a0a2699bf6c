// TRSM driver (reference: BLAS/tc_trsm.cu:31-174, tc_cumpsgemm_trsm.cu).
//
// Method (the reference's): recursive halving of the triangular operand.
// A node [s, e) solves its left half, applies the off-diagonal update
//   right side  B[:, mid:e] -= X[:, s:mid] * A[mid:e, s:mid]^T
//   left side   B[mid:e, :] -= A[mid:e, s:mid] * X[s:mid, :]
// as one FP16-operand / FP32-accumulate tensor-core GEMM, then solves its
// right half. Leaves are diagonal blocks of nb (<= 512) columns.
//
// B200 form of the pieces:
//  * A is converted to FP16 once (lower part only), not per level.
//  * X is converted exactly once, in the epilogue of the leaf product that
//    produces it (fused hi[/lo] copies), not re-converted at every level as
//    the reference does with B1 (BLAS/tc_trsm.cu:59-66).
//  * The leaf replaces FP32 cublasStrsm with X_b = B_b * inv(A_bb)^T (or
//    inv(A_bb) * B_b): inv(A_bb) is computed in FP64 by warp-level
//    substitution on 32x32 diagonal sub-blocks and doubling (pairs of
//    inverses joined by two products per level), and applied with the split-FP16 3-product
//    tensor-core GEMM, i.e. FP32-level accuracy like the reference's leaf.
//  * Split points are multiples of 64 so every TMA coordinate stays aligned.
//    For n = nb * 2^L (the configured 16384 / 512) the leaves coincide with
//    the reference's recursion exactly.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "tb_convert.cuh"
#include "tb_internal.h"
#include "tb_ptx.cuh"

namespace tb {

namespace {

constexpr int kLeafMax = 512;  // largest diagonal block inverted explicitly

// Where the FP16 hi/lo pairs of the leaf inverses live: leaf b's W at
// hi + b * stride (lo likewise), leading dimension ld; leaves of `leaf` rows.
struct WOut {
  __half *hi, *lo;
  long long ld, stride;
  int leaf;
};

// Inverse of each 32x32 diagonal sub-block of A (rows/cols >= n padded with
// the identity). One warp per sub-block; lane c owns column c of the inverse
// and runs forward substitution in FP64: row i's quotient is subtracted from
// all later sums at once. Output: D[t*1024 + i + 32*c] (column-major 32x32),
// and with `out` the sub-block's place in its leaf's FP16 hi/lo pair.
//
// A warp runs this once, so what it costs is mostly fetching the code: fully
// unrolled in registers (about 2500 instructions) a launch took 18 to 24 us
// however the substitution was arranged. The loop over the rows stays rolled,
// the columns in shared memory: 20 us.
struct DiagSmem {
  double L[32][33];  // L[i][j], row i
  double w[32][32];  // w[i][c]: column c of the inverse
};

template <class T>
__device__ __forceinline__ void diag_inv32_body(long long n, const T* __restrict__ A, long long lda,
                                                double* __restrict__ D, long long t, bool unit, DiagSmem& s, int c,
                                                const WOut* out) {
  const long long base = t * 32;
#pragma unroll 8
  for (int j = 0; j < 32; ++j) {  // lane c: row c of the sub-block, column j
    const long long gi = base + c, gj = base + j;
    s.L[c][j] =
        (gi < n && gj < n && (c > j || (c == j && !unit))) ? (double)A[gi + gj * lda] : (c == j ? 1.0 : 0.0);
    s.w[j][c] = c == j ? 1.0 : 0.0;
  }
  __syncwarp();
  // FP32 operands: the 32 divisors' reciprocals side by side, then quotients
  // with one residual correction (Markstein 1990), which leaves them correctly
  // rounded but for rare last bits; where a divisor or quotient is not finite
  // the plain product stands. FP64 operands divide: their reciprocals may
  // overflow.
  constexpr bool kRecip = sizeof(T) == 4;
  const double rc = kRecip ? 1.0 / s.L[c][c] : 0.0;
#pragma unroll 1
  for (int i = 0; i < 32; ++i) {
    const double x = s.w[i][c], d = s.L[i][i];
    // the rows below, in groups of 8, are on their way before the quotient is ready
    double l[32], w[32];
#pragma unroll
    for (int g = 0; g < 4; ++g)
      if (8 * g + 7 > i) {
#pragma unroll
        for (int r = 8 * g; r < 8 * g + 8; ++r) l[r] = s.L[r][i], w[r] = s.w[r][c];
      }
    double q;
    if (kRecip) {
      const double r = __shfl_sync(0xffffffffu, rc, i);
      q = x * r;
      const double e = fma(-q, d, x);
      if (fabs(e) <= 1.7976931348623157e308) q = fma(e, r, q);
    } else {
      q = x / d;
    }
    if (i < c) q = 0.0;
    s.w[i][c] = q;
#pragma unroll
    for (int g = 0; g < 4; ++g)
      if (8 * g + 7 > i) {
#pragma unroll
        for (int r = 8 * g; r < 8 * g + 8; ++r)
          if (r > i) s.w[r][c] = w[r] - l[r] * q;
      }
  }
  __syncwarp();
#pragma unroll 8
  for (int j = 0; j < 32; ++j) D[t * 1024 + c + 32 * j] = s.w[c][j];  // lane c: row c
  if (!out || base + c >= n) return;
  const long long b = base / out->leaf, l0 = base - b * out->leaf;
  __half* h = out->hi + b * out->stride + l0 + c + l0 * out->ld;
  __half* l = out->lo + b * out->stride + l0 + c + l0 * out->ld;
#pragma unroll 4
  for (int j = 0; j < 32; ++j) {
    if (base + j >= n) break;
    const double v = s.w[c][j];
    const __half x = __float2half_rn((float)v);
    h[j * out->ld] = x;
    l[j * out->ld] = __float2half_rn((float)((v - (double)__half2float(x)) * 2048.0));
  }
}

// One warp per sub-block, two to a block; out.hi == nullptr: D only.
constexpr int kDiagThreads = 64;

template <class T>
__global__ void __launch_bounds__(kDiagThreads)
    diag_inv32_kernel(long long n, const T* __restrict__ A, long long lda, double* __restrict__ D, bool unit,
                      const WOut out) {
  extern __shared__ __align__(16) uint8_t diag_smem[];
  DiagSmem* s = reinterpret_cast<DiagSmem*>(diag_smem);
  const int warp = threadIdx.x >> 5;
  const long long t = (long long)blockIdx.x * (kDiagThreads / 32) + warp;
  if (t * 32 < n)
    diag_inv32_body<T>(n, A, lda, D, t, unit, s[warp], threadIdx.x & 31, out.hi ? &out : nullptr);
}

template <class T>
tb_status diag_inv32(long long n, const T* A, long long lda, double* D, bool unit, const WOut& out, cudaStream_t st) {
  constexpr int per = kDiagThreads / 32;
  const unsigned blocks = (unsigned)(((n + 31) / 32 + per - 1) / per);
  diag_inv32_kernel<T><<<blocks, kDiagThreads, per * sizeof(DiagSmem), st>>>(n, A, lda, D, unit, out);
  TB_CUDA_TRY(cudaGetLastError());
  note_launch();
  return TB_SUCCESS;
}

// The conversions of a TRSM's preparation in one launch: FP32 -> FP16 copies
// (A's lower part and the first leaf block of B) and the zeroing of an int
// array (the persistent solve's progress counters), as consecutive ranges of
// one 1-D grid. Each job does exactly what its own kernel would (same element
// arithmetic).
struct PrepDev {
  PrepConv conv[2];
  int conv_vec[2];  // 0: element by element, 1: 16-byte stores, 2: and loads, 3: no ragged rows
  long long conv_gx[2], conv_base[2], conv_blocks[2];
  int nconv;
  int* zero;
  long long nzero, zero_base, zero_blocks;
};

constexpr int kPrepThreads = 256;

__global__ void __launch_bounds__(kPrepThreads) trsm_prep_kernel(const __grid_constant__ PrepDev p) {
  const long long b = blockIdx.x;
  for (int z = 0; z < p.nconv; ++z)
    if (b >= p.conv_base[z] && b < p.conv_base[z] + p.conv_blocks[z]) {
      const long long local = b - p.conv_base[z], gx = p.conv_gx[z];
      const long long gy = p.conv_blocks[z] / gx;
      const PrepConv& c = p.conv[z];
      if (p.conv_vec[z] == 3)
        conv::convert8_body<true>(local % gx, gx, local / gx, gy, c.rows, c.cols, c.src, c.lds, true, c.hi, c.lo,
                                  c.ldd, 2048.f, c.tri, 0);
      else if (p.conv_vec[z])
        conv::convert8_body<false>(local % gx, gx, local / gx, gy, c.rows, c.cols, c.src, c.lds, p.conv_vec[z] == 2,
                                   c.hi, c.lo, c.ldd, 2048.f, c.tri, 0);
      else
        conv::convert1_body(local % gx, gx, local / gx, gy, c.rows, c.cols, c.src, c.lds, c.hi, c.lo, c.ldd, 2048.f,
                            c.tri, 0);
      return;
    }
  if (b >= p.zero_base && b < p.zero_base + p.zero_blocks) {
    for (long long i = (b - p.zero_base) * kPrepThreads + threadIdx.x; i < p.nzero; i += p.zero_blocks * kPrepThreads)
      p.zero[i] = 0;
  }
}

// Grouped form: block b belongs to the job whose [first, first + count)
// range of sub-blocks holds b (jobs sorted by `first`).
__global__ void __launch_bounds__(32) diag_inv32_grouped_kernel(const DiagJob* __restrict__ jobs, int njobs) {
  int lo = 0, hi = njobs - 1;
  const long long b = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (jobs[mid].first <= b)
      lo = mid;
    else
      hi = mid - 1;
  }
  const DiagJob& jb = jobs[lo];
  __shared__ DiagSmem s;
  const WOut out{jb.hi, jb.lo, jb.ldw, jb.wstride, jb.leaf};
  diag_inv32_body<float>(jb.n, jb.A, jb.lda, jb.D, b - jb.first, false, s, threadIdx.x, &out);
}

// Leaf inverses by doubling. With the 32 x 32 diagonal blocks inverted, a
// level of h sub-blocks joins neighbouring inverses of h sub-blocks each,
//   W21 = -W22 * (L21 * W11),
// in two products (T = L21 W11, then -W22 T), each a launch in which every
// 32 x 32 tile of every pair of every leaf is one CTA (level 1, one tile per
// pair, does both in one). The serial path of a 512 leaf is 7 launches whose
// CTAs run at most 8 products of 32^3 each; forward substitution by column
// panels was one launch with 120 such products in a row: 371 us for the 32
// leaves of an order-16384 solve and 244 us for 9, against 145 us and 74 us.
//
// W is kept in FP64 in global memory (column-major, leading dimension ldg),
// off-diagonal sub-blocks in place, diagonal ones in D. T takes the unused
// mirrored place above the diagonal, transposed (T's rows along columns), so
// that a ragged second block always fits. Each product step stages a 32 x 32
// block of either operand through shared memory, double-buffered, the next
// step's loads in flight during the products.
// Results leave as FP64 W and as the FP16 hi/lo pair (lo scaled by 2^11) with
// the mirrored sub-block zeroed; the diagonal sub-blocks' pairs come from
// diag_inv32_body. Without hi, W itself is the result.
constexpr int kChainThreads = 128;

struct LeafRef {
  const void* A;  // rows/cols from the leaf's start
  long long lda;
  int size;
  const double* D;  // the leaf's first 32 x 32 inverse
  double* W;
  long long ldg;
  __half *hi, *lo;
  long long ldw;
};

struct InvSmem {
  double LsT[2][32][36];  // LsT[b][k][r]: left operand (r, k)
  double Rs[2][32][36];   // Rs[b][k][c]: right operand (k, c)
};

// acc += the product of left sub-block (r, k) and right sub-block (k, c) on
// the FP64 tensor cores (m8n8k4): warp w owns rows 16 (w & 1) .. + 15 and
// columns 16 (w >> 1) .. + 15 as 2 x 2 tiles; a lane's pair of tile (a, b) is
// row 8a + lane / 4, columns 8b + 2 (lane % 4) and the next. Per-thread 2 x 4
// blocks of plain FMAs loaded three 16-byte words per 8 FMAs and were bound by
// shared memory at a quarter of the FP64 rate.
__device__ __forceinline__ void inv_mma(const InvSmem& s, int buf, int wr, int wc, double (&acc)[2][2][2]) {
  const int lane = threadIdx.x & 31, kq = lane & 3, rq = lane >> 2;
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    double a[2], b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[i] = s.LsT[buf][k + kq][wr + 8 * i + rq];
      b[i] = s.Rs[buf][k + kq][wc + 8 * i + rq];
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                     : "d"(a[i]), "d"(b[j]));
  }
}

// One 32 x 32 tile of level h: PHASE 0 writes T, 1 writes W21, 2 (h == 1)
// does both. x: the tile's index among the leaf's pairs, h * h each.
template <class T, int PHASE>
__device__ __forceinline__ void inv_tile(const LeafRef& f, int h, int x) {
  __shared__ __align__(16) InvSmem s;
  const int nsub = (f.size + 31) / 32;
  const int pair = x / (h * h), i = (x / h) % h, j = x % h;
  const int gi = 2 * pair * h + h + i, gj = 2 * pair * h + j;  // sub-block row and column of W21
  if (gi >= nsub) return;
  const int tid = threadIdx.x;
  const int lr = tid & 31, lc = tid >> 5;                     // load role: row lr, columns lc + 4q
  const int wr = 16 * (lc & 1), wc = 16 * (lc >> 1);          // the warp's quadrant
  const int r0 = wr + (lr >> 2), c0 = wc + 2 * (lr & 3);      // this lane's row and column in tile (0, 0)
  const T* A = static_cast<const T*>(f.A);
  double acc[2][2][2] = {};
  double ra[8], rb[8];
  // L(gi, gk) with rows/columns beyond the leaf read as zero
  auto load_l = [&](int gk, double* v) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int gr = 32 * gi + lr, gc = 32 * gk + lc + 4 * q;
      v[q] = (gr < f.size && gc < f.size) ? (double)A[gr + (long long)gc * f.lda] : 0.0;
    }
  };
  // W(a, b), a >= b
  auto load_w = [&](int a, int b, double* v) {
    const double* p = a == b ? f.D + a * 1024 : f.W + 32 * a + 32ll * b * f.ldg;
    const long long ld = a == b ? 32 : f.ldg;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = __ldcg(p + lr + (long long)(lc + 4 * q) * ld);
  };
  // T(gk, gj), stored transposed in the mirrored place
  auto load_t = [&](int gk, double* v) {
    const double* p = f.W + 32 * gj + 32ll * gk * f.ldg;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = __ldcg(p + lr + (long long)(lc + 4 * q) * f.ldg);
  };
  // left blocks by columns (row lr, k = lc + 4q); right ones by columns of W
  // (k = lr, c = lc + 4q) or of the transposed T (c = lr, k = lc + 4q)
  auto stage = [&](int b, bool right_t) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      s.LsT[b][lc + 4 * q][lr] = ra[q];
      if (right_t)
        s.Rs[b][lc + 4 * q][lr] = rb[q];
      else
        s.Rs[b][lr][lc + 4 * q] = rb[q];
    }
  };
  const int k0 = PHASE == 1 ? 2 * pair * h + h : gj, k1 = PHASE == 1 ? gi + 1 : 2 * pair * h + h;
  auto fetch = [&](int gk) {
    if (PHASE == 1) {
      load_w(gi, gk, ra);
      load_t(gk, rb);
    } else {
      load_l(gk, ra);
      load_w(gk, gj, rb);
    }
  };
  fetch(k0);
  for (int gk = k0; gk < k1; ++gk) {
    const int b = (gk - k0) & 1;
    // buffer b was last read two steps ago, which every thread finished
    // before the barrier of the step in between
    stage(b, PHASE == 1);
    __syncthreads();
    if (gk + 1 < k1) fetch(gk + 1);
    inv_mma(s, b, wr, wc, acc);
  }
  if (PHASE == 2) {  // h == 1: the second product with this tile's own T
    load_w(gi, gi, ra);
#pragma unroll
    for (int q = 0; q < 8; ++q) s.LsT[1][lc + 4 * q][lr] = ra[q];
#pragma unroll
    for (int x2 = 0; x2 < 8; ++x2) {
      const int a = x2 >> 2, b = (x2 >> 1) & 1, e = x2 & 1;
      s.Rs[1][r0 + 8 * a][c0 + 8 * b + e] = acc[a][b][e];
      acc[a][b][e] = 0.0;
    }
    __syncthreads();
    inv_mma(s, 1, wr, wc, acc);
  }
  if constexpr (PHASE == 0) {
#pragma unroll
    for (int x2 = 0; x2 < 8; ++x2) {
      const int a = x2 >> 2, b = (x2 >> 1) & 1, e = x2 & 1;
      f.W[32 * gj + c0 + 8 * b + e + (32ll * gi + r0 + 8 * a) * f.ldg] = acc[a][b][e];
    }
  } else {
#pragma unroll
    for (int x2 = 0; x2 < 8; ++x2) {
      const int a = x2 >> 2, b = (x2 >> 1) & 1, e = x2 & 1;
      const int gr = 32 * gi + r0 + 8 * a, gc = 32 * gj + c0 + 8 * b + e;
      const double v = -acc[a][b][e];
      f.W[gr + (long long)gc * f.ldg] = v;
      if (!f.hi || gr >= f.size) continue;  // gc < gr
      const __half h16 = __float2half_rn((float)v);
      f.hi[gr + (long long)gc * f.ldw] = h16;
      f.lo[gr + (long long)gc * f.ldw] = __float2half_rn((float)((v - (double)__half2float(h16)) * 2048.0));
    }
    if (f.hi) {  // the mirrored sub-block of the pair: zeros
      for (int q = 0; q < 8; ++q) {
        const int gr = 32 * gj + lr, gc = 32 * gi + lc + 4 * q;
        if (gc >= f.size) break;
        f.hi[gr + (long long)gc * f.ldw] = __float2half_rn(0.f);
        f.lo[gr + (long long)gc * f.ldw] = __float2half_rn(0.f);
      }
    }
  }
}

// Leaves [b * leaf, (b + 1) * leaf) of one matrix of order n along blockIdx.y.
template <class T, int PHASE>
__global__ void __launch_bounds__(kChainThreads)
    trtri_level_kernel(const T* __restrict__ A, long long lda, long long n, int leaf, const double* __restrict__ D,
                       double* W, long long ldg, __half* hi, __half* lo, long long ldw, long long wstride, int h) {
  grid_dep_launch();
  grid_dep_wait();  // the previous level (or the diagonal inverses) is complete
  const long long b = blockIdx.y, s = b * leaf;
  LeafRef f;
  f.A = A + s + s * lda;
  f.lda = lda;
  f.size = (int)min((long long)leaf, n - s);
  f.D = D + s / 32 * 1024;
  f.W = W + b * wstride;
  f.ldg = ldg;
  f.hi = hi ? hi + b * wstride : nullptr;
  f.lo = lo ? lo + b * wstride : nullptr;
  f.ldw = ldw;
  inv_tile<T, PHASE>(f, h, blockIdx.x);
}

// Grouped form: one job per (instance, leaf) along blockIdx.y, largest first.
template <int PHASE>
__global__ void __launch_bounds__(kChainThreads) trtri_level_grouped_kernel(const ChainJob* __restrict__ jobs, int h) {
  grid_dep_launch();
  grid_dep_wait();
  const ChainJob& jb = jobs[blockIdx.y];
  LeafRef f;
  f.A = jb.A + jb.s + (long long)jb.s * jb.lda;
  f.lda = jb.lda;
  f.size = jb.size;
  f.D = jb.D + jb.s / 32 * 1024;
  f.W = jb.Wg;
  f.ldg = jb.ldw;
  f.hi = jb.Whi;
  f.lo = jb.Wlo;
  f.ldw = jb.ldw;
  inv_tile<float, PHASE>(f, h, blockIdx.x);
}

// FP64 results (no FP16 pair): the diagonal sub-blocks from D, zeros above
// the diagonal (where T was kept).
__global__ void __launch_bounds__(256) trtri_finish_f64_kernel(long long n, int leaf, const double* __restrict__ D,
                                                               double* __restrict__ W, long long ldw,
                                                               long long wstride) {
  const long long b = blockIdx.y, s = b * leaf;
  const int size = (int)min((long long)leaf, n - s);
  for (int c = blockIdx.x; c < size; c += gridDim.x)
    for (int r = threadIdx.x; r < min(size, c / 32 * 32 + 32); r += blockDim.x)
      W[b * wstride + r + (long long)c * ldw] =
          r < c / 32 * 32 ? 0.0 : D[(s / 32 + c / 32) * 1024 + (r & 31) + 32 * (c & 31)];
}

// A kernel that waits in grid_dep_wait before it reads the previous launch's
// results: its CTAs start as that launch's finish (a level's launch is 5 to 10
// us, about two of them launch latency).
template <class... P, class... Args>
tb_status launch_level(void (*kernel)(P...), dim3 grid, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kChainThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent_launch(st) ? 1 : 0;
  TB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  note_launch();
  return TB_SUCCESS;
}

// All levels of the inverses of `nleaf` leaves of at most `leaf` rows.
template <class T>
tb_status trtri_levels(const T* A, long long lda, long long n, int leaf, int nleaf, const double* D, double* W,
                       long long ldg, __half* hi, __half* lo, long long ldw, long long wstride, cudaStream_t st) {
  const int nsub = (int)((std::min<long long>(leaf, n) + 31) / 32);
  for (int h = 1; h < nsub; h *= 2) {
    const dim3 g((unsigned)((nsub + h - 1) / (2 * h) * h * h), (unsigned)nleaf);
    if (h == 1) {
      TB_TRY(launch_level(trtri_level_kernel<T, 2>, g, st, A, lda, n, leaf, D, W, ldg, hi, lo, ldw, wstride, h));
    } else {
      TB_TRY(launch_level(trtri_level_kernel<T, 0>, g, st, A, lda, n, leaf, D, W, ldg, hi, lo, ldw, wstride, h));
      TB_TRY(launch_level(trtri_level_kernel<T, 1>, g, st, A, lda, n, leaf, D, W, ldg, hi, lo, ldw, wstride, h));
    }
  }
  return TB_SUCCESS;
}


// Leaf block [s, e): X_b = B_b * W^T (right) or W * B_b (left), W = inv(A_bb),
// as a split-FP16 product. W is lower triangular, so each output tile only
// needs the K-blocks up to its own diagonal position. The FP16 hi/lo copy of
// B_b (R) was written by the epilogue of the update that last touched B_b,
// except for the first leaf, which converts it here.
tb_status leaf_solve(TrsmCtx& c, int bidx, long s, long e) {
  const long nbl = e - s;
  GemmCall g;
  g.split = Split::kHiLo;
  const bool split_x = c.split == Split::kHiLo;
  const bool need_convert = (s == 0) && !c.r0_ready;  // the set-up launch may have converted it
  if (c.right) {
    // R = B[:, s:e] (m x nbl) -> FP16 hi/lo; X_b = R * W^T
    if (need_convert) TB_TRY(convert_f32_f16(c.m, nbl, c.B + s * c.ldb, c.ldb, c.rh, c.rl, c.ldr, 2048.f, 0, c.st));
    g.a_hi = {c.rh, c.m, nbl, c.ldr, true};
    g.a_lo = {c.rl, c.m, nbl, c.ldr, true};
    g.b_hi = {c.wh + bidx * c.wstride, nbl, nbl, c.ldw, true};
    g.b_lo = {c.wl + bidx * c.wstride, nbl, nbl, c.ldw, true};
    g.C = c.B + s * c.ldb;
    g.ldc = c.ldb;
    g.M = (int)c.m;
    g.N = (int)nbl;
    g.out_hi = c.xh + s * c.ldx;
    g.out_lo = split_x ? c.xl + s * c.ldx : nullptr;
    g.ld_out = c.ldx;
  } else {
    // R = B[s:e, :] (nbl x n) -> FP16 hi/lo (K-major operand, rows = n); X_b = W * R
    if (need_convert) TB_TRY(convert_f32_f16(nbl, c.n, c.B + s, c.ldb, c.rh, c.rl, c.ldr, 2048.f, 0, c.st));
    g.a_hi = {c.wh + bidx * c.wstride, nbl, nbl, c.ldw, true};
    g.a_lo = {c.wl + bidx * c.wstride, nbl, nbl, c.ldw, true};
    g.b_hi = {c.rh, c.n, nbl, c.ldr, false};
    g.b_lo = {c.rl, c.n, nbl, c.ldr, false};
    g.C = c.B + s;
    g.ldc = c.ldb;
    g.M = (int)nbl;
    g.N = (int)c.n;
    g.out_hi = c.xh + s;
    g.out_lo = split_x ? c.xl + s : nullptr;
    g.ld_out = c.ldx;
  }
  g.alpha = 1.f;
  g.beta = 0.f;
  g.flops = (double)g.M * g.N * nbl;  // triangular solve of the leaf: other * nbl^2 flops
  g.kblocks = (int)((nbl + kGemmBK - 1) / kGemmBK);
  const int bn = gemm_bn(g.split, g.kblocks);
  std::vector<int4> plan = plan_rect(g.M, g.N, bn, 0, g.kblocks);
  for (int4& t : plan) {  // K (= columns of W) beyond the tile's last W row is zero
    const long lim = c.right ? (long)t.y + bn : (long)t.x + kGemmBM;
    const long kmax = lim < nbl ? lim : nbl;
    t.w = (int)((kmax + kGemmBK - 1) / kGemmBK);
  }
  return gemm_launch_plan(g, plan, c.st);  // uneven K ranges: host-balanced tile ranges
}

tb_status update(TrsmCtx& c, long s, long mid, long e) {
  GemmCall g;
  g.split = c.split;
  const bool hilo = c.split == Split::kHiLo;
  const long kk = mid - s;
  if (c.right) {
    // B[:, mid:e] -= X[:, s:mid] * A[mid:e, s:mid]^T
    g.a_hi = {c.xh, c.m, c.n, c.ldx, true};
    g.a_lo = {hilo ? c.xl : nullptr, c.m, c.n, c.ldx, true};
    g.b_hi = {c.ah, c.nt, c.nt, c.lda_h, true};
    g.b_lo = {hilo ? c.al : nullptr, c.nt, c.nt, c.lda_h, true};
    g.a_off = 0;
    g.b_off = (int)mid;
    g.C = c.B + mid * c.ldb;
    g.M = (int)c.m;
    g.N = (int)(e - mid);
  } else {
    // B[mid:e, :] -= A[mid:e, s:mid] * X[s:mid, :]
    g.a_hi = {c.ah, c.nt, c.nt, c.lda_h, true};
    g.a_lo = {hilo ? c.al : nullptr, c.nt, c.nt, c.lda_h, true};
    g.b_hi = {c.xh, c.n, c.m, c.ldx, false};
    g.b_lo = {hilo ? c.xl : nullptr, c.n, c.m, c.ldx, false};
    g.a_off = (int)mid;
    g.b_off = 0;
    g.C = c.B + mid;
    g.M = (int)(e - mid);
    g.N = (int)c.n;
  }
  g.k_off = (int)s;
  g.ldc = c.ldb;
  g.alpha = -1.f;
  g.beta = 1.f;
  // The next leaf is [mid, mid + leaf): this is the last update that touches
  // it, so its FP16 hi/lo copy is written here, fused into the epilogue.
  const long next = std::min<long>(c.leaf, e - mid);
  g.out_hi = c.rh;
  g.out_lo = c.rl;
  g.ld_out = c.ldr;
  if (c.right)
    g.out_n = (int)next;
  else
    g.out_m = (int)next;
  g.flops = 2.0 * g.M * g.N * kk;
  g.kblocks = (int)((kk + kGemmBK - 1) / kGemmBK);
  const std::vector<int4> plan = plan_rect(g.M, g.N, gemm_bn(g.split, g.kblocks), 0, g.kblocks);
  return gemm_launch_plan(g, plan, c.st);
}

tb_status recurse(TrsmCtx& c, long s, long e, const std::vector<long>& leaf_start) {
  if (e - s <= c.leaf) {
    const int bidx = (int)(std::lower_bound(leaf_start.begin(), leaf_start.end(), s) - leaf_start.begin());
    return leaf_solve(c, bidx, s, e);
  }
  // split at a leaf boundary near the middle (multiple of the leaf size)
  const long nleaves = (e - s + c.leaf - 1) / c.leaf;
  const long mid = s + ((nleaves + 1) / 2) * c.leaf;
  TB_TRY(recurse(c, s, mid, leaf_start));
  TB_TRY(update(c, s, mid, e));
  return recurse(c, mid, e, leaf_start);
}

}  // namespace

tb_status trsm_prep_launch(const PrepJobs& j, cudaStream_t st) {
  PrepDev p;
  memset(&p, 0, sizeof(p));
  long long next = 0;
  for (int z = 0; z < j.nconv; ++z) {
    const PrepConv& c = j.conv[z];
    if (c.rows <= 0 || c.cols <= 0) continue;
    const int k = p.nconv++;
    p.conv[k] = c;
    // the grid the conversion kernels would use (tb_convert.cu)
    const bool vec = conv::convert_vec(c.hi, c.lo, c.ldd, 0);
    long long gx = 0, gy = 0;
    conv::convert_grid(c.rows, c.cols, c.tri, vec, sm_count(), kPrepThreads, &gx, &gy);
    const bool aligned = conv::convert_aligned(c.src, c.lds);
    p.conv_vec[k] = !vec ? 0 : conv::convert_whole(c.src, c.lds, c.rows) ? 3 : aligned ? 2 : 1;
    p.conv_gx[k] = gx;
    p.conv_base[k] = next;
    p.conv_blocks[k] = gx * gy;
    next += gx * gy;
  }
  if (j.zero && j.nzero > 0) {
    p.zero = j.zero;
    p.nzero = j.nzero;
    p.zero_base = next;
    p.zero_blocks = std::min<long long>((j.nzero + kPrepThreads - 1) / kPrepThreads, 64);
    next += p.zero_blocks;
  }
  if (next == 0) return TB_SUCCESS;
  if (next > 0x7fffffffLL) return TB_ERROR_NOT_SUPPORTED;
  trsm_prep_kernel<<<(unsigned)next, kPrepThreads, 0, st>>>(p);
  TB_CUDA_TRY(cudaGetLastError());
  note_launch();
  return TB_SUCCESS;
}

// Diagonal-block inverses of many triangular matrices: one launch for the
// 32 x 32 blocks, then the doubling levels over the jobs that reach them
// (`chain` sorted by size, largest first; level_jobs[l]: how many leaves have
// more than 2^l sub-blocks).
tb_status trsm_inverses_grouped(const DiagJob* d_diag, int ndiag, long long nblocks, const ChainJob* d_chain,
                                const std::vector<int>& level_jobs, cudaStream_t st) {
  if (ndiag > 0 && nblocks > 0) {
    diag_inv32_grouped_kernel<<<(unsigned)nblocks, 32, 0, st>>>(d_diag, ndiag);
    TB_CUDA_TRY(cudaGetLastError());
    note_launch();
  }
  for (size_t l = 0; l < level_jobs.size(); ++l) {
    if (level_jobs[l] <= 0) break;
    const int h = 1 << l;
    const dim3 g((unsigned)((kLeafMax / 32 + h - 1) / (2 * h) * h * h), (unsigned)level_jobs[l]);
    if (h == 1) {
      TB_TRY(launch_level(trtri_level_grouped_kernel<2>, g, st, d_chain, h));
    } else {
      TB_TRY(launch_level(trtri_level_grouped_kernel<0>, g, st, d_chain, h));
      TB_TRY(launch_level(trtri_level_grouped_kernel<1>, g, st, d_chain, h));
    }
  }
  return TB_SUCCESS;
}

// FP64 inverses of the diagonal leaf blocks of an FP64 lower-triangular
// matrix (order nt): leaf b, rows [b * leaf, ...) of at most `leaf` (a
// multiple of 32, <= 512), gets W_b at W + b * wstride (ld ldw >= the leaf
// rounded up to 32, zeros above the diagonal). D: (nt + 31) / 32 * 1024
// doubles of scratch.
tb_status trsm_leaf_inverses_f64(long nt, const double* A, long lda, int leaf, int nleaf, double* D, double* W,
                                 long long ldw, long long wstride, cudaStream_t st, bool unit) {
  TB_TRY(diag_inv32<double>(nt, A, lda, D, unit, WOut{}, st));
  TB_TRY(trtri_levels<double>(A, lda, nt, leaf, nleaf, D, W, ldw, nullptr, nullptr, ldw, wstride, st));
  trtri_finish_f64_kernel<<<dim3((unsigned)std::min<long>(leaf, nt), (unsigned)nleaf), 256, 0, st>>>(nt, leaf, D, W,
                                                                                                    ldw, wstride);
  TB_CUDA_TRY(cudaGetLastError());
  note_launch();
  return TB_SUCCESS;
}

// Set-up shared by every right-hand side of one triangular operand: scratch
// for B blocks of at most `m` rows (right side) / `n` columns (left side),
// the FP16 copy of A's lower part and the FP64 leaf inverses as FP16 hi/lo.
// `scratch`: device memory of trsm_scratch_bytes(...) bytes, or nullptr to
// take it from the pool.
namespace {
struct TrsmLayout {
  size_t o_ah, o_al, o_xh, o_xl, o_wh, o_wl, o_rh, o_rl, o_d, o_wg, total;
};

TrsmLayout trsm_layout(TrsmCtx& c, long nleaf) {
  const long nt = c.nt;
  const bool hilo = c.split == Split::kHiLo;
  c.lda_h = round_up(nt, 64);
  // X copy: right: m x n, MN-major rows m; left: m x n col-major, K-major (K = m rows)
  c.ldx = round_up(c.m, 64);
  c.ldw = c.leaf;
  c.wstride = c.ldw * c.leaf;
  c.ldr = c.right ? round_up(c.m, 64) : c.leaf;
  const size_t a_bytes = (size_t)c.lda_h * nt * 2;
  const size_t x_bytes = (size_t)c.ldx * c.n * 2;
  const size_t w_bytes = (size_t)c.wstride * nleaf * 2;
  const size_t r_bytes = (size_t)c.ldr * (c.right ? c.leaf : c.n) * 2;
  const size_t d_bytes = (size_t)((nt + 31) / 32) * 1024 * sizeof(double);
  TrsmLayout L;
  size_t off = 0;
  auto take = [&](size_t b) {
    size_t o = off;
    off += round_up((long long)b, 256);
    return o;
  };
  L.o_ah = take(a_bytes);
  L.o_al = hilo ? take(a_bytes) : 0;
  L.o_xh = take(x_bytes);
  L.o_xl = hilo ? take(x_bytes) : 0;
  L.o_wh = take(w_bytes);
  L.o_wl = take(w_bytes);
  L.o_rh = take(r_bytes);
  L.o_rl = take(r_bytes);
  L.o_d = take(d_bytes);
  L.o_wg = take((size_t)c.wstride * nleaf * sizeof(double));  // FP64 panels of the leaf inverses
  L.total = off;
  return L;
}
}  // namespace

tb_status trsm_setup(bool right, long m, long n, const float* A, long lda, long nb, Split split, cudaStream_t st,
                     void* scratch, TrsmCtx& c, std::vector<long>& leaf_start, bool unit, float* B, long ldb) {
  if (m < 0 || n < 0 || nb <= 0) return TB_ERROR_INVALID_VALUE;
  const long nt = right ? n : m;
  if (lda < (nt > 1 ? nt : 1)) return TB_ERROR_INVALID_VALUE;
  c.right = right;
  c.m = m;
  c.n = n;
  c.nt = nt;
  c.B = nullptr;
  c.ldb = 0;
  // The reference's chunk planner (util/mat_size.cu:31-55) sends an order
  // below 2048 to FP32 cublasStrsm with no FP16 step at all
  // (BLAS/tc_trsm.cu:103-112); the plain form keeps that accuracy contract
  // by using the FP32-accurate split products for such orders.
  c.split = (split == Split::kPlain && nt < 2048) ? Split::kHiLo : split;
  c.st = st;
  long leaf = round_up(std::min<long>(nb, kLeafMax), 64);
  if (leaf > kLeafMax) leaf = kLeafMax;
  c.leaf = (int)leaf;
  const bool hilo = c.split == Split::kHiLo;

  leaf_start.clear();
  for (long s = 0; s < nt; s += leaf) leaf_start.push_back(s);
  const long nleaf = (long)leaf_start.size();
  const TrsmLayout L = trsm_layout(c, nleaf);
  char* ws = static_cast<char*>(scratch ? scratch : pool_get(L.total));
  if (!ws) {
    set_last_error("trsm: cannot allocate %zu bytes of scratch", L.total);
    return TB_ERROR_ALLOC;
  }
  c.ah = reinterpret_cast<__half*>(ws + L.o_ah);
  c.al = hilo ? reinterpret_cast<__half*>(ws + L.o_al) : nullptr;
  c.xh = reinterpret_cast<__half*>(ws + L.o_xh);
  c.xl = hilo ? reinterpret_cast<__half*>(ws + L.o_xl) : nullptr;
  c.wh = reinterpret_cast<__half*>(ws + L.o_wh);
  c.wl = reinterpret_cast<__half*>(ws + L.o_wl);
  c.rh = reinterpret_cast<__half*>(ws + L.o_rh);
  c.rl = reinterpret_cast<__half*>(ws + L.o_rl);
  double* D = reinterpret_cast<double*>(ws + L.o_d);
  double* W64 = reinterpret_cast<double*>(ws + L.o_wg);

  // 1. on the caller's stream, one conversion launch: the FP16 copy of A's
  // lower part (only off-diagonal leaf blocks are read) and, when B is known,
  // the first leaf's operand copy (the persistent solve's, with its zeroed
  // counters, when B takes that path)
  PrepJobs conv;
  if (nleaf > 1) {
    PrepConv& cv = conv.conv[conv.nconv++];
    cv.rows = nt;
    cv.cols = nt;
    cv.src = A;
    cv.lds = lda;
    cv.hi = c.ah;
    cv.lo = c.al;
    cv.ldd = c.lda_h;
    cv.tri = 2;
  }
  c.dag_prepped = false;
  c.r0_ready = false;
  if (B && trsm_dag_eligible(c, B, ldb)) {
    TB_TRY(trsm_dag_prepare(c, B, ldb, conv));
  } else if (B) {
    PrepConv& cv = conv.conv[conv.nconv++];
    const long nbl0 = std::min<long>(leaf, nt);
    cv.rows = right ? m : nbl0;
    cv.cols = right ? nbl0 : n;
    cv.src = B;
    cv.lds = ldb;
    cv.hi = c.rh;
    cv.lo = c.rl;
    cv.ldd = c.ldr;
    c.r0_ready = true;
  }
  // 2. beside it, on an auxiliary stream: the 32 x 32 FP64 inverses of A's
  // diagonal and the leaf inverses' levels (they read only A and each other), joined
  // back into the caller's stream before the solve
  const cudaStream_t sa = aux_stream(1);
  cudaEvent_t fork = nullptr, join = nullptr;
  if (sa) {
    TB_CUDA_TRY(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    TB_CUDA_TRY(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
  }
  const cudaStream_t si = sa ? sa : st;
  tb_status rs = TB_SUCCESS;
  if (sa && (cudaEventRecord(fork, st) != cudaSuccess || cudaStreamWaitEvent(sa, fork, 0) != cudaSuccess))
    rs = TB_ERROR_CUDA;
  if (rs == TB_SUCCESS) {
    rs = diag_inv32<float>(nt, A, lda, D, unit, WOut{c.wh, c.wl, c.ldw, c.wstride, c.leaf}, si);
  }
  if (rs == TB_SUCCESS) {
    rs = trtri_levels<float>(A, lda, nt, c.leaf, (int)nleaf, D, W64, c.ldw, c.wh, c.wl, c.ldw, c.wstride, si);
  }
  if (rs == TB_SUCCESS) rs = trsm_prep_launch(conv, st);
  if (sa && (cudaEventRecord(join, sa) != cudaSuccess || cudaStreamWaitEvent(st, join, 0) != cudaSuccess) &&
      rs == TB_SUCCESS)
    rs = TB_ERROR_CUDA;
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
  return rs;
}

size_t trsm_scratch_bytes(bool right, long m, long n, long nb, Split split) {
  TrsmCtx c;
  c.right = right;
  c.m = m;
  c.n = n;
  c.nt = right ? n : m;
  c.split = (split == Split::kPlain && c.nt < 2048) ? Split::kHiLo : split;
  long leaf = round_up(std::min<long>(nb, kLeafMax), 64);
  c.leaf = (int)(leaf > kLeafMax ? kLeafMax : leaf);
  return trsm_layout(c, (c.nt + c.leaf - 1) / c.leaf).total;
}

// Solves one right-hand side block with a prepared context: B is m' x n
// (right side, m' <= the set-up m) or m x n' (left side, n' <= the set-up n):
// one persistent launch for all the recursion's products where B's layout
// allows it (tb_trsm_dag.cu), else one GEMM launch per leaf and update.
tb_status trsm_solve(TrsmCtx& c, const std::vector<long>& leaf_start, float* B, long ldb, long rows, long cols) {
  if (rows % 4 == 0 && trsm_dag_eligible(c, B, ldb)) return trsm_solve_dag(c, leaf_start, B, ldb, rows, cols);
  return trsm_solve_launches(c, leaf_start, B, ldb, rows, cols);
}

tb_status trsm_solve_launches(TrsmCtx& c, const std::vector<long>& leaf_start, float* B, long ldb, long rows,
                              long cols) {
  if (ldb < (rows > 1 ? rows : 1)) return TB_ERROR_INVALID_VALUE;
  if (rows == 0 || cols == 0) return TB_SUCCESS;
  c.B = B;
  c.ldb = ldb;
  if (c.right)
    c.m = rows;
  else
    c.n = cols;
  return recurse(c, 0, c.nt, leaf_start);
}

tb_status trsm_solve_2s(TrsmCtx& c, const std::vector<long>& leaf_start, float* B, long ldb, long rows, long cols) {
  const long span = c.right ? rows : cols;  // independent systems
  // TB_TRSM_STREAMS in the environment: how many parts of B's independent
  // dimension are solved side by side on as many streams (1 to 4; read
  // once). Default 1: with the setup's preparation launches overlapped
  // (trsm_setup), plain m = n = 16384 nb 512 took 6.13 / 6.69 / 6.87 / 6.89 ms
  // with 1 / 2 / 3 / 4 parts on a B200 (6.47 / 7.03 / 7.20 / 7.22 on another):
  // a part's short launches cost as long as the whole solve's, so splitting
  // them adds latency. Plain products only: the split form's launches carry
  // three products per tile and never gained from parts.
  static const int streams = [] {
    const char* e = getenv("TB_TRSM_STREAMS");
    const int v = e ? atoi(e) : 0;
    return (v >= 1 && v <= 4) ? v : 1;
  }();
  if (rows % 4 == 0 && trsm_dag_eligible(c, B, ldb)) return trsm_solve_dag(c, leaf_start, B, ldb, rows, cols);
  int parts = (c.split == Split::kPlain && span >= 4096) ? streams : 1;
  cudaStream_t sq[4] = {c.st, nullptr, nullptr, nullptr};
  for (int p = 1; p < parts; ++p)
    if (!(sq[p] = aux_stream(p - 1))) parts = 1;
  if (parts == 1 || ldb < (rows > 1 ? rows : 1)) return trsm_solve_launches(c, leaf_start, B, ldb, rows, cols);
  const long w = round_up((span + parts - 1) / parts, 128);
  cudaEvent_t fork, join[4];
  TB_CUDA_TRY(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
  for (auto& e : join) TB_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  tb_status rs = TB_SUCCESS;
  if (cudaEventRecord(fork, c.st) != cudaSuccess) rs = TB_ERROR_CUDA;
  // the parts after the first on the auxiliary streams, the first on the
  // caller's stream; X and R scratch are laid out along the split dimension
  for (int p = parts - 1; p >= 0 && rs == TB_SUCCESS; --p) {
    const long lo = std::min(span, p * w), hi = std::min(span, (p + 1) * w);
    if (hi <= lo) continue;
    TrsmCtx cp = c;
    cp.st = sq[p];
    const long long xo = c.right ? lo : (long long)lo * c.ldx;
    const long long ro = c.right ? lo : (long long)lo * c.ldr;
    cp.xh = c.xh + xo;
    cp.xl = c.xl ? c.xl + xo : nullptr;
    cp.rh = c.rh + ro;
    cp.rl = c.rl + ro;
    if (p > 0 && cudaStreamWaitEvent(sq[p], fork, 0) != cudaSuccess) {
      rs = TB_ERROR_CUDA;
      break;
    }
    rs = c.right ? trsm_solve_launches(cp, leaf_start, B + lo, ldb, hi - lo, cols)
                 : trsm_solve_launches(cp, leaf_start, B + lo * ldb, ldb, rows, hi - lo);
    if (p > 0 && (cudaEventRecord(join[p], sq[p]) != cudaSuccess || cudaStreamWaitEvent(c.st, join[p], 0) != cudaSuccess))
      rs = TB_ERROR_CUDA;
  }
  cudaEventDestroy(fork);
  for (auto& e : join) cudaEventDestroy(e);
  return rs;
}

tb_status trsm_impl(bool right, long m, long n, const float* A, long lda, float* B, long ldb, long nb, Split split,
                    cudaStream_t st) {
  if (m < 0 || n < 0 || nb <= 0) return TB_ERROR_INVALID_VALUE;
  const long nt = right ? n : m;
  if (lda < (nt > 1 ? nt : 1) || ldb < (m > 1 ? m : 1)) return TB_ERROR_INVALID_VALUE;
  if (m == 0 || n == 0) return TB_SUCCESS;
  TrsmCtx c;
  std::vector<long> leaf_start;
  TB_TRY(trsm_setup(right, m, n, A, lda, nb, split, st, nullptr, c, leaf_start, false, B, ldb));
  const tb_status rs = trsm_solve_2s(c, leaf_start, B, ldb, m, n);
  c.r0_ready = false;
  return rs;
}


// ------------------------------------------------------------------ all BLAS flag combinations
// The two solved forms (left/lower/no-trans and right/lower/trans) cover the
// other six through index maps: with J the order reversal,
//   op(A) lower in a left solve  -> L = op(A)           (A^T copied when op(A) = U^T)
//   op(A) upper in a left solve  -> J op(A) J is lower: J X = solve(J op(A) J, J B)
//   op(A) upper in a right solve -> A' = op(A)^T lower  (native when op(A) = L^T)
//   op(A) lower in a right solve -> X J (J op(A) J) = B J with J op(A) J = A'^T,
//                                   A' = J op(A)^T J lower
// The remapped lower triangle is copied once into scratch; B's rows (left)
// or columns (right) are reversed in place around the solve when J appears.
namespace {
__global__ void tri_remap_kernel(long long n, const float* __restrict__ src, long long lds, float* __restrict__ dst,
                                 long long ldd, int transpose, int reverse) {
  for (long long j = blockIdx.y; j < n; j += gridDim.y)
    for (long long i = j + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
      const long long si = reverse ? n - 1 - i : i, sj = reverse ? n - 1 - j : j;
      dst[i + j * ldd] = transpose ? src[sj + si * lds] : src[si + sj * lds];
    }
}

// Reverses the order of the rows (cols == 0) or the columns (cols == 1) of
// an m x n column-major matrix in place.
__global__ void reverse_kernel(long long m, long long n, float* __restrict__ B, long long ldb, int cols) {
  const long long pairs = cols ? n / 2 : m / 2, other = cols ? m : n;
  for (long long q = blockIdx.y; q < other; q += gridDim.y)
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < pairs;
         p += (long long)gridDim.x * blockDim.x) {
      float* x = cols ? B + q + p * ldb : B + p + q * ldb;
      float* y = cols ? B + q + (n - 1 - p) * ldb : B + (m - 1 - p) + q * ldb;
      const float t = *x;
      *x = *y;
      *y = t;
    }
}

tb_status reverse(long long m, long long n, float* B, long long ldb, bool cols, cudaStream_t st) {
  const long long pairs = cols ? n / 2 : m / 2, other = cols ? m : n;
  if (pairs == 0 || other == 0) return TB_SUCCESS;
  dim3 g((unsigned)std::min<long long>((pairs + 255) / 256, 256), (unsigned)std::min<long long>(other, 65535));
  reverse_kernel<<<g, 256, 0, st>>>(m, n, B, ldb, cols ? 1 : 0);
  TB_CUDA_TRY(cudaGetLastError());
  note_launch();
  return TB_SUCCESS;
}
}  // namespace

// Plain solve plus one refinement sweep: X0 = plain TRSM(B); R = B - op(A) X0
// with the FP32-accurate split products (the residual is ~1e-4 of B, so its
// own error stays ~1e-7 of B); D = plain TRSM(R); X = X0 + D. The correction
// carries the plain solve's relative error (~1e-4) on a quantity ~1e-4 the
// size of X, so X reaches FP32-level accuracy.
namespace {
__global__ void add_kernel(long long m, long long n, float* __restrict__ X, long long ldx, const float* __restrict__ D,
                           long long ldd) {
  for (long long j = blockIdx.y; j < n; j += gridDim.y)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (long long)gridDim.x * blockDim.x)
      X[i + j * ldx] += D[i + j * ldd];
}
}  // namespace

tb_status trsm_refine_impl(bool right, long m, long n, const float* A, long lda, float* B, long ldb, long nb,
                           cudaStream_t st) {
  if (m < 0 || n < 0 || nb <= 0) return TB_ERROR_INVALID_VALUE;
  const long nt = right ? n : m;
  if (lda < (nt > 1 ? nt : 1) || ldb < (m > 1 ? m : 1)) return TB_ERROR_INVALID_VALUE;
  if (m == 0 || n == 0) return TB_SUCCESS;
  const size_t bytes = (size_t)m * n * sizeof(float);
  float* R = static_cast<float*>(pool_get(bytes, 1));
  if (!R) {
    set_last_error("trsm refine: cannot allocate %zu bytes for the residual", bytes);
    return TB_ERROR_ALLOC;
  }
  TB_CUDA_TRY(cudaMemcpy2DAsync(R, (size_t)m * 4, B, (size_t)ldb * 4, (size_t)m * 4, (size_t)n,
                                cudaMemcpyDeviceToDevice, st));
  TB_TRY(trsm_impl(right, m, n, A, lda, B, ldb, nb, Split::kPlain, st));
  // R = B0 - op(A) X0 (left: A X0; right: X0 A^T)
  TB_TRY(trmm_ex_impl(right, false, right, false, m, n, -1.f, A, lda, B, ldb, R, m, Split::kHiLo, nullptr, 0, st,
                      1.f));
  TB_TRY(trsm_impl(right, m, n, A, lda, R, m, nb, Split::kPlain, st));
  dim3 g((unsigned)std::min<long long>((m + 255) / 256, 64), (unsigned)std::min<long>(n, 65535));
  add_kernel<<<g, 256, 0, st>>>(m, n, B, ldb, R, m);
  TB_CUDA_TRY(cudaGetLastError());
  note_launch();
  return TB_SUCCESS;
}

tb_status trsm_ex_impl(bool right, bool upper, bool trans, bool unit, long m, long n, const float* A, long lda,
                       float* B, long ldb, long nb, Split split, cudaStream_t st) {
  if (m < 0 || n < 0 || nb <= 0) return TB_ERROR_INVALID_VALUE;
  const long nt = right ? n : m;
  if (lda < (nt > 1 ? nt : 1) || ldb < (m > 1 ? m : 1)) return TB_ERROR_INVALID_VALUE;
  if (m == 0 || n == 0) return TB_SUCCESS;
  const bool op_lower = upper == trans;
  bool tr = false, rev = false;  // how A' is read from A
  if (!right) {
    tr = trans;  // (L,N): as is; (U,T): A^T; (U,N): J A J; (L,T): J A^T J
    rev = !op_lower;
  } else {
    tr = !trans;  // (L,T): as is; (U,N): A^T; (L,N): J A^T J; (U,T): J A J
    rev = op_lower;
  }
  const bool copy = tr || rev;
  const long long ldc_ = round_up(nt, 4);
  const size_t copy_bytes = copy ? (size_t)round_up(ldc_ * nt * 4, 256) : 0;
  const size_t need = copy_bytes + trsm_scratch_bytes(right, m, n, nb, split);
  char* ws = static_cast<char*>(pool_get(need));
  if (!ws) {
    set_last_error("trsm: cannot allocate %zu bytes of scratch", need);
    return TB_ERROR_ALLOC;
  }
  const float* Ause = A;
  long ldause = lda;
  if (copy) {
    float* Ac = reinterpret_cast<float*>(ws);
    dim3 g((unsigned)std::min<long long>((nt + 255) / 256, 64), (unsigned)std::min<long long>(nt, 65535));
    tri_remap_kernel<<<g, 256, 0, st>>>(nt, A, lda, Ac, ldc_, tr ? 1 : 0, rev ? 1 : 0);
    TB_CUDA_TRY(cudaGetLastError());
    note_launch();
    Ause = Ac;
    ldause = (long)ldc_;
  }
  if (rev) TB_TRY(reverse(m, n, B, ldb, right, st));
  TrsmCtx c;
  std::vector<long> leaf_start;
  TB_TRY(trsm_setup(right, m, n, Ause, ldause, nb, split, st, ws + copy_bytes, c, leaf_start, unit, B, ldb));
  TB_TRY(trsm_solve_2s(c, leaf_start, B, ldb, m, n));
  c.r0_ready = false;
  if (rev) TB_TRY(reverse(m, n, B, ldb, right, st));
  return TB_SUCCESS;
}

}  // namespace tb

extern "C" tb_status tb_strsm(char side, long m, long n, const float* A, long lda, float* B, long ldb, long nb,
                              int precision) {
  if (nb == TB_NB_AUTO) return tb::auto_strsm(side, m, n, A, lda, B, ldb, precision);
  bool right;
  if (side == 'R' || side == 'r')
    right = true;
  else if (side == 'L' || side == 'l')
    right = false;
  else
    return TB_ERROR_INVALID_VALUE;
  if (precision == TB_PREC_REFINE) return tb::trsm_refine_impl(right, m, n, A, lda, B, ldb, nb, tb::current_stream());
  if (precision != TB_PREC_PLAIN && precision != TB_PREC_SPLIT) return TB_ERROR_INVALID_VALUE;
  return tb::trsm_impl(right, m, n, A, lda, B, ldb, nb,
                       precision == TB_PREC_SPLIT ? tb::Split::kHiLo : tb::Split::kPlain, tb::current_stream());
}

extern "C" tb_status tb_strsm_ex(char side, char uplo, char transa, char diag, long m, long n, const float* A,
                                 long lda, float* B, long ldb, long nb, int precision) {
  auto flag = [](char c, char a, char b, bool* v) {
    if (c == a || c == a + ('a' - 'A')) {
      *v = false;
      return true;
    }
    if (c == b || c == b + ('a' - 'A')) {
      *v = true;
      return true;
    }
    return false;
  };
  bool right, upper, trans, unit;
  if (!flag(side, 'L', 'R', &right) || !flag(uplo, 'L', 'U', &upper) || !flag(diag, 'N', 'U', &unit))
    return TB_ERROR_INVALID_VALUE;
  if (!flag(transa, 'N', 'T', &trans) && !flag(transa, 'N', 'C', &trans)) return TB_ERROR_INVALID_VALUE;
  if (precision != TB_PREC_PLAIN && precision != TB_PREC_SPLIT) return TB_ERROR_INVALID_VALUE;
  return tb::trsm_ex_impl(right, upper, trans, unit, m, n, A, lda, B, ldb, nb,
                          precision == TB_PREC_SPLIT ? tb::Split::kHiLo : tb::Split::kPlain, tb::current_stream());
}

// ------------------------------------------------------------------ reference C++ API
#include "../../include/TensorBLAS.h"

void tc_trsm(cublasHandle_t, long int m, long int n, float* A, long int lda, float* B, long int ldb, __half*,
             long int nb) {
  tb_status s = tb::trsm_impl(true, m, n, A, lda, B, ldb, nb, tb::Split::kPlain, tb::current_stream());
  if (s != TB_SUCCESS) fprintf(stderr, "TensorBLAS tc_trsm: %s %s\n", tb_status_string(s), tb_last_error());
}

void tc_cumpsgemm_trsm(cublasHandle_t, cumpsgemm::handle_t, long int m, long int n, float* A, long int lda, float* B,
                       long int ldb, long int nb) {
  tb_status s = tb::trsm_impl(true, m, n, A, lda, B, ldb, nb, tb::Split::kHiLo, tb::current_stream());
  if (s != TB_SUCCESS) fprintf(stderr, "TensorBLAS tc_cumpsgemm_trsm: %s %s\n", tb_status_string(s), tb_last_error());
}
