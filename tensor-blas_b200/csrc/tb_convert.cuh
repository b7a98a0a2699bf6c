// FP32 -> FP16 conversion bodies shared by the conversion kernels
// (tb_convert.cu) and the TRSM preparation kernel (tb_trsm.cu), which runs
// several conversions and the 32 x 32 inverses as block ranges of one grid.
// A body covers the matrix with blocks (bx, by) of a gx x gy grid of
// blockDim.x threads; the element arithmetic is the conversion kernels'.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace tb {
namespace conv {

__device__ __forceinline__ float4 ld_stream(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t pack2(__half a, __half b) {
  return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
}

// Band of the triangle modes 4 / 5: a GEMM tile of at most 256 rows whose K
// range starts (upper) or ends (lower) at its own diagonal block reads the
// other triangle only within 256 of the diagonal.
constexpr long long kTriBand = 256;

// Up to eight (nv) consecutive values of one column; al: 16-byte aligned.
// Columns that are not are read as eight 4-byte loads a thread, whose sectors
// the warp's later loads find in L1. WHOLE: nv == 8 and al always hold, which
// keeps the ragged code out of the kernel (a small conversion is bound by
// fetching its code: 3.0 us against 4.7).
template <bool WHOLE>
__device__ __forceinline__ void load8(const float* s, int nv, bool al, float* f) {
  if (WHOLE || (nv == 8 && al)) {
    const float4 a = ld_stream(s), b = ld_stream(s + 4);
    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
    f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = e < nv ? __ldg(s + e) : 0.f;
  }
}

// nv converted values of one column to hi (and lo), and their copies `dup`
// elements further on; elements beyond nv are not touched.
template <bool WHOLE>
__device__ __forceinline__ void store8(const float* f, int nv, __half* __restrict__ hi, __half* __restrict__ lo,
                                       long long off, long long dup, float lo_scale) {
  __half h[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) h[e] = __float2half_rn(f[e]);
  if (!WHOLE && nv < 8) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (e >= nv) break;
      hi[off + e] = h[e];
      if (dup) hi[off + dup + e] = h[e];
      if (lo) {
        const __half l = __float2half_rn((f[e] - __half2float(h[e])) * lo_scale);
        lo[off + e] = l;
        if (dup) lo[off + dup + e] = l;
      }
    }
    return;
  }
  uint4 o;
  o.x = pack2(h[0], h[1]);
  o.y = pack2(h[2], h[3]);
  o.z = pack2(h[4], h[5]);
  o.w = pack2(h[6], h[7]);
  *reinterpret_cast<uint4*>(hi + off) = o;
  if (dup) *reinterpret_cast<uint4*>(hi + dup + off) = o;
  if (lo) {
    __half l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) l[e] = __float2half_rn((f[e] - __half2float(h[e])) * lo_scale);
    uint4 q;
    q.x = pack2(l[0], l[1]);
    q.y = pack2(l[2], l[3]);
    q.z = pack2(l[4], l[5]);
    q.w = pack2(l[6], l[7]);
    *reinterpret_cast<uint4*>(lo + off) = q;
    if (dup) *reinterpret_cast<uint4*>(lo + dup + off) = q;
  }
}

// Vector path: a thread owns 8 rows of a column (the last group of a column
// may be shorter) and writes them with 16-byte stores: ldd a multiple of 8,
// 16-byte aligned hi and lo. al: the source's columns are 16-byte aligned
// (lds a multiple of 4). Ragged and unaligned sources took a one-row-per-thread
// path before: A's lower part and the first leaf's 6003 x 512 rows of a TRSM
// of order 4100 went from 277 to 37 us.
// Whole matrices (tri 0): a thread walks the columns by, by + gy, ... four at
// a time, with the four columns' loads (128 bytes) in flight together; grids
// of a few blocks per SM then keep enough bytes in flight to run at the HBM
// rate.
template <bool WHOLE>
__device__ __forceinline__ void convert8_body(long long bx, long long gx, long long by, long long gy, long long rows,
                                              long long cols, const float* __restrict__ src, long long lds, bool al,
                                              __half* __restrict__ hi, __half* __restrict__ lo, long long ldd,
                                              float lo_scale, int tri, long long dup) {
  const long long rows8 = (rows + 7) >> 3;
  // rows [8v, ...) of the columns by, by + gy, ... below jend
  auto walk = [&](long long v, long long jend) {
    const long long i = v << 3;
    const int nv = (int)min(8LL, rows - i);
    long long j = by;
    for (; j + 3 * gy < jend; j += 4 * gy) {
      float f[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) load8<WHOLE>(src + i + (j + u * gy) * lds, nv, al, f[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) store8<WHOLE>(f[u], nv, hi, lo, i + (j + u * gy) * ldd, dup, lo_scale);
    }
    for (; j < jend; j += gy) {
      float f[8];
      load8<WHOLE>(src + i + j * lds, nv, al, f);
      store8<WHOLE>(f, nv, hi, lo, i + j * ldd, dup, lo_scale);
    }
  };
  if (tri == 2) {
    // lower part: row group v (rows 8v .. 8v + 7) has the columns j < 8v + 8.
    // A thread takes row groups t and rows8 - 1 - t, so every thread has
    // about the same number of columns.
    const long long half = (rows8 + 1) >> 1;
    for (long long t = bx * blockDim.x + threadIdx.x; t < half; t += gx * blockDim.x) {
      for (int w = 0; w < 2; ++w) {
        const long long v = w ? rows8 - 1 - t : t;
        if (w && v == t) break;
        walk(v, min(cols, (v << 3) + 8));
      }
    }
    return;
  }
  if (tri == 0) {
    for (long long v = bx * blockDim.x + threadIdx.x; v < rows8; v += gx * blockDim.x) walk(v, cols);
    return;
  }
  for (long long j = by; j < cols; j += gy) {
    long long v0 = bx * blockDim.x + threadIdx.x, vend = rows8;
    if (tri == 4) vend = min(rows8, (j / kTriBand + 1) * (kTriBand / 8));  // rows i < band end
    if (tri == 5) v0 += (j / kTriBand) * (kTriBand / 8);                   // rows i >= band start
    for (long long v = v0; v < vend; v += gx * blockDim.x) {
      const long long i = v << 3;
      const int nv = (int)min(8LL, rows - i);
      float f[8];
      load8<WHOLE>(src + i + j * lds, nv, al, f);
      if (tri == 1 || tri == 5) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (i + e < j) f[e] = 0.f;
      } else if (tri == 3 || tri == 4) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (i + e > j) f[e] = 0.f;
      }
      store8<WHOLE>(f, nv, hi, lo, i + j * ldd, dup, lo_scale);
    }
  }
}

// Whether a conversion can take convert8_body, and with aligned loads.
inline bool convert_vec(const void* hi, const void* lo, long long ldd, long long dup) {
  return ldd % 8 == 0 && dup % 8 == 0 && reinterpret_cast<uintptr_t>(hi) % 16 == 0 &&
         reinterpret_cast<uintptr_t>(lo) % 16 == 0;
}
inline bool convert_aligned(const void* src, long long lds) {
  return lds % 4 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0;
}
// Its WHOLE form: aligned loads and no partial group.
inline bool convert_whole(const void* src, long long lds, long long rows) {
  return rows % 8 == 0 && convert_aligned(src, lds);
}

// Grid (gx, gy) of convert8_body / convert1_body for a rows x cols operand:
// whole matrices and lower parts on the vector path take about 16 blocks of
// 256 threads per SM, each thread walking many columns; the other forms one
// column per block row.
inline void convert_grid(long long rows, long long cols, int tri, bool vec, int sms, int threads, long long* gx,
                         long long* gy) {
  long long units = vec ? (rows + 7) / 8 : rows;
  if (vec && tri == 2) units = (units + 1) / 2;  // two row groups per thread
  long long x = (units + threads - 1) / threads;
  if (x > 1024) x = 1024;
  long long y = cols < 65535 ? cols : 65535;
  if (vec && (tri == 0 || tri == 2)) {
    const long long want = (16LL * sms + x - 1) / x;
    y = want < y ? want : y;
    if (y < 1) y = 1;
  }
  *gx = x;
  *gy = y;
}

// Scalar fallback for destinations that 16-byte stores cannot address.
__device__ __forceinline__ void convert1_body(long long bx, long long gx, long long by, long long gy, long long rows,
                                              long long cols, const float* __restrict__ src, long long lds,
                                              __half* __restrict__ hi, __half* __restrict__ lo, long long ldd,
                                              float lo_scale, int tri, long long dup) {
  for (long long j = by; j < cols; j += gy) {
    long long i0 = bx * blockDim.x + threadIdx.x, iend = rows;
    if (tri == 2) i0 += (j >> 3) << 3;
    if (tri == 4) iend = min(rows, (j / kTriBand + 1) * kTriBand);
    if (tri == 5) i0 += (j / kTriBand) * kTriBand;
    for (long long i = i0; i < iend; i += gx * blockDim.x) {
      float f = src[i + j * lds];
      if (((tri == 1 || tri == 5) && i < j) || ((tri == 3 || tri == 4) && i > j)) f = 0.f;
      const __half h = __float2half_rn(f);
      hi[i + j * ldd] = h;
      if (dup) hi[dup + i + j * ldd] = h;
      if (lo) {
        const __half l = __float2half_rn((f - __half2float(h)) * lo_scale);
        lo[i + j * ldd] = l;
        if (dup) lo[dup + i + j * ldd] = l;
      }
    }
  }
}

}  // namespace conv
}  // namespace tb
