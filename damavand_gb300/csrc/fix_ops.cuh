// Device arithmetic of the fixed-point passes (fix_window.cuh, kernels_adjoint.cu):
// amplitudes as pairs of 64-bit integers under a tile exponent.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"
#include "tma.cuh"

namespace dmv {

// A tile's largest component starts at 57 bits. Between phases the tile is
// brought back below 2^57 when one has grown past 2^58, and up to there when
// all have shrunk below 2^55.
constexpr int kFixTopBits = 26;  // of the high word
constexpr int kFixLowBits = 24;

// The shift (right, or left when negative) that a largest high word `m` asks for.
__device__ __forceinline__ int fix_renorm(int m) {
  const int bits = 32 - __clz(m);
  return bits > kFixTopBits || bits < kFixLowBits ? bits - (kFixTopBits - 1) : 0;
}

template <int N>
__device__ __forceinline__ void fix_shift(long long (&r)[N], int s) {
  if (s > 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] >>= s;
  } else if (s < 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] <<= -s;
  }
}

// The largest |high word| (x >= 0: x, else ~x) of the registers.
template <int N>
__device__ __forceinline__ int fix_top(const long long (&r)[N]) {
  int hi = 0, lo = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    hi = max(hi, (int)(r[j] >> 32));
    lo = min(lo, (int)(r[j] >> 32));
  }
  return max(hi, ~lo);
}

__device__ __forceinline__ uint32_t fix_slot(uint32_t l) { return l ^ (((l >> 3) ^ (l >> 6) ^ (l >> 9)) & 7u); }

__device__ __forceinline__ long long fix_wide(int a, int b) {
  long long p;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(p) : "r"(a), "r"(b));
  return p;
}

// x m / 2^64 = high + low for |x| < 2^62 and the multiplier m = mh 2^32 + ml
// (0 <= mh < 2^31, ml signed). x's low word is taken as signed too, so low
// stays within 2^30 + 2^29; the two truncated middle products average to the
// 1 that is added. Three bare products: with the sums inside the 64-bit
// multiply-adds a rotation took 24 cycles per warp output and SM quarter, so
// 20; volatile keeps the compiler from hoisting products of other pairs,
// which spills (23 without it).
__device__ __forceinline__ void fix_mul(long long x, int mh, int ml, long long& high, int& low) {
  const int xl = (int)x, xh = (int)(x >> 32) + (int)((unsigned)xl >> 31);
  int q1, q2;
  asm volatile("mul.hi.s32 %0, %1, %2;" : "=r"(q1) : "r"(xl), "r"(mh));
  asm volatile("mul.hi.s32 %0, %1, %2;" : "=r"(q2) : "r"(xh), "r"(ml));
  asm volatile("mul.wide.s32 %0, %1, %2;" : "=l"(high) : "r"(xh), "r"(mh));
  low = q1 + q2 + 1;
}

// x + q and x - q for a 32-bit q.
__device__ __forceinline__ long long fix_add(long long x, int q) {
  unsigned l = (unsigned)x, h = (unsigned)(x >> 32);
  asm("{add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;}" : "+r"(l), "+r"(h) : "r"(q), "r"(q >> 31));
  return (long long)((unsigned long long)h << 32 | l);
}
__device__ __forceinline__ long long fix_sub(long long x, int q) {
  unsigned l = (unsigned)x, h = (unsigned)(x >> 32);
  asm("{sub.cc.u32 %0, %0, %2;\n\tsubc.u32 %1, %1, %3;}" : "+r"(l), "+r"(h) : "r"(q), "r"(q >> 31));
  return (long long)((unsigned long long)h << 32 | l);
}

// x in double -> round(x 2^(1079 - emax)) for |x| < 2^(emax - 1022): below 2^57.
__device__ __forceinline__ long long fix_from_double(double x, int emax) {
  const int hi = __double2hiint(x);
  const int E = (hi >> 20) & 0x7FF;
  const unsigned long long M =
      ((unsigned long long)(unsigned)((hi & 0xFFFFF) | 0x100000) << 32 | (unsigned)__double2loint(x)) << 11;
  const int s = 6 + emax - E;  // the leading one goes from bit 63 to bit 57 - (emax - E), one bit kept to round
  unsigned long long X = E > 0 && s < 64 ? M >> s : 0ull;
  X = (X + 1) >> 1;
  const long long sg = (long long)(hi >> 31);
  return ((long long)X ^ sg) - sg;
}

// round(x) 2^(e - 1075) as a double (e: the biased exponent of 2^52 in x's
// units, the result normal), ties away from zero. Integer operations only: the
// conversion instruction runs at the FP64 rate, 75 cycles per warp.
__device__ __forceinline__ double fix_to_double(long long x, int e) {
  const unsigned sign = (unsigned)(x >> 32) & 0x80000000u;
  const unsigned long long a = x < 0 ? 0ull - (unsigned long long)x : (unsigned long long)x;
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a;
  const int lz = ah ? __clz((int)ah) : 32 + __clz((int)al);
  const unsigned long long m = (((a << (lz & 63)) >> 1) + 0x200ull) >> 10;  // 53 bits, or 2^53
  const unsigned long long r =
      m + ((unsigned long long)(unsigned)(e + 10 - lz) << 52);  // the leading one adds 1 to the exponent
  return a == 0 ? 0.0 : __longlong_as_double((long long)(r | (unsigned long long)sign << 32));
}

// The rotation [[1, -w], [w, 1]] of every register pair along bit TP; the
// multiplier is w, or 1 - w (COMP: w >= 1/2).
template <int NA, int TP, bool COMP>
__device__ __forceinline__ void fix_rot(long long (&r)[2 * NA], int mh, int ml) {
#pragma unroll
  for (int j = 0; j < NA; ++j) {
    if (j & (1 << TP)) continue;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      long long& a = r[2 * j + k];
      long long& b = r[2 * (j | (1 << TP)) + k];
      const long long x0 = a, x1 = b;
      long long h0, h1;
      int q0, q1;
      fix_mul(x0, mh, ml, h0, q0);
      fix_mul(x1, mh, ml, h1, q1);
      if constexpr (COMP) {
        a = fix_add(x0 - x1 + h1, q1);
        b = fix_sub(x1 + x0 - h0, q0);
      } else {
        a = fix_sub(x0 - h1, q1);
        b = fix_add(x1 + h0, q0);
      }
    }
  }
}

template <int NA, int TP>
__device__ __forceinline__ void fix_rot_form(long long (&r)[2 * NA], int flags, int mh, int ml) {
  if (flags & kFixComplement) fix_rot<NA, TP, true>(r, mh, ml);
  else fix_rot<NA, TP, false>(r, mh, ml);
}

// (x, y) times the Q.62 phase w = (cos, sin) (words hi 2^32 + lo with lo
// signed), one rounding per component.
__device__ __forceinline__ void fix_phase(long long& x, long long& y, const longlong2 w) {
  const int cl = (int)w.x, ch = (int)(w.x >> 32), sl = (int)w.y, sh = (int)(w.y >> 32);
  const int xl = (int)x, xh = (int)(x >> 32) + (int)((unsigned)xl >> 31);
  const int yl = (int)y, yh = (int)(y >> 32) + (int)((unsigned)yl >> 31);
  const long long b0 = fix_wide(xh, cl) + fix_wide(xl, ch) - fix_wide(yh, sl) - fix_wide(yl, sh) + (1ll << 29);
  const long long b1 = fix_wide(yh, cl) + fix_wide(yl, ch) + fix_wide(xh, sl) + fix_wide(xl, sh) + (1ll << 29);
  const long long a0 = fix_wide(xh, ch) - fix_wide(yh, sh), a1 = fix_wide(yh, ch) + fix_wide(xh, sh);
  x = (a0 << 2) + (b0 >> 30);
  y = (a1 << 2) + (b1 >> 30);
}

// First entry of a table's slice for the tile (2^k amplitudes) at `base`.
__device__ __forceinline__ int64_t fix_slice(const FixOp* op, int64_t base, int k) {
  const int4 w0 = *reinterpret_cast<const int4*>(op);
  const int4 w1 = *(reinterpret_cast<const int4*>(op) + 1);
  int gsel = 0;
  if (w0.z > 0) gsel |= (int)((base >> w0.w) & 1);
  if (w0.z > 1) gsel |= (int)((base >> w1.x) & 1) << 1;
  if (w0.z > 2) gsel |= (int)((base >> w1.y) & 1) << 2;
  return (int64_t)w0.y + ((int64_t)gsel << k);
}

// Asynchronous copy of 16 bytes (L2 -> shared memory) by this thread.
__device__ __forceinline__ void fix_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void fix_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void fix_copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Slot of register j.
__device__ __forceinline__ uint32_t fix_reg(uint32_t base, const uint32_t (&pr)[4], int j) {
  uint32_t s = base;
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if ((j >> b) & 1) s ^= pr[b];
  return s;
}

}  // namespace dmv
