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
// (0 <= mh < 2^31, ml signed). x's low word is taken as signed too, so the sum
// of the middle products stays below 2^62 + 2^61 and low within 2^30 + 2^29. It
// is rounded once, so 0 times anything, and anything times 0, is exactly 0: two
// truncated products with the mean of their errors added as a constant left +-1
// in the place of amplitudes that a circuit keeps at zero, and took longer (28
// qubits: 328 ms, 315 so). The high product stays bare: with all three in one
// chain of 64-bit multiply-adds a rotation took 24 cycles per warp output and
// SM quarter, against 20 for the truncated products. volatile keeps the
// compiler from hoisting products of other pairs, which spills.
__device__ __forceinline__ void fix_mul(long long x, int mh, int ml, long long& high, int& low) {
  const int xl = (int)x, xh = (int)(x >> 32) + (int)((unsigned)xl >> 31);
  long long mid;
  asm volatile("mul.wide.s32 %0, %1, %2;" : "=l"(mid) : "r"(xl), "r"(mh));
  asm volatile("mad.wide.s32 %0, %1, %2, %0;" : "+l"(mid) : "r"(xh), "r"(ml));
  asm volatile("mul.wide.s32 %0, %1, %2;" : "=l"(high) : "r"(xh), "r"(mh));
  low = (int)(mid >> 32) + (int)((unsigned)mid >> 31);
}

// x + q for a 32-bit q.
__device__ __forceinline__ long long fix_add(long long x, int q) {
  unsigned l = (unsigned)x, h = (unsigned)(x >> 32);
  asm("{add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;}" : "+r"(l), "+r"(h) : "r"(q), "r"(q >> 31));
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
        a = x0 - x1 + h1 + (long long)q1;
        b = x1 + x0 - h0 - (long long)q0;
      } else {
        a = x0 - h1 - (long long)q1;
        b = x1 + h0 + (long long)q0;
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

// ---------------------------------------------------------------------------
// A tile of 2^12 amplitudes by 256 threads (fix_window.cuh, batch.cu).
// ---------------------------------------------------------------------------
constexpr int kFixThreads = 256;
constexpr int kFixThreadBits = 8;
constexpr int kFixAmps = 16;  // per thread
constexpr size_t kFixStage = (size_t)8 * kFixThreads * 16;  // table entries on their way

// What decides how a tile runs.
struct FixScan {
  uint32_t mx, mn, any, cnt;  // largest and smallest nonzero amplitude (top words), low words, nonzero amplitudes
  uint32_t mass;              // sum of the squares of the amplitudes' larger components, in 2^-18 M^2 (fixed)
  __device__ int emax() const { return (int)(mx >> 20); }
  __device__ bool zero() const { return mx == 0 && any == 0; }
  // In range, with no more than the pass's (`sparse`) numbers of unreached
  // qubits: log2 (4096 / nonzero amplitudes).
  __device__ bool fixed(uint32_t sparse) const {
    const int unreached = 12 - (31 - __clz((int)cnt | 1));
    return emax() - (int)(mn >> 20) <= kFixRange && emax() > 200 && emax() < 1800 && ((sparse >> unreached) & 1u);
  }
  // Whether the amplitudes outweigh the rounding of the fixed point. With
  // u = 2^-57 M, M the power of two above the largest component, a rotation
  // leaves an error of variance 0.09 u^2 in a component (the rounding of one
  // product and the part of it that is left out) and a table 0.3 u^2; in FP64
  // it is 0.045 and 0.06 times 2^-104 x^2 in a component x. At three or four
  // rotations to a table the two are even where the squares of 2^13 components
  // add up to 22 M^2, or 16 M^2 over each amplitude's larger one, which is the
  // line, in proportion to the nonzero amplitudes: zeros round to zero. Dense
  // random tiles have 100 to 400 M^2, one that a single amplitude dominates 1
  // to 2: 360 small rotations left 2.5e-15 of such a tile, in FP64 3.8e-16.
  __device__ bool heavy() const { return mass >= ((16u << 18) >> 12) * cnt; }
};

// Over the CTA, of amplitudes raw (double bits); s: 5 x 8 words of shared memory.
// MASS: for heavy(); the registers it needs cost the FP32-pair kernel 5 %.
template <bool MASS>
__device__ __forceinline__ FixScan fix_scan(const long long (&raw)[2 * kFixAmps], uint32_t (*s)[kFixThreads / 32]) {
  uint32_t mx = 0, mn = ~0u, any = 0, cnt = 0;
#pragma unroll
  for (int u = 0; u < kFixAmps; ++u) {
    const uint32_t h = max((uint32_t)(raw[2 * u] >> 32) & 0x7FFFFFFFu, (uint32_t)(raw[2 * u + 1] >> 32) & 0x7FFFFFFFu);
    const uint32_t lo = (uint32_t)raw[2 * u] | (uint32_t)raw[2 * u + 1];
    mx = max(mx, h);
    any |= lo;
    if (h | lo) {
      mn = min(mn, h);
      ++cnt;
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  mn = __reduce_min_sync(0xffffffffu, mn);
  any = __reduce_or_sync(0xffffffffu, any);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  uint32_t mass = 0;
  if constexpr (MASS) {  // the squares, in units of the warp's largest exponent: floats in [0, 2)
    float q = 0.f;
    const int unit = ((int)(mx >> 20) - 127) << 20;
#pragma unroll
    for (int u = 0; u < kFixAmps; ++u) {
      const int h = max((int)(raw[2 * u] >> 32) & 0x7FFFFFFF, (int)(raw[2 * u + 1] >> 32) & 0x7FFFFFFF);
      const float f = __int_as_float(max(h - unit, 0) << 3);
      q = fmaf(f, f, q);
    }
    mass = __reduce_add_sync(0xffffffffu, (uint32_t)(q * 65536.f));  // 2^9 2^2 2^16 at most
  }
  if ((threadIdx.x & 31) == 0) {
    const int w = (int)threadIdx.x >> 5;
    s[0][w] = mx;
    s[1][w] = mn;
    s[2][w] = any;
    s[3][w] = cnt;
    if constexpr (MASS) s[4][w] = mass;
  }
  __syncthreads();
  cnt = 0;
#pragma unroll
  for (int w = 0; w < kFixThreads / 32; ++w) {
    mx = max(mx, s[0][w]);
    mn = min(mn, s[1][w]);
    any |= s[2][w];
    cnt += s[3][w];
  }
  if constexpr (MASS) {
    mass = 0;
#pragma unroll
    for (int w = 0; w < kFixThreads / 32; ++w) mass += s[4][w] >> min(2 * ((mx >> 20) - (s[0][w] >> 20)), 31u);
  }
  return FixScan{mx, mn, any, cnt, mass};
}

// The tile's amplitudes (thread tid holds tid + 256 u) into its slots as integers.
__device__ __forceinline__ void fix_put(const long long (&raw)[2 * kFixAmps], unsigned char* tile, int emax) {
  longlong2* ti = reinterpret_cast<longlong2*>(tile);
#pragma unroll
  for (int u = 0; u < kFixAmps; ++u)
    ti[fix_slot(threadIdx.x + kFixThreads * u)] = make_longlong2(fix_from_double(__longlong_as_double(raw[2 * u]), emax),
                                                                 fix_from_double(__longlong_as_double(raw[2 * u + 1]), emax));
}

// Every op of a pass on the tile in its slots; leaves amplitude tid + 256 u in
// r[2u], r[2u + 1] and returns the halvings beyond the planned ones. `stage`:
// this thread's place in kFixStage bytes; s_top: three words, zero.
__device__ __forceinline__ int fix_run(long long (&r)[2 * kFixAmps], unsigned char* tile, longlong2* stage,
                                       const FixOp* ops, int num_ops, const longlong2* tab, int64_t base, int* s_top) {
  const int tid = (int)threadIdx.x, lane = tid & 31;
        uint32_t pr[4] = {0, 0, 0, 0};
        uint32_t pbase = 0, cx = 0;
        int phase = -1;  // of the registers
        int renorm = 0;  // further halvings so far
        const longlong2* ahead = nullptr;  // the entries of the table being fetched
        int4 nxt = *reinterpret_cast<const int4*>(ops);
        for (int o = 0; o < num_ops; ++o) {
          const FixOp* op = ops + o;
          const int4 w0 = nxt;
          if (o + 1 < num_ops) nxt = *reinterpret_cast<const int4*>(op + 1);
          if (w0.x == FIX_ROT) {
            switch (w0.y & 3) {
              case 0: fix_rot_form<kFixAmps, 0>(r, w0.y, w0.z, w0.w); break;
              case 1: fix_rot_form<kFixAmps, 1>(r, w0.y, w0.z, w0.w); break;
              case 2: fix_rot_form<kFixAmps, 2>(r, w0.y, w0.z, w0.w); break;
              default: fix_rot_form<kFixAmps, 3>(r, w0.y, w0.z, w0.w); break;
            }
            if (w0.y & kFixShift) {
  #pragma unroll
              for (int j = 0; j < 2 * kFixAmps; ++j) r[j] >>= 1;
            }
          } else if (w0.x == FIX_TABLE) {
            // groups of four entries: wait for this one, then start the one after the next
  #pragma unroll
            for (int g = 0; g < 4; ++g) {
              if (g < 3) fix_copy_wait<1>();
              else fix_copy_wait<0>();
              longlong2 t[4];
  #pragma unroll
              for (int j = 0; j < 4; ++j) t[j] = stage[kFixThreads * (4 * (g & 1) + j)];
  #pragma unroll
              for (int j = 0; j < 4; ++j) fix_phase(r[2 * (4 * g + j)], r[2 * (4 * g + j) + 1], t[j]);
              if (g < 2) {
  #pragma unroll
                for (int j = 0; j < 4; ++j) fix_copy16(stage + kFixThreads * (4 * g + j), ahead + kFixThreads * (4 * g + 8 + j));
                fix_copy_commit();
              }
            }
          } else if (w0.x == FIX_FETCH) {
            ahead = tab + fix_slice(op, base, 12) + tid;
  #pragma unroll
            for (int g = 0; g < 2; ++g) {
  #pragma unroll
              for (int j = 0; j < 4; ++j) fix_copy16(stage + kFixThreads * (4 * g + j), ahead + kFixThreads * (4 * g + j));
              fix_copy_commit();
            }
          } else if (w0.x == FIX_XOR) {
            if ((base >> w0.y) & 1) cx ^= (uint32_t)w0.z;
          } else {  // FIX_PHASE, FIX_END
            const int4 w1 = *(reinterpret_cast<const int4*>(op) + 1);
            if (phase >= 0) {
  #pragma unroll
              for (int j = 0; j < kFixAmps; ++j) *reinterpret_cast<longlong2*>(tile + fix_reg(pbase, pr, j)) = make_longlong2(r[2 * j], r[2 * j + 1]);
              const int top = __reduce_max_sync(0xffffffffu, fix_top(r));
              if (lane == 0) atomicMax(&s_top[phase % 3], top);
              // the next phase's word: last read before the barrier before this one
              if (tid == 0) s_top[(phase + 1) % 3] = 0;
            }
            __syncthreads();
            const uint32_t img[6] = {(uint32_t)w0.y, (uint32_t)w0.z, (uint32_t)w0.w,
                                     (uint32_t)w1.x, (uint32_t)w1.y, (uint32_t)w1.z};
            // as byte offsets
            pr[0] = (img[0] & 0xFFFFu) << 4;
            pr[1] = img[0] >> 16 << 4;
            pr[2] = (img[1] & 0xFFFFu) << 4;
            pr[3] = img[1] >> 16 << 4;
            cx ^= (uint32_t)op->a[8];
            pbase = cx;
  #pragma unroll
            for (int b = 0; b < 8; ++b) {
              const uint32_t im = (b & 1) ? img[2 + b / 2] >> 16 : img[2 + b / 2] & 0xFFFFu;
              if ((tid >> b) & 1) pbase ^= im;
            }
            pbase <<= 4;
  #pragma unroll
            for (int j = 0; j < kFixAmps; ++j) {
              const longlong2 v = *reinterpret_cast<const longlong2*>(tile + fix_reg(pbase, pr, j));
              r[2 * j] = v.x;
              r[2 * j + 1] = v.y;
            }
            if (phase >= 0) {
              const int sh = fix_renorm(s_top[phase % 3]);
              fix_shift(r, sh);
              renorm += sh;
            }
            ++phase;
          }
        }
  return renorm;
}

}  // namespace dmv
