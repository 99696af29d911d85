// Adjoint gradient sweep of complex128 states in windows.
//
// A run of uncontrolled gates on one qubit is one 2x2 in the sweep, and the
// gradients of all its rotations follow from three sums over the state,
// Im <lambda| P |psi> for P = X, Y, Z on that qubit at the run's end: undoing a
// gate of the run conjugates P inside it. So a run of RX, RY, RZ costs one
// measurement and one update of psi and lambda instead of three of each, and a
// window pass (the forward planner's windows over the reversed gate list)
// holds a tile of both states while it applies many runs. The updates are the
// forward pass's rotations, phase tables and exchanges, in the fixed-point
// arithmetic of fix_ops.cuh (2^-57 of a tile's largest component: psi and
// lambda are scratch, and the sums they end in are no finer than that where
// the tile's norm is spread). Concentrated tiles (the last ones before |0...0>),
// and any out of the exponent range, non-finite ones among them, run in FP64.
// A gate at a time in FP64 (k_adjoint_step) spends about 26 FP64 multiply-adds
// per amplitude pair and rotation, one per 75 cycles and warp, and streams both
// states from HBM for each gate.
//
// Tiles are 2^11 amplitudes of each state, 8 per thread of 256 in registers (64
// of 128 registers), two CTAs per SM, so that one's loads overlap the other's
// arithmetic. A state of fewer qubits is one tile padded with zeros.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "fix_ops.cuh"
#include "policies.cuh"

namespace dmv {
namespace {

constexpr int kAdjBits = 11;
constexpr int kAdjThreads = 256;
constexpr int kAdjThreadBits = 8;
constexpr int kAdjAmps = 8;
constexpr int kAdjWarps = kAdjThreads / 32;
// A tile is taken when a sixteenth of either state is within 2^kAdjSpread of its
// largest component. The forward's stricter lines (FixScan) guard the norm of
// the error, which 2^12 components of a concentrated tile share out; a gradient
// is an inner product with the other state, and what 2^-57 M in every component
// adds to it is that times the other's norm, however M is shared out. On states
// around a product state, also with weights that vanish at its largest
// amplitude, the gradients' errors against 64 bits are 0.3 to 1 times those of
// the sweep in FP64 gate by gate.
constexpr int kAdjSpread = 6;  // binary orders
constexpr int kAdjGrads = 48;  // measurements per launch (a longer window runs as several launches)

struct AdjFixParams {
  double2* psi;
  double2* lam;
  int32_t low, nh;
  int32_t high[16];
  int32_t num_tiles;
  int32_t num_ops, num_fix_ops, num_grads;
  int32_t shifts, scale_exp;  // halvings over the pass; the states leave it times 2^scale_exp
  const Op* ops;              // the FP64 form
  const double2* tab;
  const FixOp* fix_ops;
  const longlong2* fix_tab;
  double* partial;  // [3 * grad + component][CTA]
  int32_t cols;
};

constexpr size_t kAdjStage = (size_t)4 * kAdjThreads * 16;
constexpr size_t kAdjSmem = ((size_t)2 << kAdjBits) * 16 + kAdjStage + (size_t)kFixSmemOps * sizeof(FixOp) +
                            (size_t)kAdjGrads * 3 * (kAdjWarps * 12 + 8);

// A sum of products of two fixed-point values in units of 2^64: h + f 2^-26.
// The low words' products count: with amplitudes near 2^54 what lies below the
// unit is 2^-44 of a product, and a gradient is no larger than the rounding of
// a sum of that many terms (dropping it left 7.5e-14 of the 22-qubit gradient
// where FP64 leaves 8e-15).
//
// How large it gets. A phase starts with components below 2^58 (fix_renorm), and
// the stored norm at most doubles until the next (`grown` from 1/sqrt 2 to
// sqrt 2). So over a thread's 16 components of each state the sum is at most
// 16 2^116 4 / 2^64 = 2^58, and over a tile's 2^12 it is 2^66, which 64 bits do
// not hold: what leaves the thread is in units of 2^(64 + kGradShift), at most
// 2^62 over the tile.
constexpr int kGradShift = 4;
struct FixSum {
  long long h;
  unsigned f;
};

__device__ __forceinline__ int fix_hi(int a, int b) {
  int q;
  asm volatile("mul.hi.s32 %0, %1, %2;" : "=r"(q) : "r"(a), "r"(b));
  return q;
}

// s + a b - c d (x: high word, y: low word, both signed; |high| < 2^30). f
// grows by less than 2^26 a call.
__device__ __forceinline__ void fix_dot2(FixSum& s, int2 a, int2 b, int2 c, int2 d) {
  const int q = fix_hi(a.y, b.y) - fix_hi(c.y, d.y);
  const long long m =
      fix_add(fix_wide(a.y, b.x) + fix_wide(a.x, b.y) - fix_wide(c.y, d.x) - fix_wide(c.x, d.y), q);
  s.h = fix_add(s.h + fix_wide(a.x, b.x) - fix_wide(c.x, d.x), (int)(m >> 32));
  s.f += (unsigned)m >> 6;
}

__device__ __forceinline__ int2 fix_words(long long x) {
  return make_int2((int)(x >> 32) + (int)((unsigned)x >> 31), (int)x);
}

// Im <lambda| P |psi> of X, Y, Z on register bit TP over this thread's pairs.
template <int TP>
__device__ __forceinline__ void fix_grad(const long long (&p)[2 * kAdjAmps], const long long (&l)[2 * kAdjAmps],
                                         FixSum (&g)[3]) {
#pragma unroll
  for (int j = 0; j < kAdjAmps; ++j) {
    if (j & (1 << TP)) continue;
    const int j1 = j | (1 << TP);
    const int2 p0r = fix_words(p[2 * j]), p0i = fix_words(p[2 * j + 1]);
    const int2 p1r = fix_words(p[2 * j1]), p1i = fix_words(p[2 * j1 + 1]);
    const int2 l0r = fix_words(l[2 * j]), l0i = fix_words(l[2 * j + 1]);
    const int2 l1r = fix_words(l[2 * j1]), l1i = fix_words(l[2 * j1 + 1]);
    fix_dot2(g[0], l0r, p1i, l0i, p1r);
    fix_dot2(g[0], l1r, p0i, l1i, p0r);
    fix_dot2(g[1], l1r, p0r, l0r, p1r);
    fix_dot2(g[1], l1i, p0i, l0i, p1i);
    fix_dot2(g[2], l0r, p0i, l0i, p0r);
    fix_dot2(g[2], l1i, p1r, l1r, p1i);
  }
}

// Exact sum over the warp.
__device__ __forceinline__ long long warp_sum(long long s) {
  const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)s & 0xFFFFFFu);
  const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(s >> 24) & 0xFFFFFFu);
  const int hi = __reduce_add_sync(0xffffffffu, (int)(s >> 48));
  return (long long)lo + ((long long)mid << 24) + (long long)((unsigned long long)(long long)hi << 48);
}

__global__ void __launch_bounds__(kAdjThreads, 2) k_adjoint_fix(const __grid_constant__ AdjFixParams p) {
  constexpr int NT = kAdjThreads, NA = kAdjAmps, T = 1 << kAdjBits;
  extern __shared__ __align__(16) unsigned char adj_raw[];
  __shared__ uint32_t s_mx[2][kAdjWarps], s_any[kAdjWarps], s_cnt[kAdjWarps];
  __shared__ double s_red[kAdjWarps][3];
  __shared__ int64_t s_slot[NA];
  __shared__ int s_top[2][3];     // largest component of psi and lambda, by phase
  __shared__ int s_exp[kAdjGrads];  // halvings of both states before each measurement
  longlong2* tp = reinterpret_cast<longlong2*>(adj_raw);
  longlong2* tl = tp + T;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  longlong2* stage = tl + T + tid;
  FixOp* sops = reinterpret_cast<FixOp*>(tl + T + 4 * NT);
  long long* s_acc = reinterpret_cast<long long*>(sops + kFixSmemOps);  // [grad][3][warp]
  double* s_sum = reinterpret_cast<double*>(s_acc + (size_t)kAdjGrads * 3 * kAdjWarps);
  unsigned* s_frac = reinterpret_cast<unsigned*>(s_sum + (size_t)kAdjGrads * 3);
  const int low = p.low, nh = p.nh, kv = low + nh;
  int64_t t_off = 0;
  for (int i = 0; i < min(kv, kAdjThreadBits); ++i)
    t_off |= (int64_t)((tid >> i) & 1) << (i < low ? i : p.high[i - low]);
  if (tid < NA) {
    int64_t off = 0;
    for (int i = kAdjThreadBits; i < kv; ++i) off |= (int64_t)((tid >> (i - kAdjThreadBits)) & 1) << (i < low ? i : p.high[i - low]);
    s_slot[tid] = off;
  }
  if (tid < 6) s_top[tid / 3][tid % 3] = 0;
  for (int i = tid; i < 3 * p.num_grads; i += NT) s_sum[i] = 0.0;
  const FixOp* fops = p.fix_ops;
  if (p.num_fix_ops <= kFixSmemOps) {
    int4* dst = reinterpret_cast<int4*>(sops);
    const int4* src = reinterpret_cast<const int4*>(p.fix_ops);
    for (int i = tid; i < p.num_fix_ops * 3; i += NT) dst[i] = src[i];
    fops = sops;
  }
  __syncthreads();

  for (int tix = (int)blockIdx.x; tix < p.num_tiles; tix += (int)gridDim.x) {
    int64_t base = (int64_t)tix << low;
    for (int i = 0; i < nh; ++i) base = insert_zero(base, p.high[i]);
    const int64_t at = base | t_off;
    long long a[2 * NA], b[2 * NA];
    uint32_t mx[2] = {0, 0}, any = 0;
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      const bool valid = (tid + NT * u) >> kv == 0;
      longlong2 v = make_longlong2(0, 0), w = v;
      if (valid) {
        v = *reinterpret_cast<const longlong2*>(p.psi + (at | s_slot[u]));
        w = *reinterpret_cast<const longlong2*>(p.lam + (at | s_slot[u]));
      }
      a[2 * u] = v.x;
      a[2 * u + 1] = v.y;
      b[2 * u] = w.x;
      b[2 * u + 1] = w.y;
    }
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      if ((tid + NT * u) >> kv) continue;
      const uint32_t h = max((uint32_t)(a[2 * u] >> 32) & 0x7FFFFFFFu, (uint32_t)(a[2 * u + 1] >> 32) & 0x7FFFFFFFu);
      const uint32_t g = max((uint32_t)(b[2 * u] >> 32) & 0x7FFFFFFFu, (uint32_t)(b[2 * u + 1] >> 32) & 0x7FFFFFFFu);
      mx[0] = max(mx[0], h);
      mx[1] = max(mx[1], g);
      any |= (uint32_t)a[2 * u] | (uint32_t)a[2 * u + 1] | (uint32_t)b[2 * u] | (uint32_t)b[2 * u + 1];
    }
    any = __reduce_or_sync(0xffffffffu, any);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      mx[s] = __reduce_max_sync(0xffffffffu, mx[s]);
      if (lane == 0) s_mx[s][warp] = mx[s];
    }
    if (lane == 0) s_any[warp] = any;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kAdjWarps; ++w) {
#pragma unroll
      for (int s = 0; s < 2; ++s) mx[s] = max(mx[s], s_mx[s][w]);
      any |= s_any[w];
    }
    const int ea = (int)(mx[0] >> 20), eb = (int)(mx[1] >> 20);
    const bool zero = mx[0] == 0 && mx[1] == 0 && any == 0;
    bool fixed = ea > 200 && ea < 1800 && eb > 200 && eb < 1800;
    if (fixed) {
      // a sixteenth of either state within 2^kAdjSpread of its largest
      uint32_t cnt = 0;
#pragma unroll
      for (int u = 0; u < NA; ++u) {
        const uint32_t h = max((uint32_t)(a[2 * u] >> 32) & 0x7FFFFFFFu, (uint32_t)(a[2 * u + 1] >> 32) & 0x7FFFFFFFu);
        const uint32_t g = max((uint32_t)(b[2 * u] >> 32) & 0x7FFFFFFFu, (uint32_t)(b[2 * u + 1] >> 32) & 0x7FFFFFFFu);
        cnt += (int)(h >> 20) >= ea - kAdjSpread ? 1u : 0u;
        cnt += (int)(g >> 20) >= eb - kAdjSpread ? 0x10000u : 0u;
      }
      cnt = __reduce_add_sync(0xffffffffu, cnt);
      if (lane == 0) s_cnt[warp] = cnt;
      __syncthreads();
      cnt = 0;
#pragma unroll
      for (int w = 0; w < kAdjWarps; ++w) cnt += s_cnt[w];
      fixed = 16 * (cnt & 0xFFFFu) >= (1u << kv) && 16 * (cnt >> 16) >= (1u << kv);
    }
    if (fixed) {
#pragma unroll
      for (int u = 0; u < NA; ++u) {
        const uint32_t s = fix_slot((uint32_t)(tid + NT * u));
        tp[s] = make_longlong2(fix_from_double(__longlong_as_double(a[2 * u]), ea),
                               fix_from_double(__longlong_as_double(a[2 * u + 1]), ea));
        tl[s] = make_longlong2(fix_from_double(__longlong_as_double(b[2 * u]), eb),
                               fix_from_double(__longlong_as_double(b[2 * u + 1]), eb));
      }
      uint32_t pr[4] = {0, 0, 0, 0};
      uint32_t pbase = 0, cx = 0;
      int phase = -1;              // of the registers
      int halved = 0, na = 0, nb = 0;  // halvings so far: planned, and of each state
      const longlong2* ahead = nullptr;  // the entries of the table being fetched
      for (int o = 0; o < p.num_fix_ops; ++o) {
        const FixOp* op = fops + o;
        const int4 w0 = *reinterpret_cast<const int4*>(op);
        if (w0.x == FIX_ROT) {
          switch (w0.y & 3) {
            case 0:
              fix_rot_form<NA, 0>(a, w0.y, w0.z, w0.w);
              fix_rot_form<NA, 0>(b, w0.y, w0.z, w0.w);
              break;
            case 1:
              fix_rot_form<NA, 1>(a, w0.y, w0.z, w0.w);
              fix_rot_form<NA, 1>(b, w0.y, w0.z, w0.w);
              break;
            default:
              fix_rot_form<NA, 2>(a, w0.y, w0.z, w0.w);
              fix_rot_form<NA, 2>(b, w0.y, w0.z, w0.w);
              break;
          }
          if (w0.y & kFixShift) {
#pragma unroll
            for (int j = 0; j < 2 * NA; ++j) {
              a[j] >>= 1;
              b[j] >>= 1;
            }
            ++halved;
          }
        } else if (w0.x == FIX_GRAD) {
          FixSum g[3] = {};
          if (tid == 0) s_exp[w0.z] = 2 * halved + na + nb;
          switch (w0.y & 3) {
            case 0: fix_grad<0>(a, b, g); break;
            case 1: fix_grad<1>(a, b, g); break;
            default: fix_grad<2>(a, b, g); break;
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const long long h = warp_sum(g[c].h >> kGradShift);
            // units of 2^-26 of g.h: f < 8 x 2^26, so the sum is below 2^31
            const unsigned fr = g[c].f + (((unsigned)g[c].h & ((1u << kGradShift) - 1u)) << 26);
            const unsigned f = __reduce_add_sync(0xffffffffu, fr >> 5);
            if (lane == 0) {
              const int at_w = (w0.z * 3 + c) * kAdjWarps + warp;
              s_acc[at_w] = h;
              s_frac[at_w] = f;
            }
          }
        } else if (w0.x == FIX_TABLE) {
          // groups of two entries: wait for this one, then start the one after the next
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (g < 3) fix_copy_wait<1>();
            else fix_copy_wait<0>();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const longlong2 t = stage[NT * (2 * (g & 1) + j)];
              const int i = 2 * (2 * g + j);
              fix_phase(a[i], a[i + 1], t);
              fix_phase(b[i], b[i + 1], t);
            }
            if (g < 2) {
#pragma unroll
              for (int j = 0; j < 2; ++j) fix_copy16(stage + NT * (2 * g + j), ahead + NT * (2 * g + 4 + j));
              fix_copy_commit();
            }
          }
        } else if (w0.x == FIX_FETCH) {
          ahead = p.fix_tab + fix_slice(op, base, kAdjBits) + tid;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int j = 0; j < 2; ++j) fix_copy16(stage + NT * (2 * g + j), ahead + NT * (2 * g + j));
            fix_copy_commit();
          }
        } else if (w0.x == FIX_XOR) {
          if ((base >> w0.y) & 1) cx ^= (uint32_t)w0.z;
        } else {  // FIX_PHASE, FIX_END
          const int4 w1 = *(reinterpret_cast<const int4*>(op) + 1);
          if (phase >= 0) {
#pragma unroll
            for (int j = 0; j < NA; ++j) {
              unsigned char* q = adj_raw + fix_reg(pbase, pr, j);
              *reinterpret_cast<longlong2*>(q) = make_longlong2(a[2 * j], a[2 * j + 1]);
              *reinterpret_cast<longlong2*>(q + T * 16) = make_longlong2(b[2 * j], b[2 * j + 1]);
            }
            const int ta = __reduce_max_sync(0xffffffffu, fix_top(a)), tb = __reduce_max_sync(0xffffffffu, fix_top(b));
            if (lane == 0) {
              atomicMax(&s_top[0][phase % 3], ta);
              atomicMax(&s_top[1][phase % 3], tb);
            }
            // the next phase's words: last read before the barrier before this one
            if (tid < 2) s_top[tid][(phase + 1) % 3] = 0;
          }
          __syncthreads();
          const uint32_t img[6] = {(uint32_t)w0.y, (uint32_t)w0.z, (uint32_t)w0.w,
                                   (uint32_t)w1.x, (uint32_t)w1.y, (uint32_t)w1.z};
          // as byte offsets
          pr[0] = (img[0] & 0xFFFFu) << 4;
          pr[1] = img[0] >> 16 << 4;
          pr[2] = (img[1] & 0xFFFFu) << 4;
          cx ^= (uint32_t)op->a[8];
          pbase = cx;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t im = (i & 1) ? img[2 + i / 2] >> 16 : img[2 + i / 2] & 0xFFFFu;
            if ((tid >> i) & 1) pbase ^= im;
          }
          pbase <<= 4;
#pragma unroll
          for (int j = 0; j < NA; ++j) {
            const unsigned char* q = adj_raw + fix_reg(pbase, pr, j);
            const longlong2 v = *reinterpret_cast<const longlong2*>(q);
            const longlong2 w = *reinterpret_cast<const longlong2*>(q + T * 16);
            a[2 * j] = v.x;
            a[2 * j + 1] = v.y;
            b[2 * j] = w.x;
            b[2 * j + 1] = w.y;
          }
          if (phase >= 0) {
            const int sa = fix_renorm(s_top[0][phase % 3]), sb = fix_renorm(s_top[1][phase % 3]);
            fix_shift(a, sa);
            fix_shift(b, sb);
            na += sa;
            nb += sb;
          }
          ++phase;
        }
      }
      {  // the sums were written before the last barrier
        for (int o = tid; o < p.num_fix_ops; o += NT) {
          const FixOp* op = fops + o;
          if (op->kind != FIX_GRAD) continue;
          double f;
          memcpy(&f, &op->a[3], sizeof(f));
          // product of two fixed-point values / 2^64 -> product of the amplitudes
          const int e = ea + eb - 2 * 1079 + 64 + kGradShift + s_exp[op->a[1]];
          for (int c = 0; c < 3; ++c) {
            const int i = op->a[1] * 3 + c;
            long long h = 0, r = 0;
#pragma unroll
            for (int w = 0; w < kAdjWarps; ++w) {
              h += s_acc[i * kAdjWarps + w];
              r += s_frac[i * kAdjWarps + w];
            }
            s_sum[i] += scalbn(fma((double)r, 0x1p-25, (double)h) * f, e);
          }
        }
        const int ep = ea - 1079 + p.shifts + na + 1075 + p.scale_exp, el = eb - 1079 + p.shifts + nb + 1075 + p.scale_exp;
#pragma unroll
        for (int u = 0; u < NA; ++u) {
          if ((tid + NT * u) >> kv) continue;
          p.psi[at | s_slot[u]] = make_double2(fix_to_double(a[2 * u], ep), fix_to_double(a[2 * u + 1], ep));
          p.lam[at | s_slot[u]] = make_double2(fix_to_double(b[2 * u], el), fix_to_double(b[2 * u + 1], el));
        }
      }
    } else if (!zero) {
      double2* dp = reinterpret_cast<double2*>(tp);
      double2* dl = reinterpret_cast<double2*>(tl);
#pragma unroll
      for (int u = 0; u < NA; ++u) {
        tp[tid + NT * u] = make_longlong2(a[2 * u], a[2 * u + 1]);
        tl[tid + NT * u] = make_longlong2(b[2 * u], b[2 * u + 1]);
      }
      constexpr int kFit = (int)(kAdjStage / sizeof(Op));  // ops staged at a time
      for (int o = 0; o < p.num_ops; ++o) {
        if (o % kFit == 0) {
          __syncthreads();
          const int4* src = reinterpret_cast<const int4*>(p.ops + o);
          int4* dst = reinterpret_cast<int4*>(tl + T);
          for (int i = tid; i < min(kFit, p.num_ops - o) * (int)(sizeof(Op) / sizeof(int4)); i += NT) dst[i] = src[i];
          __syncthreads();
        }
        const Op& op = reinterpret_cast<const Op*>(tl + T)[o % kFit];
        if (op.ctrl_kind == CTRL_GLOBAL && !((base >> op.ctrl) & 1)) continue;  // uniform per tile
        if (op.cls == OP_GRAD) {
          double gx = 0.0, gy = 0.0, gz = 0.0;
          for (int q = tid; q < T / 2; q += NT) {
            const uint32_t i0 = insert_zero32((uint32_t)q, op.target), i1 = i0 | (1u << op.target);
            const double2 p0 = dp[i0], p1 = dp[i1], l0 = dl[i0], l1 = dl[i1];
            if (!any_bits(l0, l1) || !any_bits(p0, p1)) continue;
            gx += fma(l0.x, p1.y, -l0.y * p1.x) + fma(l1.x, p0.y, -l1.y * p0.x);
            gy += -fma(l0.x, p1.x, l0.y * p1.y) + fma(l1.x, p0.x, l1.y * p0.y);
            gz += fma(l0.x, p0.y, -l0.y * p0.x) - fma(l1.x, p1.y, -l1.y * p1.x);
          }
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) {
            gx += __shfl_xor_sync(0xffffffffu, gx, d);
            gy += __shfl_xor_sync(0xffffffffu, gy, d);
            gz += __shfl_xor_sync(0xffffffffu, gz, d);
          }
          if (lane == 0) {
            s_red[warp][0] = gx;
            s_red[warp][1] = gy;
            s_red[warp][2] = gz;
          }
          __syncthreads();
          if (tid < 3) {
            double s = 0.0;
            for (int w = 0; w < kAdjWarps; ++w) s += s_red[w][tid];
            s_sum[op.param * 3 + tid] += s * op.m[0];
          }
          __syncthreads();
          continue;
        }
        if (op.cls == OP_ROT) {
          tile_rot(dp, T, op);
          tile_rot(dl, T, op);
        } else if (op.cls == OP_PHASE) {
          tile_phase(dp, T, op, p.tab, base);
          tile_phase(dl, T, op, p.tab, base);
        } else {  // an exchange
          tile_op<PolF64, OP_SWAP>(dp, T, op);
          tile_op<PolF64, OP_SWAP>(dl, T, op);
        }
        __syncthreads();
      }
      __syncthreads();
      const double f = scalbn(1.0, p.scale_exp);
#pragma unroll
      for (int u = 0; u < NA; ++u) {
        if ((tid + NT * u) >> kv) continue;
        const double2 v = dp[tid + NT * u], w = dl[tid + NT * u];
        p.psi[at | s_slot[u]] = make_double2(v.x * f, v.y * f);
        p.lam[at | s_slot[u]] = make_double2(w.x * f, w.y * f);
      }
    }
    __syncthreads();
    if (tid < 6) s_top[tid / 3][tid % 3] = 0;
  }
  __syncthreads();
  for (int i = tid; i < 3 * p.num_grads; i += NT) p.partial[(int64_t)i * p.cols + blockIdx.x] = s_sum[i];
}

// A 2x2 product a b.
void mul2(const double a[8], const double b[8], double out[8]) { matmul2(a, b, out); }

// 1/2 Re tr(Q g P g^dagger), Q and P Paulis (0 X, 1 Y, 2 Z): how <P> after
// undoing g reads in terms of <Q> before.
double pauli_conjugate(const double g[8], int q, int p) {
  static const double pauli[3][8] = {{0, 0, 1, 0, 1, 0, 0, 0}, {0, 0, 0, -1, 0, 1, 0, 0}, {1, 0, 0, 0, 0, 0, -1, 0}};
  double gd[8], t[8], u[8];
  adjoint2(g, gd);
  mul2(pauli[p], gd, t);
  mul2(g, t, u);
  mul2(pauli[q], u, t);
  return 0.5 * (t[0] + t[6]);
}

struct AdjPass {
  Pass win;
  int64_t op_begin, op_count, fix_begin, fix_count;
  int32_t shifts, scale_exp, grad_begin, num_grads;
  double inv_c2;  // true product of the states / product of the stored ones, at the pass's start
};

struct AdjGrad {
  int32_t run, pass;
  int64_t frame;  // phase that psi and lambda carry on the set bit, in 2^-64 turns
};

}  // namespace

// The reverse sweep (see the file comment) from psi and lam, which it uses up.
// *done is false, and nothing ran, for gate lists it does not take (controls
// other than CNOT's, non-unitary matrices) and where its ops and tables, all
// reserved before the first launch, find no memory.
int adjoint_sweep_fix(dmv_state_s* s, dmv_state_s* psi, dmv_state_s* lam, const std::vector<Gate>& gates, double* grads,
                      bool* done) {
  *done = false;
  // The reversed gates and the slot of each one's parameter.
  std::vector<Gate> rev;
  std::vector<int32_t> slot, gen;
  int32_t slots = 0;
  for (const Gate& g : gates)
    if (!g.observable && is_parametrised(g.kind)) ++slots;
  for (int64_t gi = (int64_t)gates.size() - 1; gi >= 0; --gi) {
    const Gate& g = gates[(size_t)gi];
    if (g.observable) continue;
    if (g.control >= 0 && classify(g.m) != OP_SWAP) return DMV_OK;
    Gate h = g;
    adjoint2(g.m, h.m);
    rev.push_back(h);
    const bool p = is_parametrised(g.kind);
    if (p) --slots;
    slot.push_back(p ? slots : -1);
    gen.push_back(p ? rotation_generator(g.kind) : 0);
  }
  PlanOptions opt = plan_options_for(s, DMV_FUSE_WINDOW, true);
  opt.tile_bits = kAdjBits;
  opt.windows_only = true;
  std::vector<int32_t> run_of;
  opt.run_of = &run_of;
  opt.generator_of = gen.data();
  Plan plan;
  DMV_TRY(build_plan(rev, s->n, s->precision, opt, plan));

  std::vector<AdjPass> passes;
  std::vector<AdjGrad> meas;
  std::vector<Op> ops;
  std::vector<FixOp> fops;
  PhaseTables tabs;
  ScaleDD c;  // stored states = true ones times c
  for (const Pass& ps : plan.passes) {
    for (int64_t o = 0; o < ps.op_count;) {
      int64_t end = o;
      int32_t tagged = 0;
      while (end < ps.op_count && tagged < kAdjGrads) tagged += plan.ops[(size_t)(ps.op_begin + end++)].generator != 0;
      RewrittenPass r;
      rewrite_pass_rotations(plan.ops.data() + ps.op_begin + o, end - o, kAdjBits, true, r.ops, r.tab, &r.scale);
      AdjPass ap;
      ap.win = ps;
      ap.grad_begin = (int32_t)meas.size();
      ap.num_grads = 0;
      for (Op& op : r.ops)
        if (op.cls == OP_GRAD) {
          AdjGrad m;
          m.run = op.param;
          m.pass = (int32_t)passes.size();
          std::memcpy(&m.frame, op.fh, sizeof(m.frame));
          meas.push_back(m);
          op.param = ap.num_grads++;
        }
      ap.fix_begin = (int64_t)fops.size();
      if (!build_fix_pass(r.ops.data(), (int64_t)r.ops.size(), kAdjBits, fops, &ap.shifts)) return DMV_OK;
      ap.fix_count = (int64_t)fops.size() - ap.fix_begin;
      ap.op_begin = (int64_t)ops.size();
      ap.op_count = (int64_t)r.ops.size();
      if (tabs.entries + r.tab.entries > INT32_MAX) return DMV_OK;
      for (Op op : r.ops) {
        if (op.cls == OP_PHASE) op.fh[0] += (int32_t)tabs.entries;
        ops.push_back(op);
      }
      for (int64_t i = ap.fix_begin; i < (int64_t)fops.size(); ++i)
        if (fops[(size_t)i].kind == FIX_TABLE || fops[(size_t)i].kind == FIX_FETCH)
          fops[(size_t)i].a[0] += (int32_t)tabs.entries;
      for (PhaseTable t : r.tab.tables) {
        t.entry += tabs.entries;
        t.first_term += (int32_t)tabs.terms.size();
        tabs.tables.push_back(t);
      }
      tabs.terms.insert(tabs.terms.end(), r.tab.terms.begin(), r.tab.terms.end());
      tabs.entries += r.tab.entries;
      ap.inv_c2 = 1.0 / (c.hi * c.hi);
      // c / F times the power of two that brings it into [1, 2)
      const double F = r.scale.hi;
      ap.scale_exp = -std::ilogb(c.hi / F);
      c.mul(std::ldexp(1.0 / F, ap.scale_exp));
      passes.push_back(ap);
      o = end;
    }
  }

  DeviceBuffer &src = s->adj_src, &work = s->adj_work, &tab = s->adj_tab, &fix_tab = s->adj_fix_tab;
  std::vector<unsigned char> src_host;
  const int64_t tiles = int64_t(1) << std::max(0, s->n - kAdjBits);
  int sms = 0, per_sm = 0;
  DMV_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
  static const cudaError_t attr =
      cudaFuncSetAttribute(k_adjoint_fix, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAdjSmem);
  (void)attr;  // a refusal shows in the occupancy
  DMV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adjoint_fix, kAdjThreads, kAdjSmem));
  if (per_sm < 1) return set_error(DMV_ERR_CUDA, "adjoint kernel cannot fit %zu bytes of shared memory", kAdjSmem);
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)per_sm * sms);
  const size_t rows = 3 * meas.size();
  const size_t ops_bytes = ops.size() * sizeof(Op), fops_bytes = fops.size() * sizeof(FixOp);
  const size_t part_bytes = rows * (size_t)grid * sizeof(double), out_bytes = rows * sizeof(double);
  int rc = DMV_OK;
  std::vector<double> sums(rows);
  do {
    if ((rc = work.reserve(ops_bytes + fops_bytes + part_bytes + out_bytes)) != DMV_OK) break;
    if (tabs.entries > 0) {
      if ((rc = tab.reserve((size_t)tabs.entries * 16)) != DMV_OK) break;
      if ((rc = fix_tab.reserve((size_t)tabs.entries * 16)) != DMV_OK) break;
    }
    char* wp = static_cast<char*>(work.ptr);
    double* part = reinterpret_cast<double*>(wp + ops_bytes + fops_bytes);
    double* out = reinterpret_cast<double*>(wp + ops_bytes + fops_bytes + part_bytes);
    if (cudaMemcpyAsync(wp, ops.data(), ops_bytes, cudaMemcpyHostToDevice, s->stream) != cudaSuccess ||
        cudaMemcpyAsync(wp + ops_bytes, fops.data(), fops_bytes, cudaMemcpyHostToDevice, s->stream) != cudaSuccess) {
      rc = set_error(DMV_ERR_CUDA, "upload of the adjoint plan failed");
      break;
    }
    if (tabs.entries > 0) {
      PhaseTableForms forms;
      forms.f64 = static_cast<double2*>(tab.ptr);
      forms.fix = static_cast<longlong2*>(fix_tab.ptr);
      if ((rc = make_phase_tables(tabs, fops, forms, src_host, src, s->stream)) != DMV_OK) break;
    }
    for (const AdjPass& ap : passes) {
      AdjFixParams p;
      p.psi = static_cast<double2*>(psi->amps);
      p.lam = static_cast<double2*>(lam->amps);
      p.low = ap.win.low_bits;
      p.nh = ap.win.num_high;
      for (int i = 0; i < 16; ++i) p.high[i] = i < p.nh ? ap.win.high[i] : 0;
      p.num_tiles = (int32_t)tiles;
      p.num_ops = (int32_t)ap.op_count;
      p.num_fix_ops = (int32_t)ap.fix_count;
      p.num_grads = ap.num_grads;
      p.shifts = ap.shifts;
      p.scale_exp = ap.scale_exp;
      p.ops = reinterpret_cast<const Op*>(wp) + ap.op_begin;
      p.tab = static_cast<const double2*>(tab.ptr);
      p.fix_ops = reinterpret_cast<const FixOp*>(wp + ops_bytes) + ap.fix_begin;
      p.fix_tab = static_cast<const longlong2*>(fix_tab.ptr);
      p.partial = part + (size_t)3 * ap.grad_begin * grid;
      p.cols = grid;
      const int64_t tok = prof_begin(DMV_KERNEL_ADJOINT, s->stream, 4.0 * (double)psi->amp_bytes());
      k_adjoint_fix<<<grid, kAdjThreads, kAdjSmem, s->stream>>>(p);
      prof_end(tok, s->stream);
      count_launch();
    }
    if (rows > 0) {
      if ((rc = launch_reduce_rows(part, (int64_t)rows, grid, out, s->stream)) != DMV_OK) break;
      if (cudaMemcpyAsync(sums.data(), out, out_bytes, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess) {
        rc = set_error(DMV_ERR_CUDA, "gradient readback failed");
        break;
      }
    }
    if (cudaStreamSynchronize(s->stream) != cudaSuccess) rc = set_error(DMV_ERR_CUDA, "adjoint sweep failed");
  } while (false);
  if (rc == DMV_ERR_OOM) {
    clear_error();
    for (DeviceBuffer* b : {&src, &work, &tab, &fix_tab}) b->release();
    return DMV_OK;
  }
  DMV_TRY(rc);

  // The parameters of each run from its three sums.
  std::vector<int64_t> first_of_run;
  for (size_t i = 0; i < rev.size(); ++i)
    if ((size_t)run_of[i] >= first_of_run.size()) first_of_run.resize((size_t)run_of[i] + 1, -1);
  for (size_t i = rev.size(); i-- > 0;) first_of_run[(size_t)run_of[i]] = (int64_t)i;
  for (size_t m = 0; m < meas.size(); ++m) {
    const double k = passes[(size_t)meas[m].pass].inv_c2;
    const double mx = sums[3 * m] * k, my = sums[3 * m + 1] * k;
    const double ang = (double)meas[m].frame * (M_PI * 0x1p-63);
    double v[3] = {std::cos(ang) * mx + std::sin(ang) * my, -std::sin(ang) * mx + std::cos(ang) * my, sums[3 * m + 2] * k};
    for (size_t i = (size_t)first_of_run[(size_t)meas[m].run]; i < rev.size(); ++i) {
      if (run_of[i] != meas[m].run) continue;
      if (slot[i] >= 0) grads[(size_t)slot[i]] = v[gen[i] - 1];
      double g[8], u[3];
      adjoint2(rev[i].m, g);
      for (int pp = 0; pp < 3; ++pp)
        u[pp] = pauli_conjugate(g, 0, pp) * v[0] + pauli_conjugate(g, 1, pp) * v[1] + pauli_conjugate(g, 2, pp) * v[2];
      std::memcpy(v, u, sizeof(u));
    }
  }
  *done = true;
  return DMV_OK;
}

}  // namespace dmv
