// Window pass of complex64 states as rotations, phase tables and exchanges
// (rewrite_pass_rotations), in the fixed-point pass's register phases
// (build_fix_pass) with FP32 arithmetic.
//
// k_window_phases applies each gate as a complex 2x2: 8 multiply-adds per
// amplitude, an exchange as register moves under a predicate, and a pass of
// the 27-qubit, 20-layer forward took 2.3 ms against 0.3 for its bytes. Here a
// rotation is 2 multiply-adds per amplitude, a phase table 4 for all the
// diagonal factors of a level, and an exchange nothing.
//
// 256 threads hold 16 amplitudes each (32 of 80 registers), so that three CTAs
// fit an SM and some load or store while others compute; the loads go straight
// to registers (16 of 8 bytes in flight per thread), 128 bytes of consecutive
// amplitudes at a time. A table's entries are read in the order of the threads
// and registers, two to a load.

constexpr int kF32Threads = 256;
constexpr int kF32ThreadBits = 8;
constexpr int kF32Amps = 16;

struct F32PassParams {
  float2* amps;
  int32_t low, nh;
  int32_t high[16];
  int32_t num_ops;
  float out_scale;  // the state leaves the pass times this
  int64_t num_tiles;
  const FixOp* ops;
  const float2* tab;
};

constexpr size_t kF32Smem = ((size_t)8 << 12) + kFixSmemOps * sizeof(FixOp);

__device__ __forceinline__ uint32_t fix_slot8(uint32_t l) { return l ^ (((l >> 4) ^ (l >> 8)) & 15u); }

template <int TP>
__device__ __forceinline__ void f32_rot(float2 (&r)[kF32Amps], float w) {
#pragma unroll
  for (int j = 0; j < kF32Amps; ++j) {
    if (j & (1 << TP)) continue;
    const float2 a = r[j], b = r[j | (1 << TP)];
    r[j] = make_float2(fmaf(-w, b.x, a.x), fmaf(-w, b.y, a.y));
    r[j | (1 << TP)] = make_float2(fmaf(w, a.x, b.x), fmaf(w, a.y, b.y));
  }
}

// r times the 16 phases at e (kF32Threads float4 apart, two entries each).
__device__ __forceinline__ void f32_table(float2 (&r)[kF32Amps], const float4* e) {
#pragma unroll
  for (int g = 0; g < kF32Amps / 2; g += 4) {
    float4 t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = __ldg(e + kF32Threads * (g + j));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 &a = r[2 * (g + j)], &b = r[2 * (g + j) + 1];
      a = make_float2(fmaf(t[j].x, a.x, -t[j].y * a.y), fmaf(t[j].x, a.y, t[j].y * a.x));
      b = make_float2(fmaf(t[j].z, b.x, -t[j].w * b.y), fmaf(t[j].z, b.y, t[j].w * b.x));
    }
  }
}

// A whole phase of a table (TAB) and rotations on register bits 0 .. M - 1 in
// straight-line code, shared memory to shared memory: applied op by op in a
// loop, every op ends with its 32 registers moved to where the next expects
// them, as many moves as multiply-adds. `op`: the phase's first op.
template <int M, bool TAB>
__device__ __forceinline__ void f32_phase(unsigned char* tile, uint32_t pbase, const uint32_t (&pr)[4], const FixOp* op,
                                          const float2* tab, int64_t base) {
  float2 r[kF32Amps];
#pragma unroll
  for (int j = 0; j < kF32Amps; ++j) r[j] = *reinterpret_cast<const float2*>(tile + fix_reg(pbase, pr, j));
  if constexpr (TAB) f32_table(r, reinterpret_cast<const float4*>(tab + fix_slice(op, base, 12)) + threadIdx.x);
  const FixOp* rot = op + (TAB ? 1 : 0);
  if constexpr (M > 0) f32_rot<0>(r, __int_as_float(rot[0].a[1]));
  if constexpr (M > 1) f32_rot<1>(r, __int_as_float(rot[1].a[1]));
  if constexpr (M > 2) f32_rot<2>(r, __int_as_float(rot[2].a[1]));
  if constexpr (M > 3) f32_rot<3>(r, __int_as_float(rot[3].a[1]));
#pragma unroll
  for (int j = 0; j < kF32Amps; ++j) *reinterpret_cast<float2*>(tile + fix_reg(pbase, pr, j)) = r[j];
}

__global__ void __launch_bounds__(kF32Threads, 3) k_window_f32(const __grid_constant__ F32PassParams p) {
  constexpr int NT = kF32Threads, NA = kF32Amps, k = 12, T = 1 << k;
  extern __shared__ __align__(16) unsigned char f32_raw[];
  __shared__ int64_t s_slot[NA];
  float2* tile = reinterpret_cast<float2*>(f32_raw);
  const int tid = (int)threadIdx.x;
  const FixOp* ops = p.ops;
  const int low = p.low, nh = p.nh;
  int64_t t_off = (int64_t)(tid & ((1 << low) - 1));
  const int from_tid = min(nh, kF32ThreadBits - low);
  for (int i = 0; i < from_tid; ++i) t_off |= (int64_t)((tid >> (low + i)) & 1) << p.high[i];
  if (tid < NA) {
    int64_t off = 0;
    for (int i = from_tid; i < nh; ++i) off |= (int64_t)((tid >> (i - from_tid)) & 1) << p.high[i];
    s_slot[tid] = off;
  }
  if (p.num_ops <= kFixSmemOps) {
    int4* dst = reinterpret_cast<int4*>(tile + T);
    const int4* src = reinterpret_cast<const int4*>(p.ops);
    for (int i = tid; i < p.num_ops * 3; i += NT) dst[i] = src[i];
    ops = reinterpret_cast<const FixOp*>(dst);
  }
  __syncthreads();
  for (int64_t tix = blockIdx.x; tix < p.num_tiles; tix += gridDim.x) {
    int64_t base = tix << low;
    for (int i = 0; i < nh; ++i) base = insert_zero(base, p.high[i]);
    float2* at = p.amps + (base | t_off);
    {
      float2 r[NA];
#pragma unroll
      for (int u = 0; u < NA; ++u) r[u] = at[s_slot[u]];
#pragma unroll
      for (int u = 0; u < NA; ++u) tile[fix_slot8((uint32_t)(tid + NT * u))] = r[u];
    }
    uint32_t cx = 0;
    for (int o = 0;; ++o) {
      const FixOp* op = ops + o;
      const int4 w0 = *reinterpret_cast<const int4*>(op);
      if (w0.x == FIX_XOR) {
        if ((base >> w0.y) & 1) cx ^= (uint32_t)w0.z;
        continue;
      }
      // FIX_PHASE, FIX_END
      const int4 w1 = *(reinterpret_cast<const int4*>(op) + 1);
      const int4 w2 = *(reinterpret_cast<const int4*>(op) + 2);
      __syncthreads();
      const uint32_t img[6] = {(uint32_t)w0.y, (uint32_t)w0.z, (uint32_t)w0.w,
                               (uint32_t)w1.x, (uint32_t)w1.y, (uint32_t)w1.z};
      // as byte offsets
      const uint32_t pr[4] = {(img[0] & 0xFFFFu) << 3, img[0] >> 16 << 3, (img[1] & 0xFFFFu) << 3, img[1] >> 16 << 3};
      cx ^= (uint32_t)w2.y;
      uint32_t pbase = cx;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const uint32_t im = (b & 1) ? img[2 + b / 2] >> 16 : img[2 + b / 2] & 0xFFFFu;
        if ((tid >> b) & 1) pbase ^= im;
      }
      pbase <<= 3;
      if (w0.x == FIX_END) {
        float2 r[NA];
#pragma unroll
        for (int j = 0; j < NA; ++j) r[j] = *reinterpret_cast<const float2*>(f32_raw + fix_reg(pbase, pr, j));
#pragma unroll
        for (int u = 0; u < NA; ++u) at[s_slot[u]] = make_float2(r[u].x * p.out_scale, r[u].y * p.out_scale);
        break;
      }
      const int kind = w2.z & (kFixSimple - 1);
      if (w2.z) {
        switch (kind) {
          case 1: f32_phase<1, false>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case 2: f32_phase<2, false>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case 3: f32_phase<3, false>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case 4: f32_phase<4, false>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case kFixSimpleTable: f32_phase<0, true>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case kFixSimpleTable + 1: f32_phase<1, true>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case kFixSimpleTable + 2: f32_phase<2, true>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          case kFixSimpleTable + 3: f32_phase<3, true>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
          default: f32_phase<4, true>(f32_raw, pbase, pr, op + 1, p.tab, base); break;
        }
        o += (kind & kFixSimpleTable ? 1 : 0) + (kind & (kFixSimpleTable - 1));
        continue;
      }
      float2 r[NA];
#pragma unroll
      for (int j = 0; j < NA; ++j) r[j] = *reinterpret_cast<const float2*>(f32_raw + fix_reg(pbase, pr, j));
      for (;; ++o) {
        const FixOp* q = ops + o + 1;
        const int4 v0 = *reinterpret_cast<const int4*>(q);
        if (v0.x == FIX_ROT) {
          const float w = __int_as_float(v0.z);
          switch (v0.y & 3) {
            case 0: f32_rot<0>(r, w); break;
            case 1: f32_rot<1>(r, w); break;
            case 2: f32_rot<2>(r, w); break;
            default: f32_rot<3>(r, w); break;
          }
        } else if (v0.x == FIX_TABLE) {
          f32_table(r, reinterpret_cast<const float4*>(p.tab + fix_slice(q, base, k)) + tid);
        } else {
          break;
        }
      }
#pragma unroll
      for (int j = 0; j < NA; ++j) *reinterpret_cast<float2*>(f32_raw + fix_reg(pbase, pr, j)) = r[j];
    }
    __syncthreads();  // every thread has read its last slots
  }
}
