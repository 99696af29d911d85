// Fixed-point window pass (complex128 storage): the FP64 pass's rotations and
// phase tables (rewrite_pass_rotations) as 64-bit integer arithmetic.
//
// GB300 issues an FP64 multiply-add from one warp every ~77 cycles per SM
// quarter, a 32 x 32 -> 64-bit integer one every few. So a tile of 2^12
// amplitudes is turned into integers under one exponent: the largest
// component gets 57 bits, and a rotation output x0 - w x1 (the same f M form
// as OP_ROT) is three integer multiply-adds and one rounding to the last bit,
// 2^-57 of the tile's largest component: in the norm of the tile, as long as it
// is no more than a few times its average (FixScan::heavy), less than FP64's
// roundings. The ops run in register phases (build_fix_pass):
// 256 threads hold 16 amplitudes each, the tile crosses shared memory once per
// phase, exchanges cost nothing (they re-index the tile).
//
// Which tiles. Fixed point keeps less of a component the smaller it is, so a
// tile runs in it only when every amplitude is within 2^kFixRange of its
// largest one (entangled states: all but one tile in a few hundred) and their
// squares are not those of a few (FixScan::heavy). Any
// other tile (product states, exact zeros, infinities, NaN) takes the pass's
// ops in shared memory in the arithmetic FB (FP64, or FP32 pairs for states of
// that arithmetic). A tile of zeros is left as it is.
//
// An exact zero is in range where the pass's rotations spread no further than
// that (build_fix_pass's `sparse`): the tiles of a state that has not reached
// its last qubits yet.
//
// Headroom. A component of the tile can grow: every phase takes the largest
// when it is written back, and the next shifts all of them below 2^58. 16
// amplitudes of that size have a norm below 2^60.5, and inside a phase the
// stored norm grows at most 2 sqrt 2 times (kFixShift halves it), so no sum
// leaves 63 bits.

struct FixPassParams {
  TmaPassParams t;
  const FixOp* fix_ops;
  const longlong2* fix_tab;
  int32_t num_fix_ops;
  int32_t shifts;  // halvings over the whole pass
  uint32_t sparse; // numbers of unreached qubits a fixed-point tile may have (build_fix_pass)
};

template <typename FB>
__global__ void __launch_bounds__(kFixThreads, 2)
k_window_fix(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ FixPassParams fp) {
  constexpr int NT = kFixThreads;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_scan[5][NT / 32];
  __shared__ int s_high[16];
  __shared__ int64_t s_slot[kFixAmps];
  __shared__ int s_top[3];  // largest component, by phase
  const TmaPassParams& p = fp.t;
  unsigned char* tile =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int k = 12, T = 1 << k;
  constexpr uint32_t tile_bytes = (uint32_t)T * 16u;
  const int low = p.low, nh = p.nh, boxes = p.boxes;
  const int64_t num_tiles = p.num_tiles;
  const int tid = (int)threadIdx.x;
  if (tid < 16) s_high[tid] = p.high[tid];
  if (tid == 0) {
    s_top[0] = s_top[1] = s_top[2] = 0;
    mbar_init(&s_bar, 1);
    fence_mbar_init();
    tma_prefetch_map(&tmap);
  }
  // offset in HBM of element tid + 256 u: the thread's part and the slots' parts
  int64_t t_off = (int64_t)(tid & ((1 << low) - 1));
  const int from_tid = min(nh, kFixThreadBits - low);
  for (int i = 0; i < from_tid; ++i) t_off |= (int64_t)((tid >> (low + i)) & 1) << p.high[i];
  if (tid < kFixAmps) {
    int64_t off = 0;
    for (int i = from_tid; i < nh; ++i) off |= (int64_t)((tid >> (i - from_tid)) & 1) << p.high[i];
    s_slot[tid] = off;
  }
  __syncthreads();
  const TileGeom<16> geom{low, nh, s_high};
  const int lane = tid & 31;
  const bool mover = tid < 32;  // warp 0 issues the loads
  double2* amps = static_cast<double2*>(p.amps);
  longlong2* ti = reinterpret_cast<longlong2*>(tile);
  // Table entries on their way: two groups of four per thread, its own slots.
  longlong2* stage = ti + T + tid;
  const FixOp* ops = fp.fix_ops;
  if (fp.num_fix_ops <= kFixSmemOps) {
    int4* dst = reinterpret_cast<int4*>(ti + T + 8 * NT);
    const int4* src = reinterpret_cast<const int4*>(fp.fix_ops);
    for (int i = tid; i < fp.num_fix_ops * 3; i += NT) dst[i] = src[i];
    ops = reinterpret_cast<const FixOp*>(dst);
  }

  int64_t tix = blockIdx.x;
  uint32_t parity = 0;
  if (mover && tix < num_tiles) geom.load(&tmap, &s_bar, tile, tix, boxes, tile_bytes, lane);
  while (tix < num_tiles) {
    const bool ok = mbar_wait(&s_bar, parity, p.wait_limit);
    if (__syncthreads_or(!ok)) {
      if (mover) {
        if (lane == 0) atomicExch(p.status, 1);
        mbar_wait(&s_bar, parity, kTmaDrainLimit);  // drain the one load in flight
      }
      return;
    }
    parity ^= 1u;
    const int64_t base = geom.base(tix);
    const int64_t next = tix + gridDim.x;
    long long r[2 * kFixAmps];
#pragma unroll
    for (int u = 0; u < kFixAmps; ++u) {
      const longlong2 v = ti[tid + NT * u];
      r[2 * u] = v.x;
      r[2 * u + 1] = v.y;
    }
    constexpr bool MASS = std::is_same<FB, PolF64>::value;  // FP32 pairs round more coarsely than any fixed-point tile
    const FixScan scan = fix_scan<MASS>(r, s_scan);
    const int emax = scan.emax();
    const bool zero = scan.zero();
    const bool fixed = scan.fixed(fp.sparse) && (!MASS || scan.heavy());
    int e_out = 0;
    const bool store = !zero;
    if (fixed) {
      fix_put(r, tile, emax);
      const int renorm = fix_run(r, tile, stage, ops, fp.num_fix_ops, fp.fix_tab, base, s_top);
      e_out = emax - 1079 + fp.shifts + renorm + 1075;
    } else if (!zero) {
      using V = typename FB::T;
      static_assert(sizeof(V) == 16, "the tile is converted in place");
      V* tv = reinterpret_cast<V*>(tile);
      if constexpr (!std::is_same<V, double2>::value) {
#pragma unroll
        for (int u = 0; u < kFixAmps; ++u)
          tv[tid + NT * u] = FB::in(make_double2(__longlong_as_double(r[2 * u]), __longlong_as_double(r[2 * u + 1])));
      }
      tile_apply_ops_staged<FB>(tv, T, p.ops, p.num_ops, base, p.phase_tab, ti + T, (int)kFixStage);
#pragma unroll
      for (int u = 0; u < kFixAmps; ++u) {
        const double2 v = FB::out(tv[tid + NT * u]);
        r[2 * u] = __double_as_longlong(v.x);
        r[2 * u + 1] = __double_as_longlong(v.y);
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) s_top[0] = s_top[1] = s_top[2] = 0;
    if (mover && next < num_tiles) geom.load(&tmap, &s_bar, tile, next, boxes, tile_bytes, lane);
    if (store) {
      const int64_t at = base | t_off;
#pragma unroll
      for (int u = 0; u < kFixAmps; ++u) {
        double2 v;
        if (fixed) v = make_double2(fix_to_double(r[2 * u], e_out), fix_to_double(r[2 * u + 1], e_out));
        else v = make_double2(__longlong_as_double(r[2 * u]), __longlong_as_double(r[2 * u + 1]));
        amps[at | s_slot[u]] = v;
      }
    }
    tix = next;
  }
}
