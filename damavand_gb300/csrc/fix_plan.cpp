// Fixed-point window passes (host C++): a rewritten pass's ops scheduled into
// register phases (fix_window.cuh has the kernel).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "internal.h"

namespace dmv {
namespace {

constexpr int kMaxTileBits = 12;
constexpr int kThreadBits = 8;
constexpr int kMaxFixRegBits = kMaxTileBits - kThreadBits;

// The linear map l -> fix_slot(A l): images of the tile bits.
struct SlotMap {
  int32_t img[kMaxTileBits];
};

// Rank over GF(2) of the slots v modulo a row of 2^row_bits.
int row_rank(const int32_t* v, int n, int row_bits) {
  int32_t basis[4] = {0, 0, 0, 0};
  int r = 0;
  for (int i = 0; i < n; ++i) {
    int32_t x = v[i] & ((1 << row_bits) - 1);
    for (int b = row_bits - 1; b >= 0; --b)
      if ((x >> b) & 1) {
        if (basis[b]) x ^= basis[b];
        else {
          basis[b] = x;
          ++r;
          break;
        }
      }
  }
  return r;
}

void pack_images(FixOp& op, const int32_t* slot12) {
  for (int i = 0; i < 6; ++i) op.a[i] = slot12[2 * i] | (slot12[2 * i + 1] << 16);
}

// Thread bits of a phase: the tile bits outside `regs`, the first row_bits
// chosen so that the lanes of one 128-byte access meet all 32 banks (their
// slots differ in as many independent ways modulo a row).
void thread_bits(const SlotMap& m, int tile_bits, int row_bits, uint32_t regs, int32_t* bits) {
  int n = 0;
  uint32_t used = regs;
  int32_t pick[4];
  for (int b = 0; b < tile_bits && n < row_bits; ++b) {
    if ((used >> b) & 1u) continue;
    pick[n] = m.img[b];
    if (row_rank(pick, n + 1, row_bits) != n + 1) continue;
    bits[n++] = b;
    used |= 1u << b;
  }
  for (int b = 0; b < tile_bits; ++b)
    if (!((used >> b) & 1u)) bits[n++] = b;
}

// w 2^64 as signed words hi 2^32 + lo; false when hi would not fit 31 bits
// (w within 2^-32 of 1/2 from below, or w >= 1/2).
bool split_multiplier(double w, int32_t& hi, int32_t& lo) {
  if (!(w >= 0.0) || w >= 0.5) return false;
  const uint64_t W = (uint64_t)std::nearbyint(std::ldexp(w, 64));
  const uint64_t h = (W >> 32) + ((W >> 31) & 1u);
  if (h >= 0x80000000ull) return false;
  hi = (int32_t)h;
  lo = (int32_t)(uint32_t)W;
  return true;
}

}  // namespace

bool build_fix_pass(const Op* ops, int64_t count, int32_t tile_bits, std::vector<FixOp>& out, int32_t* shifts,
                    uint32_t* sparse, bool single) {
  const int32_t reg_bits = tile_bits - kThreadBits;
  const uint32_t all_bits = (1u << tile_bits) - 1u;
  const size_t mark = out.size();
  *shifts = 0;
  SlotMap m;
  for (int b = 0; b < tile_bits; ++b) m.img[b] = single ? fix_slot8_host(1 << b) : fix_slot_host(1 << b);
  auto blank = [](int32_t kind) {
    FixOp f;
    std::memset(&f, 0, sizeof(f));
    f.kind = kind;
    return f;
  };
  int32_t flip = 0;  // offset the next FIX_PHASE or FIX_END adds on every tile
  // An exchange takes effect at the front of the phase being built.
  auto exchange = [&](const Op& op) {
    if (op.ctrl_kind == CTRL_LOCAL) {
      m.img[op.ctrl] ^= m.img[op.target];
      return;
    }
    if (op.ctrl_kind == CTRL_NONE) {
      flip ^= m.img[op.target];
      return;
    }
    FixOp f = blank(FIX_XOR);
    f.a[0] = op.ctrl;
    f.a[1] = m.img[op.target];
    out.push_back(f);
  };
  // The stored state is the true one times `grown`, kept in (1/sqrt 2, sqrt 2].
  double grown = 1.0;
  double least[16];  // per tile bit, its least rotation multiplier
  for (double& w : least) w = 1.0;
  double factor = 1.0;  // of the rotations so far (FIX_GRAD)
  std::vector<char> done((size_t)count, 0);
  std::vector<FixOp> taken;
  int64_t left = count, first = 0;
  while (left > 0) {
    while (done[(size_t)first]) ++first;
    int32_t reg[kMaxFixRegBits];
    int nr = 0;
    uint32_t regs = 0, blocked = 0, used = 0;
    taken.clear();
    for (int64_t i = first; i < count && blocked != all_bits; ++i) {
      if (done[(size_t)i]) continue;
      const Op& op = ops[i];
      const uint32_t tb = 1u << op.target;
      if (op.cls == OP_SWAP) {
        const uint32_t qs = tb | (op.ctrl_kind == CTRL_LOCAL ? 1u << op.ctrl : 0u);
        if (qs & (blocked | used)) {
          blocked |= qs;
          continue;
        }
        exchange(op);
      } else if (op.cls == OP_PHASE) {
        const uint32_t qs = (uint32_t)op.fh[5];
        if (qs & blocked) {
          blocked |= qs;
          continue;
        }
        FixOp f = blank(FIX_TABLE);
        f.a[0] = op.fh[0];
        f.a[1] = op.fh[1];
        for (int j = 0; j < op.fh[1]; ++j) f.a[2 + j] = op.fh[2 + j];
        used |= qs;
        taken.push_back(f);
      } else if ((op.cls == OP_ROT || op.cls == OP_GRAD) && op.ctrl_kind == CTRL_NONE) {
        if (tb & blocked) continue;
        if (!(regs & tb)) {
          if (nr == reg_bits) {
            blocked |= tb;
            continue;
          }
          reg[nr++] = op.target;
          regs |= tb;
        }
        used |= tb;
        done[(size_t)i] = 1;
        --left;
        if (op.cls == OP_GRAD) {
          FixOp f = blank(FIX_GRAD);
          f.a[0] = op.target;
          f.a[1] = op.param;
          const double sq = factor * factor;
          std::memcpy(&f.a[3], &sq, sizeof(sq));
          taken.push_back(f);
          continue;
        }
        FixOp f = blank(FIX_ROT);
        f.a[0] = op.target;  // the register bit once the phase is complete
        const double w = op.m[0];
        if (w != 0.0) least[op.target] = std::min(least[op.target], std::fabs(w));
        if (single) {
          const float wf = (float)w;
          std::memcpy(&f.a[1], &wf, sizeof(wf));
          taken.push_back(f);
          continue;
        }
        if (!split_multiplier(w, f.a[1], f.a[2])) {
          f.a[0] |= kFixComplement << 8;
          if (!split_multiplier(1.0 - w, f.a[1], f.a[2])) {
            out.resize(mark);
            return false;
          }
        }
        grown *= std::sqrt(1.0 + w * w);
        factor /= std::sqrt(1.0 + w * w);
        if (grown > 1.4142135623730951) {
          f.a[0] |= kFixShift << 8;
          grown *= 0.5;
          ++*shifts;
        }
        taken.push_back(f);
        continue;
      } else {
        out.resize(mark);
        return false;
      }
      done[(size_t)i] = 1;
      --left;
    }
    if (taken.empty()) continue;
    // unused register bits from the top: the low ones serve the lanes
    for (int b = tile_bits - 1; nr < reg_bits; --b)
      if (!((regs >> b) & 1u)) {
        reg[nr++] = b;
        regs |= 1u << b;
      }
    int32_t tbits[kThreadBits], slots[kMaxTileBits] = {};
    thread_bits(m, tile_bits, single ? 4 : 3, regs, tbits);
    FixOp ph = blank(FIX_PHASE);
    for (int i = 0; i < reg_bits; ++i) slots[i] = m.img[reg[i]];
    for (int i = 0; i < kThreadBits; ++i) slots[kMaxFixRegBits + i] = m.img[tbits[i]];
    pack_images(ph, slots);
    uint32_t tpos = 0, rpos = 0;
    for (int i = 0; i < kThreadBits; ++i) tpos |= (uint32_t)tbits[i] << (4 * i);
    for (int i = 0; i < reg_bits; ++i) rpos |= (uint32_t)reg[i] << (4 * i);
    ph.a[6] = (int32_t)tpos;
    ph.a[7] = (int32_t)rpos;
    ph.a[8] = flip;
    flip = 0;
    // at most one table, then rotations on register bits 0, 1, ... once each
    {
      const size_t t0 = taken[0].kind == FIX_TABLE ? 1 : 0;
      bool simple = taken.size() - t0 <= (size_t)reg_bits;
      for (size_t i = t0; i < taken.size(); ++i)
        simple = simple && taken[i].kind == FIX_ROT && (taken[i].a[0] & 15) == reg[i - t0];
      if (simple) ph.a[9] = kFixSimple | (t0 ? kFixSimpleTable : 0) | (int32_t)(taken.size() - t0);
    }
    out.push_back(ph);
    for (FixOp& f : taken) {
      if (f.kind == FIX_ROT || f.kind == FIX_GRAD) {
        const int32_t t = f.a[0] & 15, flags = f.a[0] >> 8;
        int32_t b = 0;
        while (reg[b] != t) ++b;
        f.a[0] = b | flags;
      }
      out.push_back(f);
    }
  }
  if (sparse) {
    std::sort(least, least + tile_bits);
    double p = 1.0;
    *sparse = 1u;
    for (int z = 1; z <= tile_bits; ++z) {
      p *= least[z - 1];
      if (z <= kFixUnreached && p >= std::ldexp(1.0, -kFixRange)) *sparse |= 1u << z;
    }
  }
  FixOp end = blank(FIX_END);
  int32_t slots[kMaxTileBits] = {};
  for (int i = 0; i < reg_bits; ++i) slots[i] = m.img[kThreadBits + i];
  for (int i = 0; i < kThreadBits; ++i) slots[kMaxFixRegBits + i] = m.img[i];
  pack_images(end, slots);
  end.a[8] = flip;
  out.push_back(end);
  if (single) return true;
  // Each table's first entries load from the moment the one before it is done.
  std::vector<FixOp> body(out.begin() + (std::ptrdiff_t)mark, out.end());
  out.resize(mark);
  auto fetch = [&](size_t from) {
    for (size_t i = from; i < body.size(); ++i)
      if (body[i].kind == FIX_TABLE) {
        FixOp f = body[i];
        f.kind = FIX_FETCH;
        out.push_back(f);
        return;
      }
  };
  fetch(0);
  for (size_t i = 0; i < body.size(); ++i) {
    out.push_back(body[i]);
    if (body[i].kind == FIX_TABLE) fetch(i + 1);
  }
  return true;
}

}  // namespace dmv

// ---------------------------------------------------------------------------
// Host view of the scheduled passes (dmv_debug_fix_plan), for a test that runs
// them next to the ops they come from.
// ---------------------------------------------------------------------------
extern "C" int dmv_debug_fix_plan(const dmv_gate_t* gates, int64_t num_gates, int32_t num_qubits, int32_t form,
                                  int64_t capacity, int64_t* words, int64_t* count) {
  using namespace dmv;
  clear_error();
  if (!words || !count || form < 0 || form > 2) return set_error(DMV_ERR_INVALID, "dmv_debug_fix_plan: bad arguments");
  std::vector<Gate> g;
  DMV_TRY(parse_gates(gates, num_gates, num_qubits, g));
  dmv_state_s probe;
  probe.n = num_qubits;
  probe.precision = form == 2 ? DMV_C64 : DMV_C128;
  PlanOptions opt = plan_options_for(&probe, DMV_FUSE_WINDOW, form == 1);
  std::vector<int32_t> run_of, gen;
  if (form == 1) {  // a gradient's windows, every gate's run measured
    opt.tile_bits = 11;
    opt.windows_only = true;
    for (const Gate& x : g) gen.push_back(x.control < 0 ? 1 : 0);
    opt.run_of = &run_of;
    opt.generator_of = gen.data();
  }
  Plan plan;
  DMV_TRY(build_plan(g, num_qubits, probe.precision, opt, plan));
  std::vector<int64_t> w;
  auto bits = [](double x) {
    int64_t i;
    std::memcpy(&i, &x, sizeof(i));
    return i;
  };
  for (const Pass& ps : plan.passes) {
    const int32_t k = ps.low_bits + ps.num_high;
    if (ps.kind != 1 || k != opt.tile_bits) continue;
    RewrittenPass r;
    rewrite_pass_rotations(plan.ops.data() + ps.op_begin, ps.op_count, k, true, r.ops, r.tab, &r.scale, form == 2);
    std::vector<FixOp> fops;
    int32_t shifts = 0;
    const bool taken = build_fix_pass(r.ops.data(), (int64_t)r.ops.size(), k, fops, &shifts, nullptr, form == 2);
    w.insert(w.end(), {ps.low_bits, ps.num_high});
    w.insert(w.end(), ps.high, ps.high + ps.num_high);
    w.insert(w.end(), {ps.op_count, taken ? 1 : 0, (int64_t)fops.size(), (int64_t)r.tab.tables.size(),
                       (int64_t)r.tab.terms.size(), shifts, bits(r.scale.hi)});
    for (int64_t o = 0; o < ps.op_count; ++o) {
      const Op& op = plan.ops[(size_t)(ps.op_begin + o)];
      w.insert(w.end(), {op.target, op.ctrl, op.ctrl_kind, op.param, op.generator});
      for (double x : op.m) w.push_back(bits(x));
    }
    const size_t at = w.size();
    w.push_back(0);  // measurements: the run of each (a FIX_GRAD's slot) and its frame
    for (const Op& op : r.ops)
      if (op.cls == OP_GRAD) {
        int64_t frame;
        std::memcpy(&frame, op.fh, sizeof(frame));
        w.insert(w.end(), {op.param, frame});
        ++w[at];
      }
    for (const FixOp& f : fops) {
      w.push_back(f.kind);
      w.insert(w.end(), f.a, f.a + 11);
    }
    for (const PhaseTable& t : r.tab.tables) w.insert(w.end(), {t.entry, t.c, t.first_term, t.num_terms, t.k, t.g});
    for (const PhaseTerm& t : r.tab.terms) w.insert(w.end(), {(int64_t)t.mask, t.turn});
  }
  *count = (int64_t)w.size();
  if (*count > capacity) return set_error(DMV_ERR_INVALID, "dmv_debug_fix_plan: %lld words", (long long)*count);
  std::copy(w.begin(), w.end(), words);
  return DMV_OK;
}
