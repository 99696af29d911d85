// Internal declarations shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>
#include <cmath>
#include <vector>

#include "../../include/damavand_gpu.h"

namespace dmv {

// ---------------------------------------------------------------------------
// Error reporting: every entry point returns a status and records the last
// error (thread-local) with a message. Nothing calls exit().
// ---------------------------------------------------------------------------
int set_error(int code, const char* fmt, ...);
void clear_error();
int last_error();

#define DMV_CUDA_TRY(expr)                                                           \
  do {                                                                               \
    cudaError_t dmv_e_ = (expr);                                                     \
    if (dmv_e_ != cudaSuccess) {                                                     \
      return ::dmv::set_error(dmv_e_ == cudaErrorMemoryAllocation ? DMV_ERR_OOM      \
                                                                  : DMV_ERR_CUDA,    \
                              "%s failed: %s (%s:%d)", #expr,                        \
                              cudaGetErrorString(dmv_e_), __FILE__, __LINE__);       \
    }                                                                                \
  } while (0)

#define DMV_TRY(expr)                       \
  do {                                      \
    int dmv_rc_ = (expr);                   \
    if (dmv_rc_ != DMV_OK) return dmv_rc_;  \
  } while (0)

// Counts the library's own kernel launches (reported by the benchmark).
void count_launch(int64_t n = 1);

// Test hook (dmv_debug_fail_allocations): true when this device allocation
// must fail as if the device were out of memory.
bool injected_alloc_failure();

// Optional per-launch CUDA-event profiling (dmv_profile_*). prof_begin
// returns a token (or -1 when profiling is off); prof_end closes it.
int64_t prof_begin(int family, cudaStream_t stream, double algorithmic_bytes, double multiply_adds = 0.0);
void prof_end(int64_t token, cudaStream_t stream);

// ---------------------------------------------------------------------------
// Gate matrices and fused-op encoding
// ---------------------------------------------------------------------------
// Op arithmetic classes: the kernels specialise on them to spend as few
// FP64 operations as the matrix allows (FP64 is ~1/70 of FP32 on GB300).
enum OpClass : int32_t {
  OP_GENERAL = 0,  // full complex 2x2
  OP_DIAG = 1,     // m01 = m10 = 0
  OP_SWAP = 2,     // exactly [[0,1],[1,0]] (X, CNOT): a pure exchange
  OP_REAL = 3,     // all four entries real
  OP_ANTI = 4,     // m00 = m11 = 0 (Y and scaled exchanges)
  OP_RXLIKE = 5,   // m00, m11 real and m01, m10 imaginary (RX and its adjoint): 8 multiply-adds
  // Only in window passes rewritten by rewrite_pass_rotations (diag_plan.cpp):
  OP_ROT = 6,      // FP64: real rotation R = [[c, -s], [s, c]] (0 <= s <= c) applied as f * M, M = [[1, -w], [w, 1]]
                   //   (w = s/c, f = c), two multiply-adds per component; m[0] = w (mh[0], ml[0] its FP32 pair). The state is left divided by f; the
                   //   caller multiplies the product of the f's back.
  OP_PHASE = 7,    // every amplitude times a phase from a table (PhaseEntry); fields below
  OP_GRAD = 8      // adjoint sweeps: Im <lambda| P |psi> for P = X, Y, Z on `target` goes to slot `param`; in FP64 list
                   //   order the squared product of the rotation factors before it is m[0]
};

// Control kinds inside a fused pass.
enum CtrlKind : int32_t {
  CTRL_NONE = 0,
  CTRL_LOCAL = 1,   // control qubit is one of the pass's local bits
  CTRL_GLOBAL = 2   // control qubit is outside the tile: constant per tile
};

// One operation as the kernels see it (224 bytes).
struct alignas(16) Op {
  double m[8];        // row-major 2x2, (re, im) pairs
  float mh[8];        // m split into FP32 pairs: m = mh + ml (FP32-pair arithmetic)
  float ml[8];
  int32_t fh[8];      // m as Q.54 fixed point: round(m * 2^54) = fh * 2^31 + fl, fl in [0, 2^31)
  int32_t fl[8];
  int32_t target;     // local bit (fused) or qubit (unfused)
  int32_t ctrl;       // local bit or global qubit, per ctrl_kind
  int32_t ctrl_kind;  // CtrlKind
  int32_t cls;        // OpClass
  int32_t param;      // index of the gradient slot (adjoint) or -1
  int32_t generator;  // 0 none, 1 X, 2 Y, 3 Z: generator of a rotation (adjoint)
  int32_t unitary;    // 1 when m is unitary to 1e-12 (block fixed point relies on it)
  int32_t phase;      // register phase of a fused op (kPhase* below), 0 elsewhere
};
static_assert(sizeof(Op) == 224, "Op layout");

// An OP_PHASE op multiplies amplitude l of a tile (2^k amplitudes) by the
// phase of table entry fh[0] + (gsel << k) + l, where gsel collects the
// tile's bits at the fh[1] (at most 3) global qubits fh[2..4]. An entry holds
// the phase e^{i phi} as i^q e^{i phi'} with |phi'| <= pi/4: (x, y) is
// rotated by phi' with three shears, x += t y, y += s x, x += t y
// (t = -tan(phi'/2), s = sin phi'), then multiplied by i^q: swapped when q is
// odd and the sign words xored into the high halves of x and y.
struct alignas(32) PhaseEntry {
  double t;
  double s;
  uint32_t swap_xy;
  uint32_t sign_x;  // 0 or 0x80000000
  uint32_t sign_y;
  uint32_t pad;
};
static_assert(sizeof(PhaseEntry) == 32, "PhaseEntry layout");
constexpr int kMaxPhaseGlobals = 3;

// A phase table before its entries are made: the angle of entry (gsel << k) |
// l is c plus the turn of every term whose mask meets an odd number of set
// bits of l | gsel << kPhaseGlobalBit, in units of 2^-64 of a full turn.
constexpr int kPhaseGlobalBit = 20;
struct PhaseTerm {
  uint32_t mask;
  uint32_t pad;
  int64_t turn;
};
struct PhaseTable {
  int64_t entry;  // first entry
  int64_t c;
  int32_t first_term, num_terms;
  int32_t k, g;  // tile bits, global bits
};
struct PhaseTables {
  std::vector<PhaseTerm> terms;
  std::vector<PhaseTable> tables;
  int64_t entries = 0;
};

// Register phases of a fused pass run by the TMA window kernel: each thread
// keeps 2^rb amplitudes of the tile in registers, the ones that differ in rb
// "register bits" of the tile index, and applies every op whose target is a
// register bit without touching shared memory. An op that starts a phase
// carries the phase's register bits; the tile goes through shared memory only
// between phases.
constexpr uint32_t kPhaseStart = 0x80000000u;  // this op starts a phase
// bits 0..15: the phase's register bits, 4 bits each (valid on a phase start)
// bits 16..17: index of the op's target among the register bits
// bits 20..22: 1 + index of the op's local control among them, 0 if not one
constexpr int kPhaseTargetShift = 16;
constexpr int kPhaseCtrlShift = 20;
constexpr int kMaxRegBits = 4;

// An op as the register-phase kernel reads it from its shared-memory op
// table (complex64 passes): the FP32 matrix and the fields the loop tests.
struct alignas(16) PhaseOp {
  float m[8];         // op.mh: the matrix rounded to FP32
  uint32_t phase;     // op.phase
  int32_t ctrl;
  int32_t ctrl_kind;
  int32_t cls;
};
static_assert(sizeof(PhaseOp) == 48, "PhaseOp layout");
// Ops one launch of the register-phase kernel holds in shared memory; a
// longer pass runs as several launches over the same qubits.
constexpr int64_t kMaxPhaseOps = 128;

// Orders one fused pass's ops (tile-local targets) into register phases and
// marks them: each phase holds ops whose targets span at most rb tile bits
// (padded with unused tile bits); ops move across others only where they
// share no tile bit. Returns the number of phases.
int64_t assign_phases(Op* ops, int64_t count, int32_t tile_bits, int32_t rb);

// Fills op.mh / op.ml (FP32 pair: hi = nearest float, lo = nearest float of
// the rest), op.fh / op.fl (Q.54 limbs) and op.unitary from op.m.
void split_matrix(Op& op);

// Rewrites the ops src[0 .. count) of one FP64 window pass over a tile of
// 2^k amplitudes so that it spends fewer FP64 operations: every uncontrolled
// unitary 2x2 becomes D1 R D2 (R a real rotation; D1, D2 diagonal), and the
// diagonal factors of the whole pass (with Z-type
// and controlled-phase ops and the diagonals of Y-type ops) are collected
// into as few per-amplitude phase tables as the rotations allow: a diagonal
// factor moves later in time through exchanges (re-indexed) and through
// rotations on other bits, and earlier into the last table when nothing in
// between touches its bits. Appends the new ops to `dst` and the tables to
// `tab`; returns the number of ops appended.
// `rot_ops` true: rotations as OP_ROT (the FP64 kernels: two multiply-adds
// per component, the state left divided by each rotation's factor f, whose
// product over the pass is multiplied into *scale); false: as OP_REAL 2x2 ops
// (with their FP32-pair, Q.54 and FP32 forms), for the int64 arithmetic and
// for FP32 pairs outside the fixed-point passes.
// A product of many factors kept to about 2^-100 relative (error-free
// products through fma), for the OP_ROT factors.
struct ScaleDD {
  double hi = 1.0, lo = 0.0;
  void mul(double f) {
    const double p = hi * f;
    const double e = std::fma(hi, f, -p);
    const double l = std::fma(lo, f, e);
    hi = p + l;
    lo = l - (hi - p);
  }
  void mul(const ScaleDD& o) {
    const double p = hi * o.hi;
    const double e = std::fma(hi, o.hi, -p);
    const double l = std::fma(hi, o.lo, std::fma(lo, o.hi, e));
    hi = p + l;
    lo = l - (hi - p);
  }
};
// `single`: w rounded to FP32 (its factor f to match).
int64_t rewrite_pass_rotations(const Op* src, int64_t count, int32_t k, bool rot_ops, std::vector<Op>& dst,
                               PhaseTables& tab, ScaleDD* scale = nullptr, bool single = false);
// The entries of tables, on the host (the debug check; launch_plan has
// k_phase_tables make them).
void phase_entries(const PhaseTables& tabs, std::vector<PhaseEntry>& out);
// e^{i phi} of a table entry in double.
void phase_entry_value(const PhaseEntry& e, double& re, double& im);
// The FP64 kernels' 16-byte form: (t, s) with the quadrant in bit 62 of each
// (0 in both, as |t|, |s| < 2): bit 62 of t = swap_xy = q & 1, bit 62 of s =
// q >> 1 (sign_y); sign_x = the xor of the two.
void phase_tables_f64(const std::vector<PhaseEntry>& in, std::vector<double2>& out);

// Arithmetic used for complex128 storage.
enum Arith : int32_t {
  ARITH_FP64 = 0,    // IEEE FP64 multiply-adds
  ARITH_FP32X2 = 1,  // FP32-pair (double-float) error-free transformations
  ARITH_INT64 = 2,   // int64 block fixed point on the integer pipe
  ARITH_TC = 3       // int64 block fixed point, dense blocks as exact digit products on the tensor cores
};

// Host-side gate after parsing.
struct Gate {
  int32_t kind;
  int32_t target;
  int32_t control;  // -1 none
  double theta;
  double m[8];      // the gate's matrix, computed on the host (gates.cpp)
  bool observable;
};

// Matrix of a gate kind, the formulas of the reference's gates.rs.
void gate_matrix(int32_t kind, double theta, double m[8]);
int32_t classify(const double m[8]);
bool is_parametrised(int32_t kind);
// Generator P of R(theta) = exp(-i theta P / 2): 1 X, 2 Y, 3 Z, 0 none.
int32_t rotation_generator(int32_t kind);
// m = a * b (2x2 complex)
void matmul2(const double a[8], const double b[8], double out[8]);
// Conjugate transpose.
void adjoint2(const double a[8], double out[8]);
int parse_gates(const dmv_gate_t* gates, int64_t num_gates, int32_t n, std::vector<Gate>& out);

// ---------------------------------------------------------------------------
// Execution plan: a sequence of passes over the statevector.
// ---------------------------------------------------------------------------
struct Pass {
  // kind 0: single op on global qubit indices (unfused kernel).
  // kind 1: fused window: local bits = [0, low_bits) + high[0..num_high).
  int32_t kind;
  int32_t low_bits;
  int32_t num_high;
  int32_t high[16];
  int64_t op_begin;  // range in Plan::ops
  int64_t op_count;
};

struct Plan {
  std::vector<Pass> passes;
  std::vector<Op> ops;
  int64_t num_gates = 0;
  bool as_is = false;  // complex64: its passes run as 2x2 matrices, not rewritten
};

struct PlanOptions {
  int32_t fusion = DMV_FUSE_WINDOW;
  int32_t tile_bits = 12;  // log2 amplitudes per tile
  int32_t low_bits = 6;    // always-local low qubits (coalesced chunks)
  bool search_windows = false;  // choose each window by a search (next_window) instead of the first targets met
  bool windows_only = false;  // every pass a window pass (the batched kernel runs only those)
  // Adjoint sweeps: when set, no gates are merged and the op made from
  // gates[i] carries param_of[i] / generator_of[i] (Op::param, Op::generator).
  const int32_t* param_of = nullptr;
  const int32_t* generator_of = nullptr;
  // Adjoint sweeps in runs: when set (param_of null), gates are merged and
  // (*run_of)[i] gets the index of the merged gate that gates[i] joined, which
  // is also the Op::param of its op; Op::generator is set when any of its
  // gates has a generator.
  std::vector<int32_t>* run_of = nullptr;
};

int build_plan(const std::vector<Gate>& gates, int32_t n, int32_t precision,
               const PlanOptions& opt, Plan& plan);
// The reverse sweep of an adjoint gradient as a plan: the non-observable gates
// in reverse order, each replaced by U^dagger, unmerged, each op tagged with
// its gate's parameter slot (list order of the parametrised gates) and
// generator (PlanOptions::param_of / generator_of).
int build_adjoint_plan(const std::vector<Gate>& gates, int32_t n, int32_t precision, const PlanOptions& base,
                       Plan& plan);
// rewrite_pass_rotations of several window passes: pass which[j] of `plan`
// into out[j] (its own ops, its own tables with OP_PHASE offsets from 0, its
// factor product).
struct RewrittenPass {
  std::vector<Op> ops;
  PhaseTables tab;
  ScaleDD scale;
};
void rewrite_passes(const Plan& plan, const std::vector<int64_t>& which, bool rot_ops,
                    std::vector<RewrittenPass>& out, bool single = false);

// ---------------------------------------------------------------------------
// Tensor-core window passes (ARITH_TC, complex128 storage).
//
// The tile (2^12 amplitudes) is held as int64 block fixed point. A pass is
// cut into stages: exchanges (X, CNOT: integer swaps in shared memory) and
// dense blocks, the product of consecutive ops on at most 5 tile bits as one
// 32 x 32 complex matrix. A block is applied to the tile viewed as 128
// columns of 32 amplitudes: every integer is split into 7 balanced 8-bit
// digits (FP16, exact), the matrix likewise, and the 34 digit products
// whose weights 2^(-8s) have s = i + j <= 7 accumulate exactly in FP32 on the
// tensor cores (tcgen05.mma), one TMEM accumulator per weight.
// ---------------------------------------------------------------------------
constexpr int kTcBlockBits = 5;                             // qubits of a dense block
constexpr int kTcDigits = 7;                                // balanced 8-bit digits of a 56-bit integer
constexpr int kTcURows = 64 * kTcDigits;                    // rows of a block's stacked digit matrix
constexpr int64_t kTcUHalves = (int64_t)kTcURows * 64;      // FP16 elements per block (56 KB)
enum TcStageKind : int32_t { TC_BLOCK = 0, TC_SWAP = 1 };

// Exchanges are not applied to the data: the tile stays where it is and the
// kernel reads logical amplitude l at phys(l) = A l xor c, an affine map over
// the 12 tile bits. A CNOT with a control inside the tile changes A (the host
// tracks it), X and CNOTs controlled from outside the tile change c (the
// kernel, per tile).
struct TcStage {
  int32_t kind;       // TcStageKind
  int32_t img[12];    // block: A e_b for the block's 5 bits (img[0..4], block-row bits 0..4) and its 7
                      // other tile bits (img[5..11], column-index bits 0..6); swap: img[0] = mask xored into c
  int32_t gctrl;      // swap: control qubit outside the tile (c changes on tiles where it is 1), or -1
  int32_t u_index;    // block: index of its digit matrix in the plan's array
  int32_t magic;      // block: 1 when every FP32 accumulator stays below 2^22 in magnitude
  int32_t next_u;     // block: u_index of the pass's next block (cyclically), fetched during this one's epilogue
  int32_t pad[3];
};
static_assert(sizeof(TcStage) == 80, "TcStage layout");

// Cuts window pass `ps` of `plan` (a 2^12-amplitude tile) into stages,
// appended to `stages`, and appends each block's digit matrix (kTcUHalves
// FP16 bit patterns in the tensor cores' K-major layout) to `u`. Returns
// false, appending nothing, when the pass holds an op the tensor-core kernel
// does not take (a non-unitary op, or a non-exchange op controlled from
// outside the tile).
// `final_map` receives A e_b (b = 0..11) after the pass's last stage and
// `exchanges` the number of X / CNOT ops applied as relabellings.
bool build_tc_pass(const Plan& plan, const Pass& ps, std::vector<TcStage>& stages, std::vector<uint16_t>& u,
                   int32_t final_map[12], int32_t* exchanges);
// Test hook (dmv_debug_tc_convert): 1 forces the exact conversion in every block.
void set_tc_convert_mode(int32_t mode);

// ---------------------------------------------------------------------------
// Fixed-point window passes (fix_window.cuh; complex128 storage): a rewritten
// pass (rotations, phase tables, exchanges) as register phases over int64
// amplitudes.
//
// The tile's logical amplitude l sits at shared-memory slot fix_slot(A l) xor
// c: exchanges move no data, they change the linear map A (a CNOT inside the
// tile) or the offset c (X, and per tile a CNOT controlled from outside it).
// A phase keeps 16 amplitudes per thread in registers, those that differ in 4
// register bits, and applies every op whose target is one of them.
// ---------------------------------------------------------------------------
enum FixKind : int32_t {
  FIX_PHASE = 0,  // registers out, registers in: a[0..5] the images (fix_slot(A e_b)) of the 4 register bits, then of
                  // the 8 thread bits, two 16-bit words each; a[8]: c ^= a[8] first; a[9]: kFixSimple. Host only: a[6] the tile bits of the
                  // 8 thread bits, a[7] of the 4 register bits, 4 bits each
  FIX_XOR = 1,    // slot offset c ^= a[1] on tiles where qubit a[0] is 1
  FIX_ROT = 2,    // OP_ROT on register bit a[0] & 3: a[0] also holds kFixComplement and kFixShift; a[1], a[2]: the
                  // multiplier as a[1] 2^-32 + a[2] 2^-64 (both signed words)
  FIX_TABLE = 3,  // OP_PHASE: a[0] first table entry, a[1] number of global bits, a[2..4] those qubits. A table (and
                  // each slice of it) lies in the order its phase reads it: register, then thread
  FIX_FETCH = 4,  // a[0..4] as FIX_TABLE: start loading that table's first entries (the next FIX_TABLE's)
  FIX_GRAD = 5,   // OP_GRAD on register bit a[0]: slot a[1], a[3..4]: the squared product of the rotation factors
                  // before it (double)
  FIX_END = 6     // registers out; a[0..5], a[8] as FIX_PHASE for tile bits 8..11 and 0..7 under the final map
};
constexpr int32_t kFixComplement = 4;  // the multiplier is 1 - w
constexpr int32_t kFixShift = 8;       // then every amplitude is halved
// FIX_PHASE's a[9] when its ops are at most one FIX_TABLE, then one FIX_ROT on
// each of register bits 0, 1, ... (their number in the low bits).
constexpr int32_t kFixSimple = 16;
constexpr int32_t kFixSimpleTable = 8;  // with a table
struct alignas(16) FixOp {
  int32_t kind;
  int32_t a[11];
};
static_assert(sizeof(FixOp) == 48, "FixOp layout");
// FixOps the kernel holds in shared memory; a longer pass reads them from HBM.
constexpr int32_t kFixSmemOps = 256;
// Shared-memory slot of 16-byte element l: its index within a row of 8 (the 32
// banks) xored with the other three groups of 3 index bits, so that lanes that
// differ in any three bits distinct modulo 3 meet different banks.
inline int32_t fix_slot_host(int32_t l) { return l ^ (((l >> 3) ^ (l >> 6) ^ (l >> 9)) & 7); }
// The ops of one rewritten pass over a tile of 2^tile_bits amplitudes (12: 16
// per thread, 11: 8) as FixOps, appended to `out`; *shifts gets the number of
// halvings. False, appending nothing, when the pass holds any op but OP_ROT,
// OP_PHASE, OP_GRAD and an uncontrolled or CNOT-like OP_SWAP.
// Bit z of *sparse: the z smallest rotation multipliers (one per tile bit, the
// least of its rotations) have a product of at least 2^-kFixRange, so that an
// amplitude that spreads from a nonzero one over z bits stays within that
// range of it, and z is at most kFixUnreached (a tile of 2^(12-z) nonzero
// amplitudes rounds every one of 2^12).
// `single`: complex64 tiles (8-byte elements, fix_slot8), the rotations' w as
// floats in a[1], no halvings.
bool build_fix_pass(const Op* ops, int64_t count, int32_t tile_bits, std::vector<FixOp>& out, int32_t* shifts,
                    uint32_t* sparse = nullptr, bool single = false);
// Slot of an 8-byte element: the same for the 16 of a row and groups of 4 bits.
inline int32_t fix_slot8_host(int32_t l) { return l ^ (((l >> 4) ^ (l >> 8)) & 15); }
constexpr int kFixUnreached = 4;
constexpr int kFixRange = 12;  // binary orders between a fixed-point tile's largest and smallest amplitude
// Where make_phase_tables puts each form of the tables' entries (null: nowhere).
struct PhaseTableForms {
  double2* f64 = nullptr;
  float4* df = nullptr;
  int4* fx = nullptr;
  longlong2* fix = nullptr;  // in the order of fix_ops
  float2* f32 = nullptr;     // the same, single precision
};
struct DeviceBuffer;
// Makes the entries of `tabs` on the device (k_phase_tables). `src`, `src_dev`
// hold the upload.
int make_phase_tables(const PhaseTables& tabs, const std::vector<FixOp>& fix_ops, const PhaseTableForms& forms,
                      std::vector<unsigned char>& src, DeviceBuffer& src_dev, cudaStream_t stream);

// ---------------------------------------------------------------------------
// Device state
// ---------------------------------------------------------------------------
struct DeviceBuffer {
  void* ptr = nullptr;
  size_t bytes = 0;
  int reserve(size_t n);
  void release();
};

}  // namespace dmv

struct dmv_state_s {
  int32_t n = 0;
  int64_t N = 0;
  int32_t precision = DMV_C128;
  int32_t arith = dmv::ARITH_FP64;  // complex128 arithmetic (ignored for complex64)
  int device = 0;
  void* amps = nullptr;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  dmv::DeviceBuffer ops_dev;     // plan ops uploaded for the last apply
  dmv::DeviceBuffer reduce_dev;  // reduction partials
  dmv::DeviceBuffer chunk_dev;   // per-chunk probability sums (sampling)
  std::vector<dmv::Op> ops_host_pinned;  // (regular host memory; copied async from a pinned staging)
  std::vector<dmv::Op> ops_staging;      // plan ops with register phases marked, as uploaded
  std::vector<dmv::Pass> pass_staging;   // the launches of the last plan (long phase passes split)
  std::vector<dmv::PhaseOp> phase_ops;   // compact ops of the register-phase launches
  dmv::DeviceBuffer phase_ops_dev;
  dmv::PhaseTables phase_tabs;             // phase tables of the rewritten passes
  std::vector<unsigned char> phase_src;    // their terms and slices, as uploaded
  dmv::DeviceBuffer phase_src_dev;
  std::vector<dmv::ScaleDD> pass_scale;  // launch_plan: OP_ROT factor product per staged pass
  dmv::DeviceBuffer phase_tab_dev;
  dmv::DeviceBuffer phase_tab2_dev;
  std::vector<dmv::FixOp> fix_ops;         // fixed-point passes of the last plan
  dmv::DeviceBuffer fix_ops_dev, phase_tab_fix_dev;
  std::vector<dmv::TcStage> tc_stages;  // tensor-core passes of the last plan
  std::vector<uint16_t> tc_u;
  dmv::DeviceBuffer tc_stages_dev, tc_u_dev;
  void* pinned = nullptr;        // pinned host staging
  size_t pinned_bytes = 0;
  int64_t last_passes = 0, last_ops = 0, last_bytes = 0;
  int64_t last_tc_passes = 0, last_tc_blocks = 0, last_tc_swaps = 0;
  int64_t last_phase_tab_bytes = 0;  // phase tables uploaded by the last plan
  int64_t last_upload_bytes = 0;     // every host-to-device byte of the last plan (ops, tables, digit matrices)
  bool fp64_rewrite = true;          // FP64 window passes as rotations and phase tables
  // Adjoint gradients: psi and lambda, the partial sums, the plan, its tables.
  // Kept between calls for states of at most kKeepAdjointBytes (allocating and
  // freeing them took 0.3 ms of a 10-qubit gradient's 0.9 ms).
  dmv_state_s* adj_state[2] = {nullptr, nullptr};
  dmv::DeviceBuffer adj_partial, adj_src, adj_work, adj_tab, adj_fix_tab;
  cudaEvent_t ev_begin = nullptr, ev_end = nullptr;
  size_t amp_bytes() const { return (size_t)N * (precision == DMV_C128 ? 16 : 8); }
};

namespace dmv {
constexpr size_t kKeepAdjointBytes = size_t(64) << 20;
void release_adjoint(dmv_state_s* s);
int ensure_pinned(dmv_state_s* s, size_t bytes);

constexpr int32_t kSearchQubits = 20;
// Planner settings for a state: tiles of 2^12 amplitudes (the TMA window
// kernel's register phases hold 8 per thread of 512). `sweep`: a gradient's.
//
// complex64 passes are rewritten (rotations, phase tables) from kSearchQubits
// qubits on. Below, the passes of a few states overlap and the host's time per
// forward shows, which the search and the rewrite raise (17 qubits, 1290 gates:
// 289 us): three states in turn take 189 us per forward without and 316 with
// them at that size, 230 and 289 at 19 qubits and 15 layers, 31 and 66 at 13
// and 15, although one state alone gains (537 and 289 us at 17 qubits). Above,
// the device's time decides: 763 and 405 us at 21 qubits and 16 layers.
//
// On the tensor cores a pass's cost is the digit split and recombination of the
// state. Below 20 qubits the search has little to choose from: at 13 to 19 it
// takes 0.98 of the time of the first targets met on ladders and rings but 1.03
// on random circuits, 1.25 at worst; at 20 to 23 qubits 0.88 and 0.97.
inline PlanOptions plan_options_for(const dmv_state_s* s, int32_t fusion, bool sweep = false) {
  PlanOptions opt;
  opt.fusion = fusion;
  opt.tile_bits = 12;
  opt.low_bits = 4;  // a 128-byte row of complex64, two of complex128
  opt.search_windows = true;
  if (!sweep && s->n < kSearchQubits && (s->precision == DMV_C64 || s->arith == ARITH_TC)) {
    opt.search_windows = false;
    opt.low_bits = 6;  // rows of 512 and 1024 bytes
  }
  return opt;
}

// complex64 lists of a few gates from kSearchQubits qubits on, if one pass over
// the first targets' qubits holds them: a table among them costs a rewritten
// pass a launch and a phase, and with rows of 128 bytes a pass moves the state
// at 0.87 of the rate of rows of 512. Rewritten and as they are: four Hadamards
// 19.2 and 14.0 us at 20 qubits, 67.7 and 57.8 at 24, 800 and 699 at 28; six
// 19.6 and 15.5, 76.9 and 78.6, 959 and 1029.
constexpr int64_t kFewGates = 4, kFewGatesSmall = 8;
constexpr int32_t kFewGatesSmallQubits = 22;  // fewer: the launches decide
// The plan of a gate list on a state.
inline int plan_for(const dmv_state_s* s, const std::vector<Gate>& gates, int32_t fusion, Plan& plan) {
  if (s->precision == DMV_C64 && s->n >= kSearchQubits && gates.size() <= 64) {
    PlanOptions opt;
    opt.fusion = fusion;
    DMV_TRY(build_plan(gates, s->n, s->precision, opt, plan));
    bool tables = false;
    for (const Op& op : plan.ops) {  // exchanges and rotations [[c, -s], [s, c]], 0 < s <= c, leave none
      const bool rotation = op.cls == OP_REAL && op.m[0] == op.m[6] && op.m[2] == -op.m[4] && op.m[4] > 0.0 &&
                            op.m[0] >= op.m[4];
      tables = tables || (op.cls != OP_SWAP && !rotation);
    }
    plan.as_is = plan.passes.size() == 1 && tables &&
                 (int64_t)plan.ops.size() <= (s->n < kFewGatesSmallQubits ? kFewGatesSmall : kFewGates);
    if (plan.as_is) return DMV_OK;
  }
  plan.as_is = false;
  return build_plan(gates, s->n, s->precision, plan_options_for(s, fusion), plan);
}

// Kernel launchers (kernels_*.cu). All stream-ordered on s->stream.
int launch_set_zero(dmv_state_s* s);
// The state times a real factor (complex128).
int launch_scale_state(dmv_state_s* s, double f);
int launch_plan(dmv_state_s* s, const Plan& plan);
int launch_probabilities(dmv_state_s* s, double* probs_device);
int launch_expect_z(dmv_state_s* s, double* expect_host, double* norm_host);
int launch_sample(dmv_state_s* s, const double* uniforms_host, int64_t k, uint64_t* samples_host);
// Draws k samples on the device (uniforms from the host, or from the seeded
// SplitMix64 stream when uniforms_host is null) and counts, per bit position,
// the samples with that bit set; the samples never leave the device.
int launch_sample_counts(dmv_state_s* s, const double* uniforms_host, uint64_t seed, int64_t k,
                         unsigned long long counts_host[64]);
int sample_from_device_probs(const double* probs_device, int64_t num_probs, int32_t num_bits,
                             cudaStream_t stream, const double* uniforms_host, int64_t k,
                             uint64_t* samples_host);
int launch_inner_product(dmv_state_s* a, dmv_state_s* b, double* re, double* im);
int launch_scale_by_z_observable(dmv_state_s* dst, dmv_state_s* src, const double* weights_host);
int adjoint_sweep_fix(dmv_state_s* s, dmv_state_s* psi, dmv_state_s* lam, const std::vector<Gate>& gates, double* grads,
                      bool* done);
int launch_reduce_rows(const double* in, int64_t rows, int cols, double* out, cudaStream_t stream);
int launch_adjoint_step(dmv_state_s* psi, dmv_state_s* lam, const Op& op, double* grad_slot_device);
int adjoint_gradient(dmv_state_s* s, const std::vector<Gate>& gates, const double* weights,
                     double* loss, double* grads);
int upload_ops(dmv_state_s* s, const Op* ops, int64_t count);
// DMV_ERR_TIMEOUT (and clears the flag) when a TMA window pass or the
// bulk-staged chunk-mass pass gave up waiting for a load since the last
// check; synchronises the device.
int check_window_status();
// Polls before a TMA load wait gives up; negative restores the default.
void set_tma_wait_limit(int64_t polls);
uint32_t tma_wait_limit();
// The device word those waits set to 1 when they give up.
int* tma_status_word();

// The Pauli-Z mass pass of one state (bulk-staged) into caller-provided device
// buffers: `partial` holds own_mass_partials doubles, `sums` the n + 1 sums. The
// first call for a kind is not made inside a capture.
int64_t own_mass_partials(int src_kind, int n);
int launch_own_mass(const void* src, int src_kind, int n, double* partial, double* sums, cudaStream_t stream);
// The same for many circuits of a batch in one pass: circuit c's
// CTAs first_cta .. + ctas leave n + 1 sums each at `partial`, and columns
// first_column .. + n of `sums` get the mass with bit q set (q < n), then the total.
struct BatchMass {
  int64_t amp_offset;
  int64_t partial;  // doubles
  int32_t n, first_cta, ctas, first_column;
};
int batch_mass_ctas(int n);
int launch_batch_mass(const BatchMass* circuits, const int32_t* circuit_of_cta, int ctas, const int32_t* circuit_of_column,
                      int columns, const void* arena, int src_kind, double* partial, double* sums,
                      cudaStream_t stream);
}  // namespace dmv
