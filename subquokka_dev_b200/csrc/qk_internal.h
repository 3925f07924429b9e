// Internal types shared by the host code (C++) and the kernels (CUDA).
#pragma once

#include <cstddef>
#include <cstdint>
#include <functional>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "quokka_gpu.h"

namespace qk {

// Kernel-level operation.  Every parsed gate lowers to one of these; the
// coefficients are complex FP64 values computed on the host with the
// reference's own formulas (src/circuit.cpp:2655-2991).
enum OpKind : int32_t {
    OP_DENSE1 = 0,  // 2x2 matrix m[0..3] on q[0]                 (H X Y U1 RX RY)
    OP_PHASE1 = 1,  // amplitudes with bit q[0] set *= m[0]        (Z P)
    OP_DIAG1 = 2,   // bit q[0] = 0: *= m[0], = 1: *= m[1]         (RZ)
    OP_DENSE2 = 3,  // 4x4 matrix on (q[0], q[1]), index bit0=q[0] (U2)
    OP_PHASE2 = 4,  // amplitudes with bits q[0], q[1] set *= m[0] (CP)
    OP_DIAG2 = 5,   // *= m[b0 + 2 b1]                             (RZZ)
    OP_SWAP2 = 6,   // exchange |01> and |10> of (q[0], q[1])      (SWAP, VSWAP_1_1: aux = 1)
    OP_PERM = 7,    // swap bit q[i] with bit q[k+i], i < k = nq/2 (VSWAP_k_k)
    OP_GRAD = 8,    // adjoint sweep: grad[aux] += Im <lambda|G|psi>, G on q[0] = X/Y/Z by m[0] = 1/2/3
    OP_CX = 9,      // flip bit q[1 - aux] where bit q[aux] is set (a U2 that is exactly a CNOT)
    OP_CDENSE1 = 10,  // 2x2 on q[0]: m[0..7] where bit q[1] is 0, m[8..15] where it is 1 (planner-made)
    OP_K = 11,  // factored one-qubit unitary on q[0], without its scalar (planner-made, qk_factor.cpp):
                // right phase m[2..3] on the upper half, then x' = x - t y, y' = t x + y, t = m[0], then
                // left phase m[4..5]; scalar m[6..7]; aux = kRightPhase | kLeftPhase.  aux & kFull:
                // x' = x + B y, y' = F x + y, B = m[0..1], F = m[2..3], then the left phase
    OP_X = 12,  // flip bit q[0] (planner-made, qk_factor.cpp)
};
constexpr int kRightPhase = 1, kLeftPhase = 2, kFull = 4, kGiven = 8;   // kGiven: a circuit's own matrix (U1)

struct Op {
    int32_t kind;
    int32_t nq;
    int32_t q[QK_MAX_TARGETS];
    int32_t aux;   // OP_GRAD: parameter index; OP_CX: control index; OP_SWAP2 / OP_PERM: 1 from a VSWAP
    double m[32];  // complex coefficients, (re, im) interleaved
};

// Thread-local error message; returns code so callers can `return fail(...)`.
int fail(int code, const char *fmt, ...) noexcept __attribute__((format(printf, 2, 3)));
void clear_error();

// f()'s code, or QK_ERR_OOM where it runs out of host memory: nothing is
// thrown past the planners, whose callers are C entry points.
template <typename F> int no_throw(F &&f) {
    try {
        return f();
    } catch (const std::bad_alloc &) {
    } catch (const std::length_error &) {
    }
    return fail(QK_ERR_OOM, "out of host memory");
}

// task(0) .. task(n - 1) on up to n host threads, this one among them (all of
// them on this one where no thread can be had).  Returns the first failing
// task's code, with its message.
int run_tasks(size_t n, const std::function<int(size_t)> &task);

// Lower a parsed gate to a kernel op (host, FP64).
int lower_gate(const qk_gate &g, Op &op);

// True when the op is diagonal in the computational basis.
inline bool op_is_diagonal(const Op &op) {
    return op.kind == OP_PHASE1 || op.kind == OP_DIAG1 || op.kind == OP_PHASE2 ||
           op.kind == OP_DIAG2;
}

// Qubits of an op that a fused pass must hold in registers: q[reg_first(op)
// .. + reg_count(op)).  None for diagonal ops, the target for OP_CX and
// OP_CDENSE1 (the control / condition may be any qubit, as for a diagonal
// op), all of them otherwise.
inline int op_reg_count(const Op &op) {
    return op_is_diagonal(op) ? 0 : (op.kind == OP_CX || op.kind == OP_CDENSE1) ? 1 : op.nq;
}
inline int op_reg_first(const Op &op) { return op.kind == OP_CX ? 1 - op.aux : 0; }

}  // namespace qk

// Parsed circuit container behind the opaque qk_circuit handle.
struct qk_circuit {
    std::vector<qk_gate> gates;
    std::vector<int32_t> group_sizes;
};

namespace qk {

// ---------------------------------------------------------------------------
// Fused passes.  A pass stages tiles of 2^T amplitudes (tile bits bpos[0..T))
// and runs a small program on them; each thread keeps R = 2^r amplitudes in
// registers, indexed by r "register" tile bits, the rest of the tile bits
// index the thread.  Programs are built on the host (qk_plan.cpp).
// ---------------------------------------------------------------------------
constexpr int kPassMaxBits = 14;
constexpr int kPassMaxReg = 5;

enum TOpKind : uint8_t {
    TOP_REMAP = 0,  // re-distribute the tile: register slot s <- tile bit bits[s] (bits[4..7]: the
                    // same ascending)
    TOP_G1 = 1,     // dense 2x2 on register slot a; coef -> 4 complex
    TOP_G2 = 2,     // dense 4x4 on register slots a < b (index bit0 = a); coef -> 16 complex
    TOP_DIAG = 3,   // amplitude *= coef[bit(a) + 2 bit(b)]; a, b are qubit codes
    TOP_PHASE = 4,  // amplitude *= coef[0] where bit(a) = bit(b) = 1 (Z, P, CP; b may be none)
    TOP_GRAD = 5,   // two-state passes: gacc[coef] += Im <lambda|G|psi>, G = X/Y/Z (b = 1/2/3) on slot a
    TOP_CX = 6,     // swap register slot a's pairs where qubit code b is 1 (controlled X)
    TOP_CG1 = 7,    // dense 2x2 on slot a: coef[0..3] or coef[4..7] by qubit code b (not a register slot)
    TOP_R1 = 8,     // real 2x2 on slot a: coef[0] = (m00, m01), coef[1] = (m10, m11)
    TOP_R2 = 9,     // real 4x4 on slots a < b (index bit0 = a): coef[2 r + h] = (m[r][2h], m[r][2h + 1])

    // Steps of factored programs (PassDesc.form = 1, qk_factor.cpp); nbits of a TOP_REMAP or TOP_LAYER
    // counts the 16-byte words that follow it and are no steps themselves.  Their
    // slots are ascending in the tile bits, the first op is the TOP_REMAP the
    // tile is loaded under, and the last TOP_REMAP the one it is stored under.
    // TOP_REMAP: the slots in bits, b = 1 if a TOP_LCX ran since the last one; the next word holds five
    // 16-bit values, the exchange-buffer byte offset of each slot's tile bit.
    // TOP_LAYER: factored one-qubit unitaries on several slots.  First, with kLayerSigns in b,
    // amplitudes whose slots x and y are both 1 change sign for each pair x < y in the mask bits[0..1].
    // Then for each slot s in a, ascending, a unitary with coefficients t and right phase: the slot's
    // upper half y takes the right phase (kLayerPending: the pending factor instead) and, with
    // kLayerWords, a sign, the parity of (tile label & w[s]) and (tile number & u[s]); the next two
    // words hold u, five 32-bit values, and w, five 16-bit values.  Then x' = x - t y, y' = t x + y.
    // With kLayerFull (programs with f_full) the coefficients are complex, B and F: y takes the sign alone,
    // then x' = x + B y, y' = F x + y
    TOP_LAYER = 14,
    TOP_LCX = 15,   // label step: tile bit a ^= qubit code b (a CX whose swap the next TOP_REMAP performs),
                    // b = kNoQubit: flipped (an X; programs with f_flips)
    TOP_PH2 = 16,   // 16 + slot_pair(a, b): amplitude *= coef[0] where slots a and b are 1
    TOP_LAM = 28,   // pending factor of the next TOP_LAYER *= the entries of two tables: coef[i], i the
                    // bits of the first four condition codes in bits, and (nbits > 4)
                    // coef[16 + j], j those of the others.  A code: a tile bit, or kOuterFlag | bit of
                    // the tile number
    TOP_SCALE = 29, // amplitude *= coef[0] (b = 1: complex, 0: its real part)
};
constexpr uint8_t kLayerFull = 0x10, kLayerWords = 0x20, kLayerSigns = 0x40, kLayerPending = 0x80;   // TOP_LAYER, high half of b
constexpr uint8_t kSignFlag = 0x40;   // condition codes of factored steps: the factor is -1
// index of the slot pair a < b among 0..9 (five slots)
constexpr int slot_pair(int a, int b) { return b * (b - 1) / 2 + a; }
// The kernel instance for passes marked xops carries factors that are the
// same for all of a thread's amplitudes (TOP_DIAG / TOP_PHASE on qubits
// outside the register slots) as one pending scalar, applied before the
// tile is re-distributed or stored -- except where the register amplitudes
// take 256 bytes or more (complex128 with 16 a thread, two states of 8
// complex128 or 16 complex64): those kernels run at their register limit,
// and the scalar's registers cost spills.
constexpr bool pending_scalar_ok(int amp_bytes, int reg_amps, int nstates) {
    return amp_bytes * reg_amps * nstates < 256;
}

// Qubit codes of TOP_DIAG / TOP_PHASE: < 0x80 tile-local bit; 0x80 | q global
// qubit q that is not a tile bit (constant over a tile); 0xFF no qubit (bit =
// 0 for TOP_DIAG, 1 for TOP_PHASE).
constexpr uint8_t kOuterFlag = 0x80;
constexpr uint8_t kNoQubit = 0xFF;

// Place of tile element j in a shared-memory tile: the low index bits XORed
// with folds of the higher ones, so that a warp's lanes, which differ in
// three (complex128) or four (complex64) consecutive thread bits wherever the
// register slots sit, address distinct banks.
constexpr uint32_t tile_swizzle(uint32_t j, bool c128) {
    return c128 ? j ^ (((j >> 3) ^ (j >> 6) ^ (j >> 9) ^ (j >> 12)) & 7u) : j ^ (((j >> 4) ^ (j >> 8) ^ (j >> 12)) & 15u);
}

struct TOp {
    uint8_t kind;
    uint8_t a, b;
    uint8_t nbits;
    uint8_t bits[kPassMaxReg + 3];
    uint32_t coef;
};
static_assert(sizeof(TOp) == 16, "TOp must stay 16 bytes");
static_assert(offsetof(TOp, bits) == 4 && offsetof(TOp, coef) == 12, "step words follow the fields");
constexpr uint8_t kNoSlot = 0xFF;   // TOp.bits[k] of a condition qubit held in no register slot

struct PassDesc {
    int32_t T;                    // tile bits
    int32_t L;                    // tile bits 0..L-1 are state bits 0..L-1 (contiguous runs)
    int32_t bpos[kPassMaxBits];   // state bit of each tile bit, ascending
    int32_t prog0, nprog;         // program slice in the plan's op array
    int32_t coef0, ncoef;         // coefficient slice (complex values) used by the program
    int32_t grad0, ngrad;         // gradient slots of the pass: plan.grad_params[grad0 .. grad0 + ngrad)
    int32_t perm;                 // 1: a qubit-permutation pass (VSWAP), prog unused
    int32_t nperm;
    int32_t perm_a[6], perm_b[6]; // tile-local bit pairs swapped on store (perm passes)
    int32_t xops;                 // 1: the program has real or diagonal ops (TOP_R1, TOP_R2, TOP_DIAG,
                                  // TOP_PHASE), run by the kernel instance that specialises them
    int32_t form;                 // 1: a factored program (k_fpass)
    int32_t last;                 // factored: index of the program's last TOP_REMAP
    int32_t fpos[kPassMaxReg], lpos[kPassMaxReg];  // factored: state bits of the first / last mapping's slots
};

// Host plan: passes + programs + complex coefficient pool (FP64).
struct HostPlan {
    int n = 0;
    int dtype = 0;
    int T = 0, r = 0;
    std::vector<PassDesc> passes;
    std::vector<TOp> ops;
    std::vector<double> coef;  // (re, im) pairs
    std::vector<int32_t> grad_params;  // parameter index of each pass's gradient slots
    int nstates = 1;           // 2: adjoint passes over (psi, lambda)
    size_t nremaps = 0, ngates = 0;
    // factored programs: program operations, a re-mapping and the steps that
    // run under it counting one each
    size_t nbodies = 0;
    size_t program_ops() const { return nbodies ? nremaps + nbodies : ops.size(); }
};

struct PlanOptions {
    int dtype;
    int tile_bits;   // T
    int reg_bits;    // r
    int plain_ops = 0;    // 1: no TOP_R1 / TOP_R2 (real ops as TOP_G1 / TOP_G2) and no pass marked
                          // xops (plans of the batched kernel, which has one instance)
    // plan_forward / plan_adjoint: tile and register bits of factored programs,
    // which are made where they can be (0: general programs only)
    int f_tile_bits = 0, f_reg_bits = 0;
    int f_wide_bits = 0;  // tile bits a forward plan takes instead where that means fewer passes of little work
    int f_flips = 0;      // 1: factored programs may flip a tile bit (TOP_LCX with kNoQubit); 0: two rotations instead
    int f_full = 0;       // 1: factored programs may hold layers of full unitaries (kLayerFull); 0: rotations only
    int threads = 0;      // 1: the factored planner tries its candidates on several host threads
};

// The fused plan of a flat gate list / of a backward sweep as the engine runs
// it: factored programs (qk_factor.cpp) where every one-qubit gate is a
// unitary and every two-qubit gate diagonal, a CX or a SWAP, and the kernel has
// the tile shape (complex128 only for backward sweeps); else the general programs of build_plan /
// build_adjoint_plan.
int plan_forward(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, HostPlan &plan);
int plan_adjoint(const qk_gate *gates, size_t ng, const int32_t *pidx, int n, const PlanOptions &o, HostPlan &plan);
// Whether a plan of these options and gates is factored.
bool plan_is_factored(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, int nstates);
int check_options(const PlanOptions &o, int n);
int pass_low_bits(const PlanOptions &o, int n);
int perm_tile_bits(int dtype);
// Build a fused plan for a flat gate list (greedy tile-bit choice).
int build_plan(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, HostPlan &plan);
// One permutation pass (an OP_PERM of 1 to 6 bit pairs), with no program.
int build_perm_plan(const Op &op, int n, const PlanOptions &o, HostPlan &plan);
// Op-list rewrites before planning (qk_rewrite.cpp).
bool one_qubit(const Op &op);
void as_matrix(const Op &op, double (&m)[8]);
void mat2_mul(const double (&x)[8], const double (&y)[8], double (&z)[8]);
void asap_order(std::vector<Op> &ops, int n);
std::vector<size_t> asap_positions(const std::vector<Op> &ops, int n);   // the ops in that order
void merge_one_qubit_runs(std::vector<Op> &ops, int n);
void absorb_into_two_qubit_ops(std::vector<Op> &ops, int n, bool keep_real = false);
bool op_is_real(const Op &op);
void hoist_gradients(std::vector<Op> &ops, int n);
void pair_gradients(std::vector<Op> &ops);
void relabel_perms(std::vector<Op> &ops, int n, int L, int max_bits, int max_pairs, bool swaps);
// Plan of a subcircuit file (the subcircuit path): the gates of all groups
// as one gate list, VSWAPs as renamings of the qubits after them.
int build_group_plan(const qk_gate *gates, const int32_t *sizes, size_t ngroups, int n, const PlanOptions &o,
                     HostPlan &plan);
PlanOptions default_plan_options(int dtype, int n);
// the default options with factored programs allowed
PlanOptions factored_plan_options(int dtype, int n);
PlanOptions factored_adjoint_options(int dtype, int n);

// Dense fused blocks: consecutive gates on at most kDenseQubits qubits
// multiplied (FP64, host) into one 2^k x 2^k unitary, applied as a
// tensor-core contraction.  A block with perm != 0 is a VSWAP instead.
constexpr int kDenseQubits = 6;
constexpr int kDenseDim = 1 << kDenseQubits;
struct DenseBlock {
    int q[kDenseQubits];               // block qubits, ascending; local bit b = q[b]
    std::vector<double> u;             // 64 x 64 complex, row-major, (re, im)
    int perm = 0;                      // VSWAP: the Op below instead of u
    Op perm_op;
    int ngates = 0;
};
// width (5 or 6): most qubits a block's gates may touch; blocks are padded to
// kDenseQubits with idle qubits.  dtype sets the tile limits of the
// permutation blocks.
int build_dense_blocks(const qk_gate *gates, size_t ng, int n, int width, int dtype, std::vector<DenseBlock> &blocks);

// A dense block's pass over the state: a supertile is the block's qubits plus
// the lowest other state bits (tile-local bits ascending in state position).
struct DenseDesc {
    PassDesc p;         // tile bits T, contiguous run L
    uint32_t blockmask; // tile-local bits that are the block's qubits
};
DenseDesc dense_block_desc(const DenseBlock &b, int n, int max_tile_bits);

// complex128 blocks (qk_dense_i8.cu): 64 x 64 supertiles; the operand of a
// block is its digit planes (128 rows x 224 words) and 128 row scales.
constexpr int kI8TileBits = 12;
constexpr int kI8Digits = 7;
constexpr size_t kI8OperandWords = 128 * 32 * kI8Digits;
constexpr size_t kI8OperandBytes = kI8OperandWords * 4 + 128 * sizeof(double);
void dense_i8_operand(const DenseBlock &b, std::vector<uint32_t> &out);   // kI8OperandBytes / 4 words
// complex64 blocks (qk_dense_tc.cu): W split into bf16 hi and lo operands
void dense_block_operand(const DenseBlock &b, std::vector<uint16_t> &out);   // 2 x 128 x 128
// Bytes of one block's device operand for dtype.
size_t dense_operand_bytes(int dtype);
// Backward sweep of an adjoint gradient: the inverses of gates[ng-1..0] on
// (psi, lambda), with the gradient of trainable gates (pidx[i] >= 0) taken
// just before their inverse.
int build_adjoint_plan(const qk_gate *gates, size_t ng, const int32_t *pidx, int n, const PlanOptions &o,
                       HostPlan &plan);
PlanOptions default_adjoint_options(int dtype, int n);
void invert_op(Op &op);

}  // namespace qk
