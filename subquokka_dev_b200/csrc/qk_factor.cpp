// Planner of factored pass programs (host).
//
// A one-qubit unitary is a scalar times diag(1, p) R diag(1, l): two phases
// and a real rotation.  Divided by its cosine the rotation needs one
// multiply-add a component (x' = x - t y, y' = t x + y), so
// the unitary costs 2 (rotation) + 2 a phase multiply-adds an amplitude, where
// the dense 2x2 of the general programs costs 8.  What is divided out is one
// scalar for the whole state, multiplied back at the end of the plan.  Three
// more rules shorten the programs:
// - a left phase commutes with diagonal gates and CX controls and moves into
//   the right phase of the next one-qubit unitary on its qubit;
// - a two-qubit phase waits for the next one-qubit unitary on one of its
//   qubits and then is a factor of that unitary's right phase, chosen by the
//   other qubit's bit (one multiply a thread instead of one for half of its
//   amplitudes), unless both qubits are register slots;
// - CX and SWAP gates change no amplitudes: they change the labels (tile
//   indices) a thread's amplitudes carry, and the next re-mapping writes them
//   to their new places;
// - an X moves on through the gates after it into the next one-qubit unitary
//   on its qubit, at no cost, or is a label change where there is none.  A
//   unitary whose rotation is by more than 45 degrees is an X after one by
//   less, so tangents are small, and an X, a Y or any other unitary without a
//   diagonal moves the amplitudes and nothing else.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <complex>
#include <cstring>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include "qk_internal.h"

namespace qk {

int run_tasks(size_t n, const std::function<int(size_t)> &task) {
    return no_throw([&]() -> int {
        std::vector<int> rc(n, QK_OK);
        std::vector<std::string> what(n);
        std::atomic<size_t> next{0};
        auto work = [&]() {
            for (size_t i = next++; i < n; i = next++) {
                rc[i] = no_throw([&]() { return task(i); });
                if (rc[i]) no_throw([&]() { return what[i] = qk_last_error(), QK_OK; });
            }
        };
        const size_t threads = std::min<size_t>(n, std::max(1u, std::thread::hardware_concurrency()));
        std::vector<std::thread> pool;
        pool.reserve(threads);
        try {
            for (size_t t = 1; t < threads; ++t) pool.emplace_back(work);
        } catch (const std::system_error &) {
            // no more threads: those that run, and this one, take the tasks
        } catch (const std::bad_alloc &) {
            // (the same)
        }
        work();
        for (std::thread &t : pool) t.join();
        for (size_t i = 0; i < n; ++i)
            if (rc[i]) return fail(rc[i], "%s", what[i].c_str());
        return QK_OK;
    });
}

// Tile and register bits of factored passes.  complex128: 1024-amplitude
// tiles, 16 amplitudes a thread (64 threads, eight CTAs an SM); with 2048 the
// 28-qubit 20-layer brick circuit takes as long (65 ms) and the 28-qubit QFT
// 25.0 against 23.9 ms, with 8 amplitudes a thread the brick takes 91 ms.
// complex64: 4096-amplitude tiles, 32 amplitudes a thread: 75 ms on the
// 29-qubit brick circuit against 76 ms with 2048 and 84 ms with 16 amplitudes.
// Up to 17 qubits (complex128 18) there are not tiles enough for that: 1024
// amplitudes, 8 a thread, so that more warps share a tile's chain of steps.
// Microseconds with the large shapes and with these, complex64: 16 qubits, 20
// brick layers 104 / 86, 12 HEA layers 178 / 147 (general programs 137, 145);
// 13 qubits 82 / 54 and 139 / 107 (94, 99); 19 qubits 139 / 162 and 229 / 262.
// complex128: 16 qubits 122 / 98 and 187 / 158 (174, 167); 18 qubits 158 / 139
// and 217 / 194 (203, 195); 19 qubits 198 / 201 and 279 / 279.  Between them,
// complex64 with 18 qubits: 2048, 16 a thread, 132 / 105 and 216 / 181 (167,
// 180).
// complex128 plans of little work a pass are bound by HBM and take 2048
// amplitudes where that means fewer passes (below 36 units a pass, a unitary
// 4, a two-qubit phase 1): 27 qubits, a layer of H 3.12 -> 2.55 ms, 2 HEA
// layers 9.54 -> 9.21 (general programs 10.3); above, 28 qubits, 12 HEA layers
// (53 units) 97.5 -> 100.8.
constexpr int kWideTileBits = 11;
constexpr size_t kPassWork = 36;
PlanOptions factored_plan_options(int dtype, int n) {
    PlanOptions o = default_plan_options(dtype, n);
    const bool c128 = dtype == QK_C128, small = n <= (c128 ? 18 : 17), mid = !c128 && n == 18;
    o.f_tile_bits = std::min(n, small || c128 ? 10 : mid ? 11 : 12);
    o.f_reg_bits = std::min(o.f_tile_bits, small ? 3 : c128 || mid ? 4 : 5);
    if (c128 && !small) o.f_wide_bits = kWideTileBits;
    o.f_flips = 1;
    o.f_full = c128;
    return o;
}

// Two-state passes, complex128 only: 512-amplitude tiles, 8 amplitudes of each
// state a thread (24-qubit HEA of 12 layers: 25.8 ms a sweep; 26.5 with 1024,
// 33.0 with 2048, 28.4 with 16 amplitudes).
PlanOptions factored_adjoint_options(int dtype, int n) {
    PlanOptions o = default_adjoint_options(dtype, n);
    if (dtype == QK_C128) {
        o.f_tile_bits = std::min(n, 9);
        o.f_reg_bits = std::min(o.f_tile_bits, 3);
        o.f_flips = o.f_full = 1;
    }
    return o;
}

namespace {

using cd = std::complex<double>;
// Scalars and the factors on their way to a coefficient, which alone is
// rounded to double (or to the state's type): with these in double the
// 28-qubit brick circuit was 7.6e-15 off in the 2-norm.
using cl = std::complex<long double>;

cd cget(const double *m, int k) { return {m[2 * k], m[2 * k + 1]}; }
void cset(double *m, int k, cd z) {
    m[2 * k] = z.real();
    m[2 * k + 1] = z.imag();
}
cl unit(cl z) { return z / std::sqrt(std::norm(z)); }
cd to_double(cl z) { return {(double)z.real(), (double)z.imag()}; }

// ---- gate list -> factored op list ------------------------------------------

// The phases of a one-qubit gate's factors, or -1 where it is not a unitary
// (a U1 matrix): a unitary times a scalar to a few units of rounding.
int phases_of(const qk_gate &g, const Op &op) {
    switch (g.kind) {
    case QK_GATE_RY: case QK_GATE_Y: return 0;
    case QK_GATE_H: case QK_GATE_X: return kRightPhase;   // R diag(1, -1)
    case QK_GATE_RX: return kRightPhase | kLeftPhase;
    default: break;
    }
    const cd a = cget(op.m, 0), b = cget(op.m, 1), c = cget(op.m, 2), d = cget(op.m, 3);
    const double r0 = std::norm(a) + std::norm(b), r1 = std::norm(c) + std::norm(d);
    const double off = std::abs(a * std::conj(c) + b * std::conj(d));
    if (!(r0 > 1e-6 && r0 < 1e6) || !(std::fabs(r0 - r1) <= 4e-15 * r0) || !(off <= 4e-15 * r0)) return -1;
    return kRightPhase | kLeftPhase | kGiven;
}

// A two-qubit diagonal of unit entries.
bool unit_diagonal(const Op &op) {
    for (int k = 0; k < 4; ++k)
        if (!(std::fabs(std::norm(cget(op.m, k)) - 1.0) <= 4e-15)) return false;
    return true;
}

bool factorable(const qk_gate &g, Op &op) {
    if (lower_gate(g, op)) return false;
    switch (op.kind) {
    case OP_DENSE1: {
        const int ph = phases_of(g, op);
        op.aux = ph;
        return ph >= 0;
    }
    case OP_DIAG2: return unit_diagonal(op);
    case OP_PHASE1: case OP_DIAG1: case OP_PHASE2: case OP_SWAP2: case OP_CX: case OP_PERM: return true;
    default: return false;
    }
}

// What the kernel has: conditions with the tile number in 32 bits, up to 512
// threads (256 where the register amplitudes take 256 bytes), five register
// bits for complex64 and four for complex128 (two states: complex128 with
// three), exchange places as 16-bit offsets.
bool sizes_fit(const PlanOptions &o, int n, int nstates) {
    const int T = o.f_tile_bits, r = o.f_reg_bits;
    const bool c128 = o.dtype == QK_C128;
    if (nstates == 2 && !c128) return false;
    return T >= 1 && T <= std::min(n, c128 ? 12 : 13) && n - T <= 31 && r >= std::min(2, T) &&
           r <= std::min(T, nstates == 2 ? 3 : c128 ? 4 : 5) && T - r <= (((c128 ? 16 : 8) << r) * nstates >= 256 ? 8 : 9);
}

// merge_one_qubit_runs for ops that carry their phases: the product of two
// has the outer phases, and both where a phase stands between two rotations.
void merge_runs(std::vector<Op> &ops, int n) {
    std::vector<long> last(n, -1);
    std::vector<Op> out;
    out.reserve(ops.size());
    for (const Op &op : ops) {
        if (one_qubit(op) && last[op.q[0]] >= 0) {
            Op &a = out[last[op.q[0]]];
            double x[8], y[8], z[8];
            as_matrix(a, x);
            as_matrix(op, y);
            mat2_mul(y, x, z);   // op after a
            const bool da = a.kind == OP_DENSE1, db = op.kind == OP_DENSE1;
            const int pa = a.aux & ~kGiven, pb = op.aux & ~kGiven;   // (a product is rounded here)
            if (!da && !db) {
                a.kind = OP_DIAG1;
                a.m[0] = z[0]; a.m[1] = z[1]; a.m[2] = z[6]; a.m[3] = z[7];
            } else {
                if (!da) a.aux = pb | kRightPhase;
                else if (!db) a.aux = pa | kLeftPhase;
                else if ((pb & kRightPhase) || (pa & kLeftPhase)) a.aux = kRightPhase | kLeftPhase;
                else a.aux = (pa & kRightPhase) | (pb & kLeftPhase);
                a.kind = OP_DENSE1;
                std::memcpy(a.m, z, sizeof z);
            }
            continue;
        }
        for (int k = 0; k < op.nq; ++k) last[op.q[k]] = -1;
        out.push_back(op);
        if (one_qubit(op)) last[op.q[0]] = (long)out.size() - 1;
    }
    ops.swap(out);
}

// The scalar of an OP_K, m[6..9]: high and low parts.
cl scalar_of(const Op &op) {
    return {(long double)op.m[6] + op.m[8], (long double)op.m[7] + op.m[9]};
}
void set_scalar(Op &op, cl g) {
    cset(op.m, 3, to_double(g));
    op.m[8] = (double)(g.real() - op.m[6]);
    op.m[9] = (double)(g.imag() - op.m[7]);
}

// Matrices whose rounding is further than this off the rotation form have the
// full one (complex128).  With all in the rotation form the 14-qubit 20-layer
// brick circuit (U3 and CZ) is 1.64e-15 off in the 2-norm, with the line here
// 1.32e-15, with all in the full form 1.22e-15; the general programs are
// 1.38e-15 off.  28 qubits: 66.4, 70.1 and 76.0 ms, the general programs 131.
constexpr long double kFullAbove = 0.8e-16L;

// OP_DENSE1 with phases aux and no tangent above 2^10 -> OP_K and its scalar.  t and the phases are rounded to the state's type here
// and the scalar's magnitude taken from the rounded values, so that their
// rounding does not change the norm.
// ph: a phase the upper half still lacks; *defer: not null where the left
// phase moves on instead, to be returned there.
// full: the full form may be taken.
cl extract(Op &op, int dtype, cl ph, bool full, cl *defer) {
    auto rounded = [&](long double x) { return dtype == QK_C64 ? (double)(float)x : (double)x; };
    cl a = cget(op.m, 0), b = cl(cget(op.m, 1)) * ph, c = cget(op.m, 2), d = cl(cget(op.m, 3)) * ph;
    const bool right = op.aux & kRightPhase, left = op.aux & kLeftPhase;
    if (right && left && std::norm(b) > 0 && std::norm(c) > 0) {
        // The form below has seven of a matrix's eight numbers.  What it leaves
        // out, the angle of -b c / (a d), is 0 in a unitary but not in a
        // rounded one; shared among the entries as the least squares have it,
        // it is off in the 2-norm.
        const cl bc = -b * c, ad = a * d, turn = bc * std::conj(ad);
        const long double sa = std::norm(a), sb = std::norm(b),
                          e = std::fabs(turn.imag()) < 1e-8L * turn.real() ? turn.imag() / turn.real() : std::arg(turn),
                          off = e * std::sqrt(sa * sb) / (sa + sb) / 2;
        if (full && std::fabs(off) > kFullAbove) {
            const cd B = to_double(b / a), F = to_double(c / d);
            const cl g = unit(a) * std::sqrt((sa + sb) / (1 + std::norm(cl(B))));
            const cl p = unit(d) * std::sqrt((std::norm(c) + std::norm(d)) / (1 + std::norm(cl(F)))) / g;
            if (defer) *defer = p;
            op.kind = OP_K;
            op.aux |= kFull;
            std::memset(op.m, 0, sizeof op.m);
            cset(op.m, 0, B);
            cset(op.m, 1, F);
            cset(op.m, 2, defer ? cd(1) : to_double(p));
            return g;
        }
        auto turned = [](long double x) { return std::fabs(x) < 1e-8L ? cl(1 - x * x / 2, x) : std::polar(1.0L, x); };
        const cl up = turned(e * sb / (sa + sb) / 2), down = turned(-e * sa / (sa + sb) / 2);
        a *= up, d *= up, b *= down, c *= down;
    }
    // M = g [[1, -t l], [p t, p l]].  The phases keep what modulus the
    // entries give them: a matrix that is a unitary to rounding is met to
    // rounding in all its entries
    const cl q = c / a;
    cl l = 1, p = 1;
    long double tan;
    if (!left) {
        tan = q.real();
        if (right) l = d / a;
    } else if (!right) {
        tan = -(b / a).real();
        p = d / a;
    } else {
        tan = std::sqrt(std::sqrt(std::norm(q * b) / std::norm(d)));
        if (tan > 0) p = q / tan;
        l = d / a / p;
    }
    const double t = rounded(tan);
    const cd lr(rounded(l.real()), rounded(l.imag()));
    cd pr(rounded(p.real()), rounded(p.imag()));
    const long double nl = std::norm(cl(lr)), np = defer ? std::norm(p) : std::norm(cl(pr)), tt = (long double)t * t;
    const cl g = unit(a) * std::sqrt((std::norm(a) + std::norm(b) + std::norm(c) + std::norm(d)) /
                                     (1 + tt * nl + np * (tt + nl)));
    if (defer) *defer = p, pr = 1;
    op.kind = OP_K;
    std::memset(op.m, 0, sizeof op.m);
    op.m[0] = t;
    cset(op.m, 1, lr);
    cset(op.m, 2, pr);
    return g;
}

bool is_sign(cd f) { return f.real() == -1.0 && std::fabs(f.imag()) < 2e-16; }   // CP(pi)

bool diagonal_on(const Op &op, int q) {
    switch (op.kind) {
    case OP_PHASE1: case OP_DIAG1: case OP_PHASE2: case OP_DIAG2: return true;
    case OP_CX: return op.q[op.aux] == q;
    default: return false;
    }
}

// An X on q after op: OP_X, or two rotations by 45 degrees (the sums of an
// amplitude with zero are exact).
void push_x(std::vector<Op> &out, int q, const PlanOptions &o) {
    Op x;
    std::memset(&x, 0, sizeof x);
    x.nq = 1;
    x.q[0] = q;
    x.kind = o.f_flips ? OP_X : OP_K;
    if (!o.f_flips) {
        x.aux = kRightPhase;
        x.m[0] = 1;
        cset(x.m, 1, -1);
        cset(x.m, 2, 1);
        set_scalar(x, std::sqrt(0.5L));
        out.push_back(x);
        cset(x.m, 1, 1);
    }
    out.push_back(x);
}

// Merged ops -> OP_K, OP_PHASE1, OP_PHASE2, OP_CX, OP_SWAP2, OP_GRAD, OP_PERM,
// OP_X and a scalar the list lacks at its end.  `scaled`: it has ops with a
// scalar.
void factor(std::vector<Op> &ops, int n, const PlanOptions &o, cl &tail, bool &scaled) {
    // next[i] bit k: after op i, the next op on q[k] that is not diagonal
    // there is a one-qubit unitary, which takes in a phase on that qubit;
    // bit 2 + k: some one-qubit unitary follows there, which takes in an X;
    // bit 4 + k: and so on all qubits that CX gates carry the X to on the way
    std::vector<char> dense(n, 0), later(n, 0), taken(n, 0), next(ops.size(), 0);
    auto moved = [](std::vector<char> &f, const Op &op) {   // what follows an op's qubits through its swaps
        const int k = op.kind == OP_SWAP2 || op.kind == OP_PERM ? op.nq / 2 : 0;
        for (int i = 0; i < k; ++i) std::swap(f[op.q[i]], f[op.q[k + i]]);
    };
    for (size_t i = ops.size(); i-- > 0;) {
        const Op &op = ops[i];
        for (int k = 0; k < std::min<int>(op.nq, 2); ++k)
            next[i] |= (dense[op.q[k]] ? 1 << k : 0) | (later[op.q[k]] ? 4 << k : 0) | (taken[op.q[k]] ? 16 << k : 0);
        if (op.kind == OP_PERM) std::fill(dense.begin(), dense.end(), 0);
        else
            for (int k = 0; k < op.nq; ++k)
                if (!diagonal_on(op, op.q[k])) dense[op.q[k]] = op.kind == OP_DENSE1;
        moved(later, op);
        moved(taken, op);
        if (op.kind == OP_DENSE1) later[op.q[0]] = taken[op.q[0]] = 1;
        if (op.kind == OP_CX) taken[op.q[op.aux]] &= taken[op.q[1 - op.aux]];
    }
    std::vector<cl> ph(n, 1);
    std::vector<char> has(n, 0), flip(n, 0);   // flip: an X on its way
    std::vector<char> factor_waits(n, 0);      // a two-qubit phase that is no sign, since the last unitary
    std::vector<Op> out;
    out.reserve(ops.size());
    tail = 1;   // scalar of the ops so far that no OP_K has taken
    scaled = false;
    auto phase1 = [&](int q, cl p, bool deferred) {
        if (deferred) {
            ph[q] *= p;
            has[q] = 1;
            return;
        }
        Op x;
        std::memset(&x, 0, sizeof x);
        x.kind = OP_PHASE1;
        x.nq = 1;
        x.q[0] = q;
        cset(x.m, 0, to_double(p));
        out.push_back(x);
    };
    for (size_t i = 0; i < ops.size(); ++i) {
        Op op = ops[i];
        const int q = op.q[0];
        const bool f0 = flip[q], f1 = op.nq > 1 && flip[op.q[1]];
        auto swapped = [&](int j, int k) {   // entries j and k of its matrix
            const cd x = cget(op.m, j);
            cset(op.m, j, cget(op.m, k));
            cset(op.m, k, x);
        };
        switch (op.kind) {
        case OP_DENSE1: {
            scaled = true;
            const cl rest = has[q] ? ph[q] : cl(1);
            if (has[q]) op.aux |= kRightPhase;
            has[q] = 0;
            ph[q] = 1;
            if (f0) swapped(0, 1), swapped(2, 3);
            // An X that costs label changes (and with them re-mappings: 106
            // against 97 ms on the 26-qubit HEA gradient, in segments of one
            // and a half layers) is made of tangents above 2^10 alone.
            flip[q] = std::norm(cget(op.m, 2)) > (next[i] & 16 ? 1 : 0x1p20) * std::norm(cget(op.m, 0));
            if (flip[q]) swapped(0, 2), swapped(1, 3);
            // (a rotation beside an X is one with a factor -1 on the right)
            if (f0 || flip[q]) op.aux |= kRightPhase;
            const cl a = cget(op.m, 0);
            if (cget(op.m, 1) == 0.0 && cget(op.m, 2) == 0.0 && std::fabs(std::norm(a) - 1) < 1e-15L) {
                tail *= a;   // a diagonal is left; unit entries: no gradient sees where its scalar goes
                const cl p = cl(cget(op.m, 3)) / a * rest;
                if (p != cl(1)) phase1(q, p, next[i] & 1);
            } else {
                const bool defer = (op.aux & kLeftPhase) && (next[i] & 1);
                // (a full unitary can have no other qubit's phase as its factor)
                const bool full = o.f_full && (op.aux & kGiven) && !factor_waits[q];
                set_scalar(op, tail * extract(op, o.dtype, rest, full, defer ? &ph[q] : nullptr));
                tail = 1;
                has[q] = defer;
                if (defer) op.aux &= ~kLeftPhase;
                out.push_back(op);
            }
            if (flip[q] && !(next[i] & 4)) push_x(out, q, o), flip[q] = 0;
            break;
        }
        case OP_PHASE1: {
            const cl p = cget(op.m, 0);
            if (f0) tail *= p, scaled = true;
            phase1(q, f0 ? cl(1) / p : p, next[i] & 1);
            break;
        }
        case OP_DIAG1:
            if (f0) swapped(0, 1);
            scaled = true;
            tail *= cl(cget(op.m, 0));
            phase1(q, cl(cget(op.m, 1)) / cl(cget(op.m, 0)), next[i] & 1);
            break;
        case OP_DIAG2: {
            if (f0) swapped(0, 1), swapped(2, 3);
            if (f1) swapped(0, 2), swapped(1, 3);
            const cl d0 = cget(op.m, 0), d1 = cget(op.m, 1), d2 = cget(op.m, 2), d3 = cget(op.m, 3);
            scaled = true;
            tail *= d0;
            phase1(op.q[0], d1 / d0, next[i] & 1);
            phase1(op.q[1], d2 / d0, next[i] & 2);
            op.kind = OP_PHASE2;
            cset(op.m, 0, to_double(unit(d3 * d0 / (d1 * d2))));
            out.push_back(op);
            break;
        }
        case OP_PHASE2: {
            if (f0 || f1) {   // w^(b0 b1) with b = 1 - b' on the flipped qubits
                const cl w = cget(op.m, 0);
                scaled = true;
                if (f0 && f1) tail *= w;
                if (f1) phase1(op.q[0], f0 ? cl(1) / w : w, next[i] & 1);
                if (f0) phase1(op.q[1], f1 ? cl(1) / w : w, next[i] & 2);
                if (f0 != f1) cset(op.m, 0, to_double(cl(1) / w));
            }
            // CP(pi) is (-1, 1.2e-16) and runs as a change of sign.  What is
            // dropped, exp(i e b0 b1), goes where it costs nothing: b0 b1 is
            // (b0 + b1) / 2 - 1 / 4, b0 / 2 or 1 / 4 on average (left out, it
            // was two thirds of the 28-qubit brick circuit's error)
            if (is_sign(cget(op.m, 0))) {
                const long double e = std::arg(-cl(cget(op.m, 0)));
                const int k0 = (next[i] & 1) != 0, k1 = (next[i] & 2) != 0;
                if (k0) phase1(op.q[0], std::polar(1.0L, e / 2), true);
                if (k1) phase1(op.q[1], std::polar(1.0L, e / 2), true);
                tail *= std::polar(1.0L, e * (1 - k0 - k1) / 4);
                scaled = true;
            }
            out.push_back(op);
            break;
        }
        case OP_CX: {
            out.push_back(op);
            const int ctl = op.q[op.aux], tgt = op.q[1 - op.aux];
            flip[tgt] ^= flip[ctl];
            if (flip[tgt] && !(next[i] & (4 << (1 - op.aux)))) push_x(out, tgt, o), flip[tgt] = 0;
            break;
        }
        case OP_GRAD:
            if (f0) {   // X G X: the Y and Z parts change sign
                const int gen = (int)op.m[0];
                if (gen == 2 || gen == 3) {
                    op.m[0] = 4;
                    op.m[gen + 1] = 1;
                }
                for (int k : {3, 4, 6, 7}) op.m[k] = -op.m[k];
            }
            out.push_back(op);
            break;
        default:
            moved(flip, op);
            out.push_back(op);
            break;
        }
        for (int k = 0; k < op.nq; ++k) {
            char &f = factor_waits[op.q[k]];
            if (op.kind == OP_PHASE2) f |= !is_sign(cget(op.m, 0));
            else if (!diagonal_on(op, op.q[k])) f = 0;
        }
    }
    if (tail != cl(1) && std::all_of(out.begin(), out.end(), [](const Op &x) { return x.kind == OP_PERM; })) {
        // the scalar is all there is to do: on a unitary of its own
        Op x;
        std::memset(&x, 0, sizeof x);
        x.kind = OP_K;
        x.nq = 1;
        cset(x.m, 1, 1);
        cset(x.m, 2, 1);
        set_scalar(x, tail);
        tail = 1;
        out.insert(out.begin(), x);
    }
    ops.swap(out);
}

// ---- passes -----------------------------------------------------------------

bool is_work(const Op &op) { return op.kind == OP_K || op.kind == OP_GRAD; }

// Tile bits an op needs (its register slot, or the labels it changes).
int tile_bits_of(const Op &op, int (&b)[2]) {
    switch (op.kind) {
    case OP_K: case OP_GRAD: case OP_X: b[0] = op.q[0]; return 1;
    case OP_CX: b[0] = op.q[1 - op.aux]; return 1;
    case OP_SWAP2: b[0] = op.q[0]; b[1] = op.q[1]; return 2;
    default: return 0;
    }
}

// What the walks below look at, 16 bytes an op.
struct Lite {
    uint16_t cost;
    uint8_t nq, nb, work, perm;
    uint8_t q[2], diag[2], b[2];   // qubits, whether diagonal there, tile bits
};

// A factored op list in its two orders.
struct List {
    std::vector<Op> ops;
    cl tail = 1;              // scalar the ops leave out
    bool scaled = false;
    std::vector<Lite> lite;
    std::vector<size_t> order[2], rank[2];   // the ops as given and in ASAP layers; an op's place there
};

// Bytes of a pass's shared memory an op adds: steps, coefficients, accumulators.
size_t cost(const Op &op, size_t c, int threads_log) {
    switch (op.kind) {
    case OP_K: return 40 + 3 * c;   // a share of the re-mappings included
    case OP_GRAD: {
        const size_t k = (int)op.m[0] == 5 ? 2 : 1;
        return 16 + k * (2 * c + (sizeof(double) << threads_log));
    }
    case OP_SWAP2: return 64;
    default: return 24 + 4 * c;   // (a condition's share of the tables)
    }
}
void make_lite(List &list, size_t amp_bytes, int threads_log) {
    const auto &ops = list.ops;
    auto &lite = list.lite;
    lite.resize(ops.size());
    for (size_t i = 0; i < ops.size(); ++i) {
        const Op &op = ops[i];
        Lite &x = lite[i];
        std::memset(&x, 0, sizeof x);
        x.perm = op.kind == OP_PERM;
        if (x.perm) continue;
        x.cost = (uint16_t)std::min<size_t>(cost(op, amp_bytes, threads_log), 65535);
        x.nq = (uint8_t)op.nq;
        int b[2];
        x.nb = (uint8_t)tile_bits_of(op, b);
        for (int k = 0; k < op.nq; ++k) x.q[k] = (uint8_t)op.q[k], x.diag[k] = diagonal_on(op, op.q[k]);
        for (int k = 0; k < x.nb; ++k) x.b[k] = (uint8_t)b[k];
        x.work = is_work(op) ? 4 : op.kind == OP_CX || op.kind == OP_SWAP2 ? 1 : 0;
    }
}

struct Builder {
    const List &list;
    bool asap;
    int n, T, r, L;
    HostPlan &plan;
    const PlanOptions &opts;
    bool lookahead;
    const std::vector<Op> &ops = list.ops;
    const std::vector<Lite> &lite = list.lite;
    cl carry = 1;        // scalar of the ops so far, which the stored state lacks
    int grad_base = 0;
    bool mapped = false;   // the last step is a re-mapping
    // the TOP_LAYER being collected: its unitaries by slot
    struct Layer {
        int k = 0, signs = 0;   // masks
        bool pending = false, full = false;
        uint16_t w[8] = {0};
        uint32_t u[8] = {0};
        cd t[kPassMaxReg], l[kPassMaxReg];
    } layer = Layer();

    size_t amp_bytes() const { return plan.dtype == QK_C128 ? 16 : 8; }

    // Shared memory a pass's program, coefficients and gradient accumulators
    // may take besides the tile.
    size_t budget() const {
        const size_t tile = (amp_bytes() << T) * plan.nstates;
        return std::min<size_t>(48u << 10, (200u << 10) - tile);
    }
    // Walk pending ops in order; an op joins a pass on tile bits inB when no
    // op left out before it fails to commute with it on a shared qubit, its
    // tile bits are there (or, with grow, can be added) and the budget allows.
    // blocked: 1 an op diagonal on the qubit was left out, 2 another op.
    template <typename F>
    void walk(const std::vector<size_t> &pending, std::vector<char> &inB, int *grow, F &&each) const {
        char blocked[64] = {0};
        size_t used = 256;
        const size_t lim = budget();
        for (size_t i : pending) {
            const Lite &op = lite[i];
            bool ok = !op.perm && (used == 256 || used + op.cost <= lim);
            for (int k = 0; k < op.nq && ok; ++k) ok = blocked[op.q[k]] <= op.diag[k];
            if (ok && op.nb) {
                int need = 0;
                for (int k = 0; k < op.nb; ++k) need += !inB[op.b[k]];
                ok = need == 0 || (grow && *grow + need <= T);
                if (ok && need)
                    for (int k = 0; k < op.nb; ++k)
                        if (!inB[op.b[k]]) inB[op.b[k]] = 1, ++*grow;
            }
            if (ok) {
                used += op.cost;
            } else if (op.perm) {
                std::memset(blocked, 2, sizeof blocked);
            } else {
                for (int k = 0; k < op.nq; ++k)
                    blocked[op.q[k]] = std::max<char>(blocked[op.q[k]], op.diag[k] ? 1 : 2);
            }
            each(i, ok);
        }
    }

    // The same walk on tile bits B (a mask) that do not grow, for the work
    // that joins alone: qubits as bits, up to where no more can.
    struct Masks {
        uint64_t diag, other, tile;   // qubits it is diagonal on, its other qubits, tile bits
        uint16_t cost;
        uint8_t work, perm;
    };
    static size_t count(const std::vector<Masks> &pending, uint64_t B, size_t lim) {
        uint64_t left = 0, left_other = 0;   // qubits of ops left out / of those not diagonal there
        size_t used = 256, work = 0;
        for (const Masks &op : pending) {
            if (!op.perm && !(left_other & op.diag) && !(left & op.other) && !(op.tile & ~B) &&
                (used == 256 || used + op.cost <= lim)) {
                used += op.cost;
                work += op.work;
                continue;
            }
            if (op.perm) break;
            left |= op.diag | op.other;
            left_other |= op.other;
            if (!(B & ~left)) break;
        }
        return work;
    }

    // Tile bits grown ahead: the first ops' bits, then one at a time the
    // qubit of the next pending ops that lets the most work join.
    void choose_tile(const std::vector<size_t> &pending, std::vector<char> &inB, int &nB) const {
        std::vector<Masks> masks(pending.size());
        for (size_t j = 0; j < pending.size(); ++j) {
            const Lite &op = lite[pending[j]];
            Masks &m = masks[j];
            m = {0, 0, 0, op.cost, op.work, op.perm};
            for (int k = 0; k < op.nq; ++k) (op.diag[k] ? m.diag : m.other) |= 1ull << op.q[k];
            for (int k = 0; k < op.nb; ++k) m.tile |= 1ull << op.b[k];
        }
        uint64_t B = 0;
        for (int q = 0; q < n; ++q) B |= (uint64_t)(inB[q] != 0) << q;
        const size_t lim = budget();
        size_t base = count(masks, B, lim);
        while (nB < T) {
            int cands[64], ncands = 0;
            uint64_t cand = B;
            for (size_t j = 0, seen = 0; j < pending.size() && seen < 64; ++j) {
                const Lite &op = lite[pending[j]];
                seen += op.nb > 0;
                for (int k = 0; k < op.nb; ++k) {
                    if (!((cand >> op.b[k]) & 1)) cands[ncands++] = op.b[k];
                    cand |= 1ull << op.b[k];
                }
            }
            if (!ncands) break;
            int best = -1;
            size_t bestc = base;
            for (int k = 0; k < ncands; ++k) {
                const size_t c = count(masks, B | 1ull << cands[k], lim);
                if (c > bestc) best = cands[k], bestc = c;
            }
            if (best < 0) best = cands[0];   // the earliest: a later choice may need it
            inB[best] = 1;
            B |= 1ull << best;
            ++nB;
            base = bestc;
        }
    }

    // The ops cut into passes: the ops of each and its tile bits.
    struct Part {
        std::vector<size_t> take;
        std::vector<int> B;      // empty: a permutation pass, take[0]
    };
    std::vector<Part> parts = {};
    int partition() {
        std::vector<size_t> pending = list.order[asap], rest;
        while (!pending.empty()) {
            Part p;
            if (lite[pending[0]].perm) {
                p.take.push_back(pending[0]);
                pending.erase(pending.begin());
                parts.push_back(std::move(p));
                continue;
            }
            std::vector<char> inB(n, 0);
            int nB = 0;
            for (int q = 0; q < std::min(n, L); ++q) inB[q] = 1, ++nB;
            if (lookahead) choose_tile(pending, inB, nB);
            rest.clear();
            walk(pending, inB, &nB, [&](size_t i, bool ok) {
                (ok ? p.take : rest).push_back(i);
            });
            if (p.take.empty())
                return fail(QK_ERR_ARG, "tile_bits %d: an operation needs %d tile qubits", T, lite[pending[0]].nb);
            defer(p.take, rest);
            for (int q = 0; q < n && nB < T; ++q)
                if (!inB[q]) inB[q] = 1, ++nB;
            for (int q = 0; q < n; ++q)
                if (inB[q]) p.B.push_back(q);
            parts.push_back(std::move(p));
            pending.swap(rest);
        }
        return QK_OK;
    }

    // limit: give up (plan.nremaps at least that) where the plan is no better
    int compile_parts(size_t limit) {
        size_t last = parts.size();   // the last compute pass
        while (last && parts[last - 1].B.empty()) --last;
        for (size_t k = 0; k < parts.size(); ++k) {
            if (!parts[k].B.empty()) {
                int rc = compile(parts[k].take, parts[k].B, k + 1 == last, limit);
                if (rc || plan.nremaps >= limit) return rc;
                continue;
            }
            flush();
            HostPlan one;
            int rc = build_perm_plan(ops[parts[k].take[0]], n, opts, one);
            if (rc) return rc;
            plan.passes.push_back(one.passes[0]);
            plan.ngates += 1;
        }
        return QK_OK;
    }

    // Ops of the pass that no unitary or gradient of it follows wait for a
    // later pass when one does there: a phase then joins that unitary, a CX
    // the re-mapping before it.
    void defer(std::vector<size_t> &take, std::vector<size_t> &rest) const {
        std::vector<char> touched(n, 0);   // by ops of rest: 1 diagonal only, 2 else
        bool any = false;
        for (size_t i : rest)
            if (ops[i].kind != OP_PERM)
                for (int k = 0; k < ops[i].nq; ++k)
                    touched[ops[i].q[k]] = std::max<char>(touched[ops[i].q[k]], diagonal_on(ops[i], ops[i].q[k]) ? 1 : 2);
        std::vector<char> keep(take.size(), 0), need(n, 0);   // need: by kept ops, as touched
        for (size_t k = take.size(); k-- > 0;) {
            const Op &op = ops[take[k]];
            // (an X comes after the qubit's last unitary)
            bool kp = is_work(op) || op.kind == OP_X, later = false;
            for (int j = 0; j < op.nq; ++j) {
                const bool dg = diagonal_on(op, op.q[j]);
                kp = kp || need[op.q[j]] > (dg ? 1 : 0);
                later = later || touched[op.q[j]] > (dg ? 1 : 0);
            }
            kp = kp || !later;
            keep[k] = kp;
            any = any || kp;
            if (kp)
                for (int j = 0; j < op.nq; ++j)
                    need[op.q[j]] = std::max<char>(need[op.q[j]], diagonal_on(op, op.q[j]) ? 1 : 2);
        }
        if (!any) return;
        std::vector<size_t> t2;
        for (size_t k = 0; k < take.size(); ++k)
            (keep[k] ? t2 : rest).push_back(take[k]);
        take.swap(t2);
        std::sort(rest.begin(), rest.end(), [&](size_t a, size_t b) { return list.rank[asap][a] < list.rank[asap][b]; });
    }

    // ---- one pass ----
    struct Span {
        const int *b, *e;
        const int *begin() const { return b; }
        const int *end() const { return e; }
    };
    struct Pass {
        std::vector<size_t> idx;
        std::vector<int> work;       // positions of unitaries and gradients not yet done
        std::vector<int> other;      // and of the others
        std::vector<int> pred_list, pred0;   // op k's predecessors: pred_list[pred0[k] .. pred0[k + 1])
        Span preds(int k) const { return {pred_list.data() + pred0[k], pred_list.data() + pred0[k + 1]}; }
        std::vector<char> done;
        std::vector<int> local, Q;   // state bit -> tile bit or -1; slots (tile bits, ascending)
        uint32_t qmask = 0;          // the bits of Q
        std::vector<int> outer;      // state bit outside the tile -> bit of the tile number
        std::vector<char> dirty;     // per state bit: 1 CX control, 2 label changed since the re-mapping
        size_t left = 0, work_left = 0;
        std::vector<int> head, next_work;   // a qubit's work in order: the first, and after each the next, or -1
        std::vector<int> phases;            // (of mark_work)
    };

    int slot(const Pass &P, int q) const {
        const int b = P.local[q];
        if (b < 0) return -1;
        const auto it = std::find(P.Q.begin(), P.Q.end(), b);
        return it == P.Q.end() ? -1 : (int)(it - P.Q.begin());
    }
    bool is_slot(const Pass &P, int q) const { return P.local[q] >= 0 && ((P.qmask >> P.local[q]) & 1); }
    bool is_phase(const Op &op) const { return op.kind == OP_PHASE1 || op.kind == OP_PHASE2; }
    bool is_phase(const Lite &op) const { return !op.nb && !op.perm; }

    // Undone predecessors of op k that are phases which can run now; false
    // when another predecessor is undone.
    bool pending_phases(const Pass &P, int k, std::vector<int> *out) const {
        out->clear();
        for (int p : P.preds(k)) {
            if (P.done[p]) continue;
            const Lite &o = lite[P.idx[p]];
            if (!is_phase(o)) return false;
            for (int j = 0; j < o.nq; ++j)
                if (P.dirty[o.q[j]] > 1) return false;
            for (int pp : P.preds(p))
                if (!P.done[pp]) return false;
            out->push_back(p);
        }
        return true;
    }

    // Run (emit) the work that can run under slots P.Q.
    void run_work(Pass &P) {
        std::vector<int> ph;
        for (bool progress = true; progress;) {
            progress = false;
            for (int k : P.work) {
                const int q = lite[P.idx[k]].q[0];
                if (P.done[k] || !is_slot(P, q) || P.dirty[q]) continue;
                if (!pending_phases(P, k, &ph)) continue;
                const Op &op = ops[P.idx[k]];
                for (int p : ph) P.done[p] = 1;
                P.done[k] = 1;
                progress = true;
                P.left -= 1 + ph.size();
                --P.work_left;
                if (op.kind == OP_K) emit_k(P, op, ph);
                else {
                    for (int p : ph) emit_phase(P, ops[P.idx[p]]);
                    emit_grad(P, op);
                }
            }
        }
        trim(P, P.work);
    }
    static void trim(const Pass &P, std::vector<int> &list) {
        list.erase(std::remove_if(list.begin(), list.end(), [&](int k) { return P.done[k] != 0; }), list.end());
    }

    // Mark done what can run when qubit q joins the slots among `slots`, under
    // which nothing more can: q's next work, then what that lets run.  What is
    // marked goes to `marked`; returns the number of unitaries and gradients.
    size_t mark_work(Pass &P, std::vector<int> &slots, int q, std::vector<int> &marked) const {
        size_t cnt = 0;
        auto run_queue = [&](int x) {   // x's work, in order
            size_t before = cnt;
            for (int k = P.head[x]; k >= 0; k = P.next_work[k]) {
                if (P.done[k]) continue;
                if (P.dirty[x] || !pending_phases(P, k, &P.phases)) break;
                for (int p : P.phases) P.done[p] = 1, marked.push_back(p);
                P.done[k] = 1;
                marked.push_back(k);
                ++cnt;
            }
            return cnt != before;
        };
        if (!run_queue(q)) return 0;
        for (bool progress = true; progress;) {
            progress = false;
            for (int x : slots) progress = run_queue(x) || progress;
            progress = run_queue(q) || progress;
        }
        return cnt;
    }

    // CX, SWAP and X labels (and, once no work is left, the remaining phases).
    bool run_labels(Pass &P) {
        bool changed = false;
        std::vector<int> ph;
        for (bool progress = true; progress;) {
            progress = false;
            for (int k : P.other) {
                if (P.done[k]) continue;
                const Op &op = ops[P.idx[k]];
                if (is_phase(op)) {
                    if (P.work_left) continue;
                    bool ok = true;
                    for (int j = 0; j < op.nq; ++j) ok = ok && P.dirty[op.q[j]] < 2;
                    for (int p : P.preds(k)) ok = ok && P.done[p];
                    if (!ok) continue;
                    emit_phase(P, op);
                } else {
                    if (!pending_phases(P, k, &ph)) continue;
                    for (int p : ph) {
                        emit_phase(P, ops[P.idx[p]]);
                        P.done[p] = 1;
                        --P.left;
                    }
                    changed = true;
                    if (op.kind == OP_X) {
                        label(P, op.q[0], -1);
                        P.dirty[op.q[0]] = 2;
                    } else if (op.kind == OP_CX) {
                        label(P, op.q[1 - op.aux], op.q[op.aux]);
                        P.dirty[op.q[op.aux]] = std::max<char>(P.dirty[op.q[op.aux]], 1);
                        P.dirty[op.q[1 - op.aux]] = 2;
                    } else {
                        label(P, op.q[0], op.q[1]);
                        label(P, op.q[1], op.q[0]);
                        label(P, op.q[0], op.q[1]);
                        P.dirty[op.q[0]] = P.dirty[op.q[1]] = 2;
                    }
                }
                P.done[k] = 1;
                --P.left;
                progress = true;
            }
        }
        trim(P, P.other);
        return changed;
    }

    // 16 bytes that belong to the step before.
    void word(const void *p, size_t bytes) {
        TOp x;
        std::memset(&x, 0, sizeof x);
        std::memcpy(&x, p, bytes);
        plan.ops.push_back(x);
    }
    // The collected layer as a step.
    void flush() {
        if (!layer.k && !layer.signs) return;
        const Layer y = layer;
        layer = Layer();
        bool words = false;
        for (int s = 0; s < kPassMaxReg; ++s) words = words || y.u[s] || y.w[s];
        TOp &t = step(TOP_LAYER);
        t.a = (uint8_t)y.k;
        t.b = (uint8_t)((words ? kLayerWords : 0) | (y.signs ? kLayerSigns : 0) |
                        (y.pending ? kLayerPending : 0) | (y.full ? kLayerFull : 0));
        t.bits[0] = (uint8_t)y.signs;
        t.bits[1] = (uint8_t)(y.signs >> 8);
        if (words) {
            t.nbits = 2;   // u[0..3]; u[4] and w[0..4]
            word(y.u, 16);
            unsigned char b[16] = {0};
            std::memcpy(b, y.u + 4, 4);
            std::memcpy(b + 4, y.w, 10);
            word(b, 16);
        }
        for (int s = 0; s < kPassMaxReg; ++s) {
            if (!((y.k >> s) & 1)) continue;
            push(y.t[s]);
            push(y.l[s]);
        }
    }
    TOp &step(uint8_t kind) {
        flush();
        // steps under one re-mapping count as one program operation
        if (kind == TOP_REMAP) ++plan.nremaps;
        else if (mapped) ++plan.nbodies;
        mapped = kind == TOP_REMAP;
        TOp t;
        std::memset(&t, 0, sizeof t);
        t.kind = kind;
        t.coef = (uint32_t)(plan.coef.size() / 2);
        plan.ops.push_back(t);
        return plan.ops.back();
    }
    void push(cd z) {
        plan.coef.push_back(z.real());
        plan.coef.push_back(z.imag());
    }
    uint8_t code(const Pass &P, int q) const {
        return P.local[q] >= 0 ? (uint8_t)P.local[q] : (uint8_t)(kOuterFlag | q);
    }
    void label(const Pass &P, int target, int control) {   // (control -1: an X)
        TOp &t = step(TOP_LCX);
        t.a = (uint8_t)P.local[target];
        t.b = control < 0 ? kNoQubit : code(P, control);
    }
    void remap(Pass &P, const std::vector<int> &Q, bool dirty) {
        P.Q = Q;
        std::sort(P.Q.begin(), P.Q.end());
        P.qmask = 0;
        for (int b : P.Q) P.qmask |= 1u << b;
        std::fill(P.dirty.begin(), P.dirty.end(), 0);
        TOp &t = step(TOP_REMAP);
        t.nbits = 1;
        t.b = dirty;
        uint16_t off[kPassMaxReg] = {0};
        for (int s = 0; s < r; ++s) {
            t.bits[s] = (uint8_t)P.Q[s];
            off[s] = (uint16_t)(tile_swizzle(1u << P.Q[s], plan.dtype == QK_C128) * amp_bytes());
        }
        word(off, sizeof off);
    }
    void emit_phase(Pass &P, const Op &op) {
        const int sa = slot(P, op.q[0]), sb = op.nq > 1 ? slot(P, op.q[1]) : -1;
        if (sa >= 0 && sb >= 0 && is_sign(cget(op.m, 0))) {
            // the layer's signs come before its unitaries
            if (((layer.k >> sa) | (layer.k >> sb)) & 1) flush();
            layer.signs ^= 1 << slot_pair(std::min(sa, sb), std::max(sa, sb));
            return;
        }
        if (sa >= 0 && sb >= 0) {
            step((uint8_t)(TOP_PH2 + slot_pair(std::min(sa, sb), std::max(sa, sb))));
        } else {
            TOp &t = step(TOP_PHASE);
            t.a = code(P, op.q[0]);
            t.b = op.nq > 1 ? code(P, op.q[1]) : kNoQubit;
            t.bits[0] = sa >= 0 ? (uint8_t)sa : kNoSlot;
            t.bits[1] = sb >= 0 ? (uint8_t)sb : kNoSlot;
        }
        push(cget(op.m, 0));
    }
    void emit_k(Pass &P, const Op &op, const std::vector<int> &ph) {
        // conditions: phases whose other qubit is the same for all of a
        // thread's amplitudes; those between two slots run as steps before
        std::vector<std::pair<uint8_t, cd>> cond;
        for (int p : ph) {
            const Op &o = ops[P.idx[p]];
            const int x = o.nq == 1 ? -1 : o.q[0] == op.q[0] ? o.q[1] : o.q[0];
            // (a full unitary's conditions are signs)
            if (x >= 0 && (slot(P, x) >= 0 || ((op.aux & kFull) && !is_sign(cget(o.m, 0))))) {
                emit_phase(P, o);
                continue;
            }
            const cd f = cget(o.m, 0);
            cond.push_back({x < 0 ? kNoQubit : (uint8_t)(code(P, x) | (is_sign(f) ? kSignFlag : 0)), f});
        }
        // Amplitudes grow by 1 / |scalar|.  Before their magnitude is 2^16
        // (2^48 for complex128) times their own it is set back, by a power of
        // two: exact, and so much closer to the type's largest number an
        // amplitude may be.
        const long double range = plan.dtype == QK_C128 ? 0x1p-48L : 0x1p-16L, after = std::abs(carry * scalar_of(op));
        if (!(after >= range && after <= 1 / range)) {
            const int lim = plan.dtype == QK_C128 ? 500 : 60;
            const double f = std::ldexp(1.0, std::max(-lim, std::min(lim, std::ilogb(std::abs(carry)))));
            if (f != 1) {
                step(TOP_SCALE);
                push(f);
                carry /= f;
            }
        }
        carry *= scalar_of(op);
        bool simple = true;   // conditions that only change the sign
        for (const auto &c : cond) simple = simple && c.first != kNoQubit && (c.first & kSignFlag);
        const int s = slot(P, op.q[0]);
        if (!simple) {
            // tables of the factors' products, the right phase and factors
            // without a condition in the first
            cl all = (op.aux & kRightPhase) ? cl(cget(op.m, 1)) : cl(1);
            std::vector<std::pair<uint8_t, cd>> bits;
            for (const auto &c : cond) {
                if (c.first == kNoQubit) all *= cl(c.second);
                else bits.push_back({(uint8_t)(c.first & ~kSignFlag), c.second});
            }
            for (size_t c0 = 0; c0 < bits.size() || c0 == 0; c0 += 8) {
                TOp &t = step(TOP_LAM);
                t.nbits = (uint8_t)std::min<size_t>(8, bits.size() - c0);
                for (int i = 0; i < t.nbits; ++i) {
                    const uint8_t c = bits[c0 + i].first;
                    t.bits[i] = (c & kOuterFlag) ? (uint8_t)(kOuterFlag | P.outer[c & 0x3F]) : c;
                }
                const int nb = t.nbits;
                for (int i0 = 0; i0 == 0 || i0 < nb; i0 += 4)
                    for (int i = 0; i < 16; ++i) {
                        // (full where a second one follows)
                        if (i >> std::min(4, nb - i0) && (i0 || nb <= 4)) break;
                        cl f = c0 == 0 && i0 == 0 ? all : cl(1);
                        for (int k = 0; k < std::min(4, nb - i0); ++k)
                            if ((i >> k) & 1) f *= cl(bits[c0 + i0 + k].second);
                        push(to_double(f));
                    }
            }
        } else if (((layer.k >> s) & 1) || (layer.k && layer.full != ((op.aux & kFull) != 0))) {
            flush();
        }
        layer.k |= 1 << s;
        layer.full = (op.aux & kFull) != 0;
        layer.t[s] = cget(op.m, 0);
        layer.l[s] = cget(op.m, 1);
        if (!simple) {   // the pending factor is for this unitary alone
            layer.pending = true;
            flush();
        } else {
            for (const auto &c : cond) {
                if (c.first & kOuterFlag) layer.u[s] ^= 1u << P.outer[c.first & 0x3F];
                else layer.w[s] ^= (uint16_t)(1u << (c.first & 0x3F));
            }
        }
        if (op.aux & kLeftPhase) {
            TOp &t = step(TOP_PHASE);
            t.a = code(P, op.q[0]);
            t.b = kNoQubit;
            t.bits[0] = (uint8_t)s;
            t.bits[1] = kNoSlot;
            push(cget(op.m, 2));
        }
    }
    void emit_grad(Pass &P, const Op &op) {
        // both states lack the factor carry: the sums grow by its square
        const double f = (double)std::norm(carry);
        const int gen = (int)op.m[0];
        TOp &t = step(TOP_GRAD);
        t.a = (uint8_t)slot(P, op.q[0]);
        t.b = gen == 5 ? 5 : 4;
        auto param_slot = [&](int32_t p) {
            int k = grad_base;
            while (k < (int)plan.grad_params.size() && plan.grad_params[k] != p) ++k;
            if (k == (int)plan.grad_params.size()) plan.grad_params.push_back(p);
            return k - grad_base;
        };
        const int k1 = param_slot(op.aux);
        t.bits[0] = (uint8_t)(k1 & 0xFF);
        t.bits[1] = (uint8_t)(k1 >> 8);
        if (gen == 5) {
            const int k2 = param_slot((int32_t)op.m[8]);
            t.bits[2] = (uint8_t)(k2 & 0xFF);
            t.bits[3] = (uint8_t)(k2 >> 8);
        }
        const double a = gen == 1 ? 1 : gen >= 4 ? op.m[2] : 0, b = gen == 2 ? 1 : gen >= 4 ? op.m[3] : 0,
                     c = gen == 3 ? 1 : gen >= 4 ? op.m[4] : 0;
        push({f * a, f * b});
        push({f * c, 0});
        if (gen == 5) {
            push({f * op.m[5], f * op.m[6]});
            push({f * op.m[7], 0});
        }
    }

    // Slots for the next re-mapping: grown by the tile bit that lets the most
    // work run (ties: the bit of the earliest work), then the highest bits.
    // Under the first mapping the tile is loaded, so its slots leave the
    // lowest L bits to the threads (runs of contiguous amplitudes).
    std::vector<int> choose_slots(Pass &P, bool first, int lo) {
        std::vector<int> cand, Q;
        uint32_t seen = first ? (1u << lo) - 1 : 0;
        for (int k : P.work) {
            const int b = P.local[lite[P.idx[k]].q[0]];
            if (!((seen >> b) & 1)) cand.push_back(b);
            seen |= 1u << b;
            if (seen + 1 == 1u << T) break;
        }
        std::vector<int> qubits(T), slots, all, marked;   // state bits of the tile bits / of Q; what is marked done
        for (int q = 0; q < n; ++q)
            if (P.local[q] >= 0) qubits[P.local[q]] = q;
        auto undo = [&](std::vector<int> &m) {
            for (int k : m) P.done[k] = 0;
            m.clear();
        };
        while ((int)Q.size() < r && !cand.empty()) {
            int best = 0;
            size_t bestc = 0;
            for (size_t i = 0; i < cand.size(); ++i) {
                const size_t c = mark_work(P, slots, qubits[cand[i]], marked);
                undo(marked);
                if (c > bestc) best = (int)i, bestc = c;
            }
            const int q = qubits[cand[best]];
            if (bestc) mark_work(P, slots, q, all);
            slots.push_back(q);
            Q.push_back(cand[best]);
            cand.erase(cand.begin() + best);
        }
        undo(all);
        fill_high(Q);
        return Q;
    }
    void fill_high(std::vector<int> &Q) const {
        for (int b = T - 1; b >= 0 && (int)Q.size() < r; --b)
            if (std::find(Q.begin(), Q.end(), b) == Q.end()) Q.push_back(b);
    }

    int compile(const std::vector<size_t> &idx, const std::vector<int> &B, bool last_pass, size_t limit) {
        PassDesc d;
        std::memset(&d, 0, sizeof d);
        d.form = 1;
        d.T = (int)B.size();
        for (int k = 0; k < d.T; ++k) d.bpos[k] = B[k];
        while (d.L < d.T && d.bpos[d.L] == d.L) ++d.L;
        Pass P;
        P.idx = idx;
        P.local.assign(n, -1);
        for (int k = 0; k < d.T; ++k) P.local[B[k]] = k;
        P.outer.assign(n, -1);
        for (int q = 0, k = 0; q < n; ++q)
            if (P.local[q] < 0) P.outer[q] = k++;
        P.dirty.assign(n, 0);
        P.done.assign(idx.size(), 0);
        P.pred0.reserve(idx.size() + 1);
        P.pred0.push_back(0);
        P.pred_list.reserve(3 * idx.size());
        P.left = idx.size();
        // predecessors: ops that share a qubit and are not both diagonal on it
        std::vector<int> lastn(n, -1);
        std::vector<std::vector<int>> diags(n);
        for (size_t k = 0; k < idx.size(); ++k) {
            const Op &op = ops[idx[k]];
            (is_work(op) ? P.work : P.other).push_back((int)k);
            P.work_left += is_work(op);
            for (int j = 0; j < op.nq; ++j) {
                const int q = op.q[j];
                if (lastn[q] >= 0) P.pred_list.push_back(lastn[q]);
                if (diagonal_on(op, q)) {
                    diags[q].push_back((int)k);
                } else {
                    P.pred_list.insert(P.pred_list.end(), diags[q].begin(), diags[q].end());
                    diags[q].clear();
                    lastn[q] = (int)k;
                }
            }
            const auto mine = P.pred_list.begin() + P.pred0.back();
            std::sort(mine, P.pred_list.end());
            P.pred_list.erase(std::unique(mine, P.pred_list.end()), P.pred_list.end());
            P.pred0.push_back((int)P.pred_list.size());
        }
        P.head.assign(n, -1);
        P.next_work.assign(idx.size(), -1);
        for (size_t i = P.work.size(); i-- > 0;) {
            const int k = P.work[i], q = ops[idx[k]].q[0];
            P.next_work[k] = P.head[q];
            P.head[q] = k;
        }
        d.prog0 = (int)plan.ops.size();
        d.coef0 = (int)(plan.coef.size() / 2);
        d.grad0 = grad_base = (int)plan.grad_params.size();
        // slots of the first and last mapping stay off the lowest bits
        const int lo = T - L >= r ? L : 0;
        bool dirty = false;   // a label step has run since the last re-mapping
        remap(P, choose_slots(P, true, lo), false);
        for (bool first = true;; first = false) {
            const size_t before = P.left;
            run_work(P);
            dirty = run_labels(P) || dirty;
            if (!P.left) break;
            if (plan.nremaps >= limit) return QK_OK;
            if (!first && P.left == before) return fail(QK_ERR_ARG, "planner: a pass makes no progress");
            remap(P, choose_slots(P, false, lo), dirty);
            dirty = false;
        }
        flush();
        if (dirty || (!P.Q.empty() && P.Q[0] < lo)) {
            std::vector<int> Q;
            fill_high(Q);
            remap(P, Q, dirty);
        }
        if (list.scaled && last_pass) {
            TOp &t = step(TOP_SCALE);
            t.b = 1;
            push(to_double(carry * list.tail));
            carry = 1;
        }
        d.nprog = (int)plan.ops.size() - d.prog0;
        d.ncoef = (int)(plan.coef.size() / 2) - d.coef0;
        d.ngrad = (int)plan.grad_params.size() - d.grad0;
        for (int i = 0; i < d.nprog; ++i) {
            TOp &t = plan.ops[d.prog0 + i];
            if (t.kind == TOP_REMAP) d.last = i;
            else t.coef -= (uint32_t)d.coef0;
            if (t.kind == TOP_REMAP || t.kind == TOP_LAYER) i += t.nbits;   // the words after it
        }
        for (int s = 0; s < r; ++s) {
            d.fpos[s] = B[plan.ops[d.prog0].bits[s]];
            d.lpos[s] = B[plan.ops[d.prog0 + d.last].bits[s]];
        }
        plan.passes.push_back(d);
        plan.ngates += idx.size();
        return QK_OK;
    }
};

// The candidates of a plan: op lists, each in both orders and with both ways
// to choose tiles.  All are cut into passes; of those with the fewest passes
// the first and the last are compiled, the one with fewer re-mappings kept.
int build_best(std::vector<List> lists, int n, const PlanOptions &o, int nstates, HostPlan &plan) {
    PlanOptions fo = o;
    fo.tile_bits = o.f_tile_bits;
    const int L = pass_low_bits(fo, n);
    for (List &list : lists) {
        make_lite(list, o.dtype == QK_C128 ? 16 : 8, o.f_tile_bits - o.f_reg_bits);
        list.order[0].resize(list.ops.size());
        for (size_t i = 0; i < list.ops.size(); ++i) list.order[0][i] = i;
        list.order[1] = asap_positions(list.ops, n);
        for (int k = 0; k < 2; ++k) {
            list.rank[k].resize(list.ops.size());
            for (size_t i = 0; i < list.ops.size(); ++i) list.rank[k][list.order[k][i]] = i;
        }
    }
    struct Candidate {
        size_t list = 0;
        bool asap = false;
        std::vector<Builder::Part> parts;
    } first, last;
    HostPlan empty;
    empty.n = n;
    empty.dtype = o.dtype;
    empty.T = o.f_tile_bits;
    empty.r = o.f_reg_bits;
    empty.nstates = nstates;
    // (in one tile there is no choice of tiles)
    const size_t variants = n <= o.f_tile_bits ? 2 : 4;
    std::vector<Candidate> all(variants * lists.size());
    auto builder = [&](const Candidate &c, bool lookahead, HostPlan &hp) {
        return Builder{lists[c.list], c.asap, n, o.f_tile_bits, o.f_reg_bits, L, hp, o, lookahead};
    };
    auto candidate = [&](size_t k) {
        Candidate &c = all[k];
        c.list = k / variants;
        c.asap = k % 2;
        HostPlan hp = empty;
        Builder b = builder(c, k % variants >= 2, hp);
        const int rc = b.partition();
        c.parts.swap(b.parts);
        return rc;
    };
    // (threads take longer to start than candidates of fewer ops)
    const bool threads = o.threads && variants == 4 && lists[0].ops.size() >= 300;
    for (size_t k = 0; k < all.size() && !threads; ++k) {
        int rc = candidate(k);
        if (rc) return rc;
    }
    if (threads) {
        int rc = run_tasks(all.size(), candidate);
        if (rc) return rc;
    }
    bool have = false, two = false;
    for (Candidate &c : all) {
        if (have && c.parts.size() > first.parts.size()) continue;
        two = have && c.parts.size() == first.parts.size();
        std::swap(two ? last : first, c);
        have = true;
    }
    for (Candidate *c : {&first, &last}) {
        if (c == &last && !two) break;
        HostPlan hp = empty;
        Builder b = builder(*c, false, hp);
        b.parts.swap(c->parts);
        int rc = b.compile_parts(c == &first ? SIZE_MAX : plan.nremaps);
        if (rc) return rc;
        if (c == &first || hp.nremaps < plan.nremaps) plan = std::move(hp);
    }
    return QK_OK;
}

}  // namespace

// The gates lowered, where a factored program can run them.
static bool lower_factored(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, int nstates, std::vector<Op> *ops) {
    if (!sizes_fit(o, n, nstates)) return false;
    for (size_t i = 0; i < ng; ++i) {
        Op op;
        if (!factorable(gates[i], op)) return false;
        for (int k = 0; k < op.nq; ++k)
            if (op.q[k] < 0 || op.q[k] >= n) return false;
        if (ops) ops->push_back(op);
    }
    return true;
}

bool plan_is_factored(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, int nstates) {
    return lower_factored(gates, ng, n, o, nstates, nullptr);
}

static int forward(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, HostPlan &plan) {
    int rc = check_options(o, n);
    if (rc) return rc;
    std::vector<Op> lowered;
    lowered.reserve(ng);
    if (!lower_factored(gates, ng, n, o, 1, &lowered)) return build_plan(gates, ng, n, o, plan);
    bool swaps = false;
    for (const Op &op : lowered) swaps = swaps || (op.kind == OP_SWAP2 && op.aux != 1);
    // SWAP gates as label steps, or as renamings too
    std::vector<List> lists(swaps ? 2 : 1);
    for (size_t k = 0; k < lists.size(); ++k) {
        List &l = lists[k];
        if (k + 1 < lists.size()) l.ops = lowered;
        else l.ops = std::move(lowered);
        relabel_perms(l.ops, n, pass_low_bits(o, n), perm_tile_bits(o.dtype), 6, k > 0);
        merge_runs(l.ops, n);
        factor(l.ops, n, o, l.tail, l.scaled);
    }
    PlanOptions w = o;
    w.f_tile_bits = o.f_wide_bits;
    size_t work = 0;
    for (const Op &op : lists[0].ops) work += op.kind == OP_K ? 4 : op.kind == OP_PHASE2;
    const bool wide = o.f_wide_bits > o.f_tile_bits && sizes_fit(w, n, 1);
    std::vector<List> again;
    if (wide) again = lists;
    rc = build_best(std::move(lists), n, o, 1, plan);
    if (rc || !wide || work >= kPassWork * plan.passes.size()) return rc;
    HostPlan other;
    rc = build_best(std::move(again), n, w, 1, other);
    if (!rc && other.passes.size() < plan.passes.size()) plan = std::move(other);
    return rc;
}

static int adjoint(const qk_gate *gates, size_t ng, const int32_t *pidx, int n, const PlanOptions &o, HostPlan &plan) {
    int rc = check_options(o, n);
    if (rc) return rc;
    std::vector<Op> lowered;
    lowered.reserve(ng);
    if (!lower_factored(gates, ng, n, o, 2, &lowered)) return build_adjoint_plan(gates, ng, pidx, n, o, plan);
    std::vector<List> lists(1);
    std::vector<Op> &ops = lists[0].ops;
    ops.reserve(2 * ng);
    for (size_t i = ng; i-- > 0;) {
        Op &op = lowered[i];
        if (pidx && pidx[i] >= 0) {
            const int gen = gates[i].kind == QK_GATE_RX ? 1 : gates[i].kind == QK_GATE_RY ? 2 : gates[i].kind == QK_GATE_RZ ? 3 : 0;
            if (!gen) return fail(QK_ERR_UNSUPPORTED, "gate %zu: only RX, RY, RZ are trainable", i);
            Op g;
            std::memset(&g, 0, sizeof g);
            g.kind = OP_GRAD;
            g.nq = 1;
            g.q[0] = op.q[0];
            g.m[0] = gen;
            g.aux = pidx[i];
            ops.push_back(g);
        }
        invert_op(op);   // the inverse of each single gate has the gate's phases
        ops.push_back(op);
    }
    hoist_gradients(ops, n);
    merge_runs(ops, n);
    pair_gradients(ops);
    factor(ops, n, o, lists[0].tail, lists[0].scaled);
    return build_best(std::move(lists), n, o, 2, plan);
}

int plan_forward(const qk_gate *gates, size_t ng, int n, const PlanOptions &o, HostPlan &plan) {
    return no_throw([&]() { return forward(gates, ng, n, o, plan); });
}

int plan_adjoint(const qk_gate *gates, size_t ng, const int32_t *pidx, int n, const PlanOptions &o, HostPlan &plan) {
    return no_throw([&]() { return adjoint(gates, ng, pidx, n, o, plan); });
}

int build_group_plan(const qk_gate *gates, const int32_t *sizes, size_t ngroups, int n, const PlanOptions &o,
                     HostPlan &plan) {
    size_t ng = 0;
    for (size_t g = 0; g < ngroups; ++g) {
        if (sizes[g] < 0) return fail(QK_ERR_ARG, "group %zu has negative size", g);
        ng += (size_t)sizes[g];
    }
    // The groups bound nothing here: a tile can hold any qubits, and VSWAP
    // groups become renamings, so the gates of all groups are planned as one
    // gate list.
    return plan_forward(gates, ng, n, o, plan);
}

}  // namespace qk
