// CPU check of the factored planner (subquokka_dev_b200/csrc/qk_factor.cpp).
//
// The steps of factored plans are run by an emulator written from their
// definitions in qk_internal.h, with the labels of every thread and register
// element kept explicitly: an amplitude sits at the label its last
// re-mapping gave it, label steps change it, and the tile is stored under
// the last mapping.  Random circuits of unitary one-qubit gates, phases, CX
// and SWAP gates and VSWAPs with small tiles (many passes, re-mappings,
// conditions) against the dense simulation of the gate list; adjoint plans
// against the direct backward sweep.
// States and gradients agree within 1e-12 (1e-9 for gradients of circuits
// with H, whose truncated constant makes it a scaled unitary); complex64
// plans, whose coefficients are rounded to 24 bits, within 90 gates x 2
// coefficients x 2^-24 = 1.1e-5.
#include "dense_sim.h"

using namespace dense_sim;
using qk::HostPlan;
using qk::PassDesc;
using qk::TOp;

namespace {

struct Tile {
    const PassDesc &d;
    uint64_t base;
    int r, nthreads;
    std::vector<uint32_t> bm, tb;                  // slot masks, thread labels
    std::vector<std::vector<cd>> v;                // [state][thread * R + kk]
    uint32_t label(int t, int kk) const {
        uint32_t x = tb[t];
        for (int s = 0; s < r; ++s)
            if ((kk >> s) & 1) x ^= bm[s];
        return x;
    }
    void map_to(const TOp &op) {
        std::vector<char> reg(d.T, 0);
        for (int s = 0; s < r; ++s) {
            bm[s] = 1u << op.bits[s];
            reg[op.bits[s]] = 1;
            if (s && op.bits[s] <= op.bits[s - 1]) std::exit(2);   // ascending
        }
        for (int t = 0; t < nthreads; ++t) {
            tb[t] = 0;
            int j = 0;
            for (int b = 0; b < d.T; ++b)
                if (!reg[b]) tb[t] |= (uint32_t)((t >> j++) & 1) << b;
        }
    }
    bool bit(uint8_t code, int t) const {
        if (code == qk::kNoQubit) return true;
        if (code & qk::kOuterFlag) return (base >> (code & 0x3F)) & 1;
        // a condition must be the same for all of the thread's amplitudes
        for (int s = 0; s < r; ++s)
            if ((bm[s] >> (code & 0x3F)) & 1) {
                std::fprintf(stderr, "condition on a register slot\n");
                std::exit(2);
            }
        return (tb[t] >> (code & 0x3F)) & 1;
    }
};

void emulate(const HostPlan &hp, State &psi, State *lam, std::vector<double> &g) {
    const int n = hp.n, r = hp.r, R = 1 << r;
    State *states[2] = {&psi, lam};
    const int ns = lam ? 2 : 1;
    for (const PassDesc &d : hp.passes) {
        if (d.perm) {
            Op p;
            std::memset(&p, 0, sizeof p);
            p.kind = qk::OP_PERM;
            p.nq = 2 * d.nperm;
            for (int i = 0; i < d.nperm; ++i) {
                p.q[i] = d.perm == 2 ? d.perm_a[i] : d.bpos[d.perm_a[i]];
                p.q[d.nperm + i] = d.perm == 2 ? d.perm_b[i] : d.bpos[d.perm_b[i]];
            }
            std::vector<int> qs;
            const auto m = matrix_of(p, qs);
            for (int i = 0; i < ns; ++i) apply_matrix(*states[i], n, qs, m);
            continue;
        }
        if (d.form != 1) std::exit(2);
        const int T = d.T, NT = 1 << (T - r);
        std::vector<char> in(n, 0);
        for (int k = 0; k < T; ++k) in[d.bpos[k]] = 1;
        std::vector<int> outer;
        for (int q = 0; q < n; ++q)
            if (!in[q]) outer.push_back(q);
        const TOp *prog = hp.ops.data() + d.prog0;
        for (uint64_t o = 0; o < (1ull << outer.size()); ++o) {
            uint64_t base = 0;
            for (size_t k = 0; k < outer.size(); ++k)
                if ((o >> k) & 1) base |= 1ull << outer[k];
            auto addr = [&](uint32_t j) {
                uint64_t a = base;
                for (int k = 0; k < T; ++k)
                    if ((j >> k) & 1) a |= 1ull << d.bpos[k];
                return a;
            };
            Tile t{d, base, r, NT, std::vector<uint32_t>(r), std::vector<uint32_t>(NT), {}};
            t.v.assign(ns, std::vector<cd>((size_t)NT * R));
            t.map_to(prog[0]);
            for (int s = 0; s < r; ++s)
                if (d.fpos[s] != d.bpos[prog[0].bits[s]] || d.lpos[s] != d.bpos[prog[d.last].bits[s]]) std::exit(2);
            for (int i = 0; i < ns; ++i)
                for (int th = 0; th < NT; ++th)
                    for (int kk = 0; kk < R; ++kk) t.v[i][th * R + kk] = (*states[i])[addr(t.label(th, kk))];
            std::vector<cd> pend(NT, 1);
            bool dirty = false;
            for (int p = 2; p < d.nprog; ++p) {
                const TOp &op = prog[p];
                auto coef = [&](int k) {
                    const size_t i = (size_t)d.coef0 + op.coef + k;
                    if (op.coef + k >= (uint32_t)d.ncoef) std::exit(2);
                    return cd(hp.coef[2 * i], hp.coef[2 * i + 1]);
                };
                if (op.kind == qk::TOP_LAYER) {
                    uint16_t w[5] = {0};
                    uint32_t u[5] = {0};
                    const int signs = op.bits[0] | op.bits[1] << 8;
                    if (op.b & qk::kLayerWords) {
                        std::memcpy(u, &prog[p + 1], 16);
                        std::memcpy(u + 4, &prog[p + 2], 4);
                        std::memcpy(w, (const char *)&prog[p + 2] + 4, 10);
                        p += 2;
                    }
                    if (signs && !(op.b & qk::kLayerSigns)) std::exit(2);
                    for (int y = 1; y < r; ++y)
                        for (int x = 0; x < y; ++x)
                            if ((signs >> qk::slot_pair(x, y)) & 1)
                                for (auto &vec : t.v)
                                    for (int k = 0; k < NT * R; ++k)
                                        if (((k >> x) & 1) && ((k >> y) & 1)) vec[k] = -vec[k];
                    for (int s = 0, c = 0; s < r; ++s) {
                        if (!((op.a >> s) & 1)) continue;
                        const double t0 = coef(c++).real();
                        const cd right = coef(c++);
                        for (int th = 0; th < NT; ++th) {
                            for (int b = 0; b < T; ++b)
                                if ((w[s] >> b) & 1) t.bit((uint8_t)b, th);   // uniform
                            const int par = __builtin_parity(t.tb[th] & w[s]) ^ __builtin_parity((uint32_t)o & u[s]);
                            cd f = op.b & qk::kLayerPending ? pend[th] : right;
                            if (par) f = -f;
                            if (op.b & qk::kLayerPending) pend[th] = 1;
                            for (int i = 0; i < ns; ++i)
                                for (int kk = 0; kk < R; ++kk)
                                    if (!((kk >> s) & 1)) {
                                        cd &x = t.v[i][th * R + kk], &y = t.v[i][th * R + (kk | (1 << s))];
                                        const cd z = f * y, x0 = x;
                                        x = x0 - t0 * z;
                                        y = t0 * x0 + z;
                                    }
                        }
                    }
                } else if (op.kind == qk::TOP_REMAP) {
                    uint16_t off[5];
                    std::memcpy(off, &prog[++p], sizeof off);
                    const bool c128 = hp.dtype == QK_C128;
                    for (int s = 0; s < r; ++s)
                        if (off[s] != qk::tile_swizzle(1u << op.bits[s], c128) * (c128 ? 16 : 8)) std::exit(2);
                    if ((op.b != 0) != dirty) std::exit(2);
                    dirty = false;
                    for (int i = 0; i < ns; ++i) {
                        std::vector<cd> tile((size_t)1 << T);
                        for (int th = 0; th < NT; ++th)
                            for (int kk = 0; kk < R; ++kk) tile[t.label(th, kk)] = t.v[i][th * R + kk];
                        Tile u = t;
                        u.map_to(op);
                        for (int th = 0; th < NT; ++th)
                            for (int kk = 0; kk < R; ++kk) t.v[i][th * R + kk] = tile[u.label(th, kk)];
                    }
                    t.map_to(op);
                } else if (op.kind >= qk::TOP_PH2 && op.kind < qk::TOP_PH2 + 10) {
                    for (int b = 1; b < 5; ++b)
                        for (int a = 0; a < b; ++a)
                            if (op.kind - qk::TOP_PH2 == qk::slot_pair(a, b))
                                for (auto &x : t.v)
                                    for (int k = 0; k < NT * R; ++k)
                                        if (((k >> a) & 1) && ((k >> b) & 1)) x[k] *= coef(0);
                } else if (op.kind == qk::TOP_LAM) {
                    for (int th = 0; th < NT; ++th) {
                        int idx = 0;
                        for (int i = 0; i < op.nbits; ++i) {
                            const uint8_t c = op.bits[i];
                            const bool b = (c & qk::kOuterFlag) ? (o >> (c & 31)) & 1 : t.bit(c, th);
                            idx |= (int)b << i;
                        }
                        pend[th] *= coef(idx & 15);
                        if (op.nbits > 4) pend[th] *= coef(16 + (idx >> 4));
                    }
                } else if (op.kind == qk::TOP_LCX) {
                    dirty = true;
                    for (int th = 0; th < NT; ++th)
                        t.tb[th] ^= (uint32_t)((op.b & qk::kOuterFlag) ? (base >> (op.b & 0x3F)) & 1 : (t.tb[th] >> op.b) & 1) << op.a;
                    if (!(op.b & qk::kOuterFlag))
                        for (auto &m : t.bm) m ^= ((m >> op.b) & 1u) << op.a;
                } else if (op.kind == qk::TOP_PHASE) {
                    for (int th = 0; th < NT; ++th)
                        for (int kk = 0; kk < R; ++kk) {
                            const bool a = op.bits[0] != qk::kNoSlot ? (kk >> op.bits[0]) & 1 : t.bit(op.a, th);
                            const bool b = op.bits[1] != qk::kNoSlot ? (kk >> op.bits[1]) & 1 : t.bit(op.b, th);
                            if (a && b)
                                for (auto &x : t.v) x[th * R + kk] *= coef(0);
                        }
                } else if (op.kind == qk::TOP_SCALE) {
                    const cd f = op.b ? coef(0) : cd(coef(0).real());
                    for (auto &x : t.v)
                        for (cd &z : x) z *= f;
                } else if (op.kind == qk::TOP_GRAD) {
                    for (int w = 0; w < (op.b == 5 ? 2 : 1); ++w) {
                        const double a = coef(2 * w).real(), b = coef(2 * w).imag(), cz = coef(2 * w + 1).real();
                        const int slot = w ? (op.bits[2] | (op.bits[3] << 8)) : (op.bits[0] | (op.bits[1] << 8));
                        if (slot >= d.ngrad) std::exit(2);
                        const cd g00 = cz, g01 = cd(a, -b), g10 = cd(a, b), g11 = -cz;
                        double s = 0;
                        for (int th = 0; th < NT; ++th)
                            for (int kk = 0; kk < R; ++kk)
                                if (!((kk >> op.a) & 1)) {
                                    const int i0 = th * R + kk, i1 = i0 | (1 << op.a);
                                    const cd p0 = t.v[0][i0], p1 = t.v[0][i1], l0 = t.v[1][i0], l1 = t.v[1][i1];
                                    s += (std::conj(l0) * (g00 * p0 + g01 * p1) + std::conj(l1) * (g10 * p0 + g11 * p1)).imag();
                                }
                        g.at((size_t)hp.grad_params.at((size_t)(d.grad0 + slot))) += s;
                    }
                } else {
                    std::fprintf(stderr, "unknown step %d\n", op.kind);
                    std::exit(2);
                }
            }
            if (dirty) std::exit(2);   // stored under a clean mapping
            for (int i = 0; i < ns; ++i)
                for (int th = 0; th < NT; ++th)
                    for (int kk = 0; kk < R; ++kk) (*states[i])[addr(t.label(th, kk))] = t.v[i][th * R + kk];
        }
    }
}

// a random gate the factored planner takes; family 0: all kinds, 1: QFT-like
// (H, CP), 2: RY, RZ and CX, 3: U1 and CP(pi)
qk_gate gate(Gen &G, int family) {
    for (;;) {
        qk_gate g = G.gate();
        if (g.kind == QK_GATE_U2) {
            Op o = lower(g);
            if (o.kind == qk::OP_DENSE2) continue;
        }
        const int k = g.kind;
        const bool cx = k == QK_GATE_U2;
        if (family == 1 && k != QK_GATE_H && k != QK_GATE_CP) continue;
        if (family == 2 && k != QK_GATE_RY && k != QK_GATE_RZ && !cx) continue;
        if (family == 3 && k != QK_GATE_U1 && k != QK_GATE_CP) continue;
        if (family == 3 && k == QK_GATE_CP) g.param = M_PI;
        // (a U1 whose rounding leaves it less than a unitary is for the general planner)
        qk::PlanOptions o{QK_C128, 3, 2};
        o.f_tile_bits = 3;
        o.f_reg_bits = 2;
        if (!qk::plan_is_factored(&g, 1, G.n, o, 2)) continue;
        return g;
    }
}

bool rotation(const qk_gate &g) { return g.kind == QK_GATE_RX || g.kind == QK_GATE_RY || g.kind == QK_GATE_RZ; }

}  // namespace

int main() {
    int bad = 0, plans = 0;
    for (int seed = 0; seed < 120; ++seed) {
        const int family = seed % 4;
        const bool with_h = seed % 3 == 0 || family == 1;
        Gen G{std::mt19937_64(500 + seed), 5 + seed % 4, with_h};
        const int n = G.n, T = std::min(n, 3 + (seed / 2) % 4), dtype = (seed / 4) % 2 ? QK_C128 : QK_C64;
        const int r = std::max(2, 1 + (seed / 5) % std::min(dtype == QK_C64 ? 5 : 4, T));
        qk::PlanOptions o{dtype, T, 2};
        o.f_tile_bits = T;
        o.f_reg_bits = r;
        std::vector<qk_gate> gates;
        for (int i = 0; i < 90; ++i) {
            if (i % 31 == 7 && family == 0) {
                qk_gate v;
                std::memset(&v, 0, sizeof v);
                const Op p = G.vswap();
                v.kind = QK_GATE_VSWAP;
                v.nq = 4;
                for (int k = 0; k < 4; ++k) v.q[k] = p.q[k];
                gates.push_back(v);
            } else {
                gates.push_back(gate(G, family));
            }
        }
        if (!qk::plan_is_factored(gates.data(), gates.size(), n, o, 1)) {
            std::printf("seed %d: not factored\n", seed);
            ++bad;
            continue;
        }
        const State init = G.state();
        State ref = init;
        std::vector<double> none(1, 0);
        for (const qk_gate &g : gates) {
            std::vector<int> qs;
            const auto m = matrix_of(lower(g), qs);
            apply_matrix(ref, n, qs, m);
        }
        HostPlan hp;
        if (qk::plan_forward(gates.data(), gates.size(), n, o, hp)) {
            std::printf("seed %d: plan_forward failed: %s\n", seed, qk_last_error());
            ++bad;
            continue;
        }
        ++plans;
        State got = init;
        emulate(hp, got, nullptr, none);
        const bool c64 = o.dtype == QK_C64;
        if (max_diff(ref, got) > (c64 ? 1.1e-5 : 1e-12)) {
            std::printf("forward seed %d (n %d, T %d, r %d): max |d amp| %.3g, %zu passes\n", seed, n, T, r,
                        max_diff(ref, got), hp.passes.size());
            ++bad;
        }
        // adjoint: trainable rotations, some sharing a parameter
        std::vector<qk_gate> circ;
        std::vector<int32_t> pidx;
        int np = 0;
        for (int i = 0; i < 70; ++i) {
            const qk_gate g = gate(G, family);
            circ.push_back(g);
            pidx.push_back(rotation(g) ? (np > 2 && G.rng() % 4 == 0 ? (int)(G.rng() % np) : np++) : -1);
        }
        o.dtype = QK_C128;   // two-state programs: complex128, up to three register bits
        o.f_reg_bits = std::min(r, 3);
        HostPlan ap;
        if (qk::plan_adjoint(circ.data(), circ.size(), pidx.data(), n, o, ap)) {
            std::printf("seed %d: plan_adjoint failed: %s\n", seed, qk_last_error());
            ++bad;
            continue;
        }
        ++plans;
        std::vector<Op> back;
        for (size_t i = circ.size(); i-- > 0;) {
            Op op = lower(circ[i]);
            if (pidx[i] >= 0) {
                Op gr;
                std::memset(&gr, 0, sizeof gr);
                gr.kind = qk::OP_GRAD;
                gr.nq = 1;
                gr.q[0] = op.q[0];
                gr.m[0] = circ[i].kind == QK_GATE_RX ? 1 : circ[i].kind == QK_GATE_RY ? 2 : 3;
                gr.aux = pidx[i];
                back.push_back(gr);
            }
            qk::invert_op(op);
            back.push_back(op);
        }
        State psi = G.state(), lam = G.state(), psi2 = psi, lam2 = lam;
        std::vector<double> g0(np + 1, 0), g1(np + 1, 0);
        run(back, n, psi, lam, g0);
        emulate(ap, psi2, &lam2, g1);
        double dg = 0;
        for (int k = 0; k <= np; ++k) dg = std::max(dg, std::fabs(g0[k] - g1[k]));
        const double ds = std::max(max_diff(psi, psi2), max_diff(lam, lam2));
        if (dg > (with_h ? 1e-9 : 1e-12) || ds > 1e-12) {
            std::printf("adjoint seed %d (n %d, T %d): max |d grad| %.3g, max |d amp| %.3g, %zu passes\n", seed, n, T, dg,
                        ds, ap.passes.size());
            ++bad;
        }
    }
    std::printf("%d plans, %s\n", plans, bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
