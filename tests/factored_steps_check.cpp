// CPU check of factored programs (subquokka_dev_b200/csrc/qk_factor.cpp) as
// the engine plans them, in the arithmetic of the state's type.
//
// An emulator of the steps, written from their definitions in qk_internal.h,
// with every amplitude named by its label: the amplitudes of a tile are kept
// with the labels (tile indices) their thread and register element carry.
// It runs in double for complex128 plans and in float for complex64 ones (or
// in double, to see the coefficients' rounding alone).
// - X, Y, CX, SWAP and VSWAP circuits: amplitudes are moved and multiplied by
//   powers of i, so every result is exact;
// - random circuits against the dense simulation: complex128 within 1e-13
//   in the 2-norm of a normalised state (90 gates x 4 roundings of 2^-53 are
//   4e-14); complex64 coefficients within 1e-6 (180 coefficients, each 2.4e-8
//   rms in the 2-norm at most, independent: 3.3e-7, three times that), in
//   float arithmetic within 90 x 4 x 2^-24 = 2.2e-5;
// - states of amplitude 1e30 (complex64) and 1e290: finite and as accurate;
// - every tangent at most 2^10, every real scale a power of two other than 1;
// - brick circuits (U3 and CZ) in complex128 against the simulation in long
//   double: 200 unitaries of four roundings (4.6e-17 rms) and two rounded
//   coefficients (2.9e-17 rms) each, independent, are 1.42e-15;
// - adjoint plans against the direct backward sweep, within 1e-12, gradients
//   of circuits with H (whose constant is 1.1e-11 off a unitary's) 1e-9.
#include "dense_sim.h"

using namespace dense_sim;
using qk::HostPlan;
using qk::PassDesc;
using qk::TOp;

namespace {

template <typename T> using Z = std::complex<T>;
template <typename T> Z<T> times(Z<T> f, Z<T> y) {
    return {std::fma(f.real(), y.real(), -f.imag() * y.imag()), std::fma(f.real(), y.imag(), f.imag() * y.real())};
}
template <typename T> Z<T> axpy(T s, Z<T> a, Z<T> c) {
    return {std::fma(s, a.real(), c.real()), std::fma(s, a.imag(), c.imag())};
}
template <typename T> Z<T> madd(Z<T> f, Z<T> a, Z<T> c) {   // c + f a
    return {std::fma(f.real(), a.real(), std::fma(-f.imag(), a.imag(), c.real())),
            std::fma(f.real(), a.imag(), std::fma(f.imag(), a.real(), c.imag()))};
}

void die(const char *what) {
    std::fprintf(stderr, "%s\n", what);
    std::exit(2);
}

// the state(s) of a plan run step by step
template <typename T> struct Emulator {
    const HostPlan &hp;
    std::vector<Z<T>> *st[2];
    std::vector<double> *g;
    int ns, n, r;

    // a tile under way: amplitude e = thread * 2^r + element, its label lab[e]
    std::vector<uint32_t> lab;
    std::vector<Z<T>> v[2];

    static bool in(int e, int s) { return (e >> s) & 1; }
    void map_to(const PassDesc &d, const TOp &op) {
        const uint32_t N = 1u << d.T;
        lab.assign(N, 0);
        std::vector<int> rest;
        for (int b = 0; b < d.T; ++b)
            if (std::find(op.bits, op.bits + r, b) == op.bits + r) rest.push_back(b);
        for (uint32_t e = 0; e < N; ++e) {
            for (int s = 0; s < r; ++s) lab[e] |= (uint32_t)in(e, s) << op.bits[s];
            for (size_t k = 0; k < rest.size(); ++k) lab[e] |= (uint32_t)in(e >> r, k) << rest[k];
        }
    }
    // a condition: the same for all of a thread's amplitudes
    bool cond(uint8_t code, uint32_t e, uint64_t base) const {
        if (code == qk::kNoQubit) return true;
        if (code & qk::kOuterFlag) return (base >> (code & 0x3F)) & 1;
        const uint32_t t0 = e >> r << r;
        for (uint32_t k = t0; k < t0 + (1u << r); ++k)
            if (((lab[k] ^ lab[e]) >> code) & 1) die("a condition on a register slot");
        return (lab[e] >> code) & 1;
    }
    void phase(uint32_t e, Z<T> f) {
        for (int i = 0; i < ns; ++i) v[i][e] = times(f, v[i][e]);
    }

    void tile(const PassDesc &d, uint32_t o) {
        uint64_t base = 0;
        std::vector<char> inside(n, 0);
        for (int k = 0; k < d.T; ++k) inside[d.bpos[k]] = 1;
        for (int q = 0, k = 0; q < n; ++q)
            if (!inside[q]) base |= (uint64_t)((o >> k++) & 1) << q;
        auto at = [&](uint32_t label) {
            uint64_t a = base;
            for (int k = 0; k < d.T; ++k) a |= (uint64_t)((label >> k) & 1) << d.bpos[k];
            return a;
        };
        const TOp *prog = hp.ops.data() + d.prog0;
        const uint32_t N = 1u << d.T;
        map_to(d, prog[0]);
        for (int i = 0; i < ns; ++i) {
            v[i].resize(N);
            for (uint32_t e = 0; e < N; ++e) v[i][e] = (*st[i])[at(lab[e])];
        }
        std::vector<Z<T>> pend(N, 1);   // (one a thread; kept an element)
        bool dirty = false;
        for (int p = 2; p < d.nprog; ++p) {
            const TOp &op = prog[p];
            auto coef = [&](uint32_t k) {
                if (op.coef + k >= (uint32_t)d.ncoef) die("a coefficient past the pass's");
                const size_t i = 2 * ((size_t)d.coef0 + op.coef + k);
                return Z<T>((T)hp.coef[i], (T)hp.coef[i + 1]);
            };
            switch (op.kind) {
            case qk::TOP_REMAP: {
                if ((op.b != 0) != dirty) die("a re-mapping that does not know of the label steps before it");
                dirty = false;
                std::vector<uint32_t> where(N);
                for (uint32_t e = 0; e < N; ++e) where[lab[e]] = e;
                map_to(d, op);
                for (int i = 0; i < ns; ++i) {
                    const auto old = v[i];
                    for (uint32_t e = 0; e < N; ++e) v[i][e] = old[where[lab[e]]];
                }
                ++p;
                break;
            }
            case qk::TOP_LCX:
                dirty = true;
                for (uint32_t e = 0; e < N; ++e)
                    lab[e] ^= (uint32_t)((op.b & qk::kOuterFlag) ? cond(op.b, e, base) : (lab[e] >> op.b) & 1) << op.a;
                break;
            case qk::TOP_LAM:
                for (uint32_t e = 0; e < N; ++e) {
                    int idx = 0;
                    for (int i = 0; i < op.nbits; ++i) {
                        const uint8_t c = op.bits[i];
                        idx |= (int)((c & qk::kOuterFlag) ? (o >> (c & 31)) & 1 : cond(c, e, base)) << i;
                    }
                    pend[e] = times(pend[e], coef(idx & 15));
                    if (op.nbits > 4) pend[e] = times(pend[e], coef(16 + (idx >> 4)));
                }
                break;
            case qk::TOP_PHASE:
                for (uint32_t e = 0; e < N; ++e)
                    if ((op.bits[0] != qk::kNoSlot ? in(e, op.bits[0]) : cond(op.a, e, base)) &&
                        (op.bits[1] != qk::kNoSlot ? in(e, op.bits[1]) : cond(op.b, e, base)))
                        phase(e, coef(0));
                break;
            case qk::TOP_SCALE: {
                const Z<T> f = coef(0);
                int x;
                if (!op.b && (std::frexp(f.real(), &x) != 0.5 || f.real() == 1)) die("a scale that is 1 or no power of two");
                for (uint32_t e = 0; e < N; ++e)
                    for (int i = 0; i < ns; ++i) v[i][e] = op.b ? times(f, v[i][e]) : v[i][e] * f.real();
                break;
            }
            case qk::TOP_LAYER: p += layer(op, prog + p + 1, coef, o, pend); break;
            case qk::TOP_GRAD: grad(d, op, coef); break;
            default: {
                if (op.kind < qk::TOP_PH2 || op.kind >= qk::TOP_PH2 + 10) die("an unknown step");
                int a = 0, b = 1;
                while (qk::slot_pair(a, b) != op.kind - qk::TOP_PH2)
                    if (++a == b) a = 0, ++b;
                for (uint32_t e = 0; e < N; ++e)
                    if (in(e, a) && in(e, b)) phase(e, coef(0));
            }
            }
        }
        if (dirty) die("stored under changed labels");
        for (int i = 0; i < ns; ++i)
            for (uint32_t e = 0; e < N; ++e) (*st[i])[at(lab[e])] = v[i][e];
    }

    template <typename F> int layer(const TOp &op, const TOp *words, F &&coef, uint32_t o, std::vector<Z<T>> &pend) {
        uint32_t u[5] = {0};
        uint16_t w[5] = {0};
        const bool has = op.b & qk::kLayerWords;
        if (has) {
            std::memcpy(u, words, 20);
            std::memcpy(w, (const char *)words + 20, 10);
        }
        const uint32_t N = (uint32_t)lab.size();
        const int signs = (op.b & qk::kLayerSigns) ? op.bits[0] | op.bits[1] << 8 : 0;
        for (int y = 1; y < r; ++y)
            for (int x = 0; x < y; ++x)
                if ((signs >> qk::slot_pair(x, y)) & 1)
                    for (uint32_t e = 0; e < N; ++e)
                        if (in(e, x) && in(e, y))
                            for (int i = 0; i < ns; ++i) v[i][e] = -v[i][e];
        uint32_t c = 0;
        for (int s = 0; s < r; ++s) {
            if (!in(op.a, s)) continue;
            const Z<T> first = coef(c++), second = coef(c++);
            for (uint32_t e = 0; e < N; ++e) {
                if (in(e, s)) continue;
                const uint32_t e1 = e | 1u << s;
                bool neg = __builtin_parity(o & u[s]);
                for (int b = 0; b < 16; ++b)
                    if ((w[s] >> b) & 1) neg ^= cond((uint8_t)b, e, 0);
                for (int i = 0; i < ns; ++i) pair(op, first, second, neg, pend[e], v[i][e], v[i][e1]);
            }
            if (op.b & qk::kLayerPending) std::fill(pend.begin(), pend.end(), Z<T>(1));
        }
        return has ? 2 : 0;
    }
    void pair(const TOp &op, Z<T> first, Z<T> second, bool neg, Z<T> pend, Z<T> &x, Z<T> &y) {
        if (op.b & qk::kLayerFull) {
            if (op.b & qk::kLayerPending) die("a full unitary with a pending factor");
            if (neg) y = -y;
            const Z<T> x0 = x;
            x = madd(first, y, x0);
            y = madd(second, x0, y);
            return;
        }
        const T t = first.real();
        if (!(std::fabs(t) <= 1024 * (1 + 1e-6))) die("a tangent above 2^10");
        Z<T> l = (op.b & qk::kLayerPending) ? pend : second;
        if (neg) l = -l;
        const Z<T> z = times(l, y), x0 = x;
        x = axpy(-t, z, x0);
        y = axpy(t, x0, z);
    }
    template <typename F> void grad(const PassDesc &d, const TOp &op, F &&coef) {
        for (int k = 0; k < (op.b == 5 ? 2 : 1); ++k) {
            const double a = coef(2 * k).real(), b = coef(2 * k).imag(), c = coef(2 * k + 1).real();
            const int slot = op.bits[2 * k] | op.bits[2 * k + 1] << 8;
            if (slot >= d.ngrad) die("a gradient slot past the pass's");
            double s = 0;
            for (uint32_t e = 0; e < lab.size(); ++e) {
                if (in(e, op.a)) continue;
                const uint32_t e1 = e | 1u << op.a;
                const cd p0(v[0][e]), p1(v[0][e1]), l0(v[1][e]), l1(v[1][e1]);
                s += (std::conj(l0) * (c * p0 + cd(a, -b) * p1) + std::conj(l1) * (cd(a, b) * p0 - c * p1)).imag();
            }
            g->at((size_t)hp.grad_params.at((size_t)(d.grad0 + slot))) += s;
        }
    }

    void run() {
        for (const PassDesc &d : hp.passes) {
            if (!d.perm) {
                if (d.form != 1) die("a general program");
                for (uint32_t o = 0; o < 1u << (n - d.T); ++o) tile(d, o);
                continue;
            }
            for (int i = 0; i < ns; ++i) {
                const auto old = *st[i];
                for (uint64_t j = 0; j < old.size(); ++j) {
                    uint64_t to = j;
                    for (int k = 0; k < d.nperm; ++k) {
                        const int a = d.perm == 2 ? d.perm_a[k] : d.bpos[d.perm_a[k]];
                        const int b = d.perm == 2 ? d.perm_b[k] : d.bpos[d.perm_b[k]];
                        if (((j >> a) ^ (j >> b)) & 1) to ^= 1ull << a | 1ull << b;
                    }
                    (*st[i])[to] = old[j];
                }
            }
        }
    }
};

template <typename T> State emulate(const HostPlan &hp, const State &in, State *lam = nullptr, std::vector<double> *g = nullptr) {
    std::vector<Z<T>> a(in.begin(), in.end()), b;
    if (lam) b.assign(lam->begin(), lam->end());
    Emulator<T> e{hp, {&a, &b}, g, lam ? 2 : 1, hp.n, hp.r, {}, {}};
    e.run();
    if (lam) lam->assign(b.begin(), b.end());
    return State(a.begin(), a.end());
}

double norm2(const State &a) {
    long double s = 0;
    for (const cd &x : a) s += std::norm(std::complex<long double>(x));
    return (double)std::sqrt(s);
}
double dist(State a, const State &b) {
    for (size_t i = 0; i < a.size(); ++i) a[i] -= b[i];
    return norm2(a);
}

// a random gate of the factored set; family 0 all kinds, 1 X Y CX SWAP VSWAP,
// 2 rotations by and near pi among all kinds
qk_gate gate(Gen &G, int family, bool vswap) {
    for (;;) {
        qk_gate g = G.gate();
        if (vswap && G.rng() % 12 == 0) {
            const Op p = G.vswap();
            g.kind = QK_GATE_VSWAP;
            g.nq = 4;
            for (int k = 0; k < 4; ++k) g.q[k] = p.q[k];
            return g;
        }
        const bool cx = g.kind == QK_GATE_U2 && lower(g).kind != qk::OP_DENSE2;
        if (g.kind == QK_GATE_U2 && !cx) continue;
        if (family == 1 && g.kind != QK_GATE_X && g.kind != QK_GATE_Y && !cx && g.kind != QK_GATE_SWAP) continue;
        if (family == 2 && (g.kind == QK_GATE_RX || g.kind == QK_GATE_RY))
            g.param = M_PI + (G.rng() % 3 ? 0 : std::ldexp(G.u(), -(int)(G.rng() % 40)));
        qk::PlanOptions o = qk::factored_plan_options(QK_C128, G.n);
        if (g.kind == QK_GATE_U1 && !qk::plan_is_factored(&g, 1, G.n, o, 1)) continue;   // (rounded off a unitary)
        return g;
    }
}

// rms 2-norm error of 20-layer brick circuits on 10 qubits
double brick_error() {
    const int n = 10, circuits = 8;
    using cl = std::complex<long double>;
    long double sum = 0;
    for (int seed = 0; seed < circuits; ++seed) {
        Gen G{std::mt19937_64(40 + seed), n, false};
        std::uniform_real_distribution<double> angle(0, 2 * M_PI);
        std::vector<qk_gate> gates;
        qk_gate g;
        for (int layer = 0; layer < 20; ++layer) {
            for (int q = 0; q < n; ++q) {
                std::memset(&g, 0, sizeof g);
                g.kind = QK_GATE_U1;
                g.nq = 1;
                g.q[0] = q;
                const double th = angle(G.rng), ph = angle(G.rng), la = angle(G.rng);
                const cd m[4] = {std::cos(th / 2), -std::polar(1.0, la) * std::sin(th / 2),
                                 std::polar(1.0, ph) * std::sin(th / 2), std::polar(1.0, ph + la) * std::cos(th / 2)};
                std::memcpy(g.coeff, m, sizeof m);
                gates.push_back(g);
            }
            for (int q = layer % 2; q + 1 < n; q += 2) {
                std::memset(&g, 0, sizeof g);
                g.kind = QK_GATE_CP;
                g.nq = 2;
                g.q[0] = q;
                g.q[1] = q + 1;
                g.param = M_PI;
                gates.push_back(g);
            }
        }
        const State init = G.state();
        std::vector<cl> ref(init.begin(), init.end());
        for (const qk_gate &x : gates) {
            const Op op = lower(x);
            const size_t h = (size_t)1 << op.q[0], both = h | (op.nq > 1 ? (size_t)1 << op.q[1] : 0);
            for (size_t i = 0; i < ref.size(); ++i)
                if (op.nq > 1) {
                    if ((i & both) == both) ref[i] *= cl(c(op.m, 0));
                } else if (!(i & h)) {
                    const cl a = ref[i], b = ref[i | h];
                    ref[i] = cl(c(op.m, 0)) * a + cl(c(op.m, 1)) * b;
                    ref[i | h] = cl(c(op.m, 2)) * a + cl(c(op.m, 3)) * b;
                }
        }
        HostPlan hp;
        if (qk::plan_forward(gates.data(), gates.size(), n, qk::factored_plan_options(QK_C128, n), hp)) return 1;
        const State got = emulate<double>(hp, init);
        for (size_t i = 0; i < got.size(); ++i) sum += std::norm(cl(got[i]) - ref[i]);
    }
    return (double)std::sqrt(sum / circuits);
}

}  // namespace

int main() {
    int bad = 0, plans = 0;
    const double brick = brick_error();
    if (!(brick <= 1.42e-15)) {
        std::printf("brick circuits: %.3g\n", brick);
        ++bad;
    }
    double worst[4] = {0, 0, 0, 0};
    for (int seed = 0; seed < 150; ++seed) {
        const int family = seed % 3;
        const bool with_h = seed % 2;
        const bool little = seed % 5 == 4;   // a few gates on two or three qubits
        Gen G{std::mt19937_64(9000 + seed), little ? 2 + seed % 2 : 4 + seed % 6, with_h};
        const int n = G.n, count = little ? 1 + seed / 5 % 8 : 90;
        for (int dtype : {QK_C128, QK_C64}) {
            qk::PlanOptions o = qk::factored_plan_options(dtype, n);
            o.f_tile_bits = std::min(n, 3 + (seed / 2) % 6);
            o.f_reg_bits = std::max(std::min(2, n), std::min(o.f_tile_bits, 1 + (seed / 5) % (dtype == QK_C64 ? 5 : 4)));
            o.tile_bits = o.f_tile_bits;
            o.reg_bits = std::min(4, o.f_reg_bits);
            std::vector<qk_gate> gates;
            for (int i = 0; i < count; ++i) gates.push_back(gate(G, family, n >= 8));
            State init = G.state();
            if (family == 1 && seed % 2) {
                init.assign(init.size(), 0);
                init[G.rng() % init.size()] = 1;
            }
            if (dtype == QK_C64)
                for (cd &x : init) x = cd((float)x.real(), (float)x.imag());
            State ref = init;
            for (const qk_gate &g : gates) {
                std::vector<int> qs;
                const auto m = matrix_of(lower(g), qs);
                apply_matrix(ref, n, qs, m);
            }
            HostPlan hp;
            if (qk::plan_forward(gates.data(), gates.size(), n, o, hp)) {
                std::printf("seed %d: %s\n", seed, qk_last_error());
                ++bad;
                continue;
            }
            ++plans;
            const bool c64 = dtype == QK_C64;
            const State got = c64 ? emulate<float>(hp, init) : emulate<double>(hp, init);
            if (family == 1) {
                for (size_t i = 0; i < ref.size(); ++i)
                    if (got[i] != ref[i]) {
                        std::printf("seed %d dtype %d: amplitude %zu (%g, %g), not (%g, %g)\n", seed, dtype, i, got[i].real(),
                                    got[i].imag(), ref[i].real(), ref[i].imag());
                        ++bad;
                        break;
                    }
            }
            const double e = dist(got, ref), scale = c64 ? 1e30 : 1e290;
            worst[c64] = std::max(worst[c64], e);
            State big = init, bref = ref;
            for (cd &x : big) x *= scale;
            for (cd &x : bref) x *= scale;
            State bgot = c64 ? emulate<float>(hp, big) : emulate<double>(hp, big);
            for (size_t i = 0; i < bgot.size(); ++i) bgot[i] /= scale, bref[i] /= scale;
            const double eb = dist(bgot, bref), ec = c64 ? dist(emulate<double>(hp, init), ref) : 0;
            worst[2] = std::max(worst[2], ec);
            const double tol = c64 ? 2.2e-5 : 1e-13;
            if (!(e <= tol) || !(eb <= tol) || !(ec <= 1e-6)) {
                std::printf("seed %d dtype %d family %d (n %d T %d r %d): %.3g, large %.3g, coefficients %.3g\n", seed, dtype,
                            family, n, hp.T, hp.r, e, eb, ec);
                ++bad;
            }
        }
        // adjoint
        std::vector<qk_gate> circ;
        std::vector<int32_t> pidx;
        int np = 0;
        for (int i = 0; i < 70; ++i) {
            circ.push_back(gate(G, family, false));
            const int k = circ.back().kind;
            pidx.push_back(k == QK_GATE_RX || k == QK_GATE_RY || k == QK_GATE_RZ ? np++ : -1);
        }
        qk::PlanOptions o = qk::factored_adjoint_options(QK_C128, n);
        o.tile_bits = o.f_tile_bits = std::min(n, 3 + (seed / 2) % 5);
        o.reg_bits = o.f_reg_bits = std::min(3, std::max(2, o.f_tile_bits - 2));
        HostPlan ap;
        if (qk::plan_adjoint(circ.data(), circ.size(), pidx.data(), n, o, ap)) {
            std::printf("seed %d: %s\n", seed, qk_last_error());
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
        State psi = G.state(), lam = G.state(), lam2 = lam;
        std::vector<double> g0(np + 1, 0), g1(np + 1, 0);
        const State psi2 = emulate<double>(ap, psi, &lam2, &g1);
        run(back, n, psi, lam, g0);
        double dg = 0;
        for (int k = 0; k <= np; ++k) dg = std::max(dg, std::fabs(g0[k] - g1[k]));
        const double ds = std::max(dist(psi, psi2), dist(lam, lam2));
        worst[3] = std::max(worst[3], dg);
        if (!(dg <= (with_h ? 1e-9 : 1e-12)) || !(ds <= 1e-12)) {
            std::printf("adjoint seed %d: gradient %.3g, states %.3g\n", seed, dg, ds);
            ++bad;
        }
    }
    std::printf("errors: complex128 %.3g, complex64 %.3g (coefficients %.3g), gradients %.3g\n", worst[0], worst[1], worst[2],
                worst[3]);
    std::printf("%d plans, %s\n", plans, bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
