// Device building blocks of factored passes (k_fpass in qk_fpass.cu): the
// thread's part of a tile and the step interpreter.  The steps are defined in
// qk_internal.h, made by qk_factor.cpp.
//
// A thread's amplitudes are named by labels (tile indices): register element
// kk of thread tid carries label tb ^ XOR of bm[s] over the set bits s of kk.
// A re-mapping writes the registers to the exchange buffer at their labels
// and reads those of the next mapping; the label steps of CX, SWAP and X
// gates only change tb and bm.  Under the first mapping each thread loads its
// amplitudes from HBM, under the last it stores them there: both leave the
// lowest state bits to the lanes, so the accesses are the tile's contiguous
// runs and neither goes through the exchange buffer.
#pragma once

#include "qk_pass_device.cuh"

namespace qk {

// Addresses of a thread's register elements: the state at p, slot s the
// state bit pos[s].
template <int LOG2R, typename C>
__device__ __forceinline__ void slot_addresses(C *p, const int32_t (&pos)[kPassMaxReg], C *(&a)[1 << LOG2R]) {
    a[0] = p;
#pragma unroll
    for (int s = 0; s < LOG2R; ++s)
#pragma unroll
        for (int k = 0; k < (1 << s); ++k) a[k | (1 << s)] = a[k] + (1ull << pos[s]);
}

// a * s + c, both components (complex64: one packed instruction, the same
// roundings as two).
__device__ __forceinline__ double2 axpy(double s, double2 a, double2 c) {
    return make_double2(fma(s, a.x, c.x), fma(s, a.y, c.y));
}
__device__ __forceinline__ float2 axpy(float s, float2 a, float2 c) {
    union U { float2 f; unsigned long long u; } A, Cc, S, D;
    A.f = a;
    Cc.f = c;
    S.f = make_float2(s, s);
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(D.u) : "l"(S.u), "l"(A.u), "l"(Cc.u));
    return D.f;
}

// Amplitudes of slot S's upper half times l.
template <int S, typename C, int R>
__device__ __forceinline__ void k_phase(C (&v)[R], const C l) {
    if constexpr ((1 << S) < R) {
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (k & (1 << S)) {
                const C y = v[k];
                v[k].x = fma(l.x, y.x, -l.y * y.y);
                v[k].y = fma(l.x, y.y, l.y * y.x);
            }
    }
}
// A factored unitary on slot S: the upper half times l, then the rotation.
// In one piece, so that the product l y lives in temporaries and both results
// are written in place: with the two apart, every component took a register
// move besides its multiply-adds.
template <int S, typename C, int R, typename T>
__device__ __forceinline__ void k_unitary(C (&v)[R], const C l, const T t) {
    if constexpr ((1 << S) < R) {
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (!(k & (1 << S))) {
                const C y = v[k | (1 << S)];
                C z;
                z.x = fma(l.x, y.x, -l.y * y.y);
                z.y = fma(l.x, y.y, l.y * y.x);
                v[k | (1 << S)] = axpy(t, v[k], z);
                v[k] = axpy(-t, z, v[k]);
            }
    }
}

// The sign bit of x flipped where s is odd.
__device__ __forceinline__ double flip_sign(double x, uint32_t s) {
    return __hiloint2double(__double2hiint(x) ^ (int)(s << 31), __double2loint(x));
}
__device__ __forceinline__ float flip_sign(float x, uint32_t s) {
    return __uint_as_float(__float_as_uint(x) ^ (s << 31));
}

// c + f a.
template <typename C> __device__ __forceinline__ C madd(const C f, const C a, const C c) {
    C r;
    r.x = fma(f.x, a.x, fma(-f.y, a.y, c.x));
    r.y = fma(f.x, a.y, fma(f.y, a.x, c.y));
    return r;
}
// A full unitary on slot S, without its left phase: x' = x + B y, y' = F x + y.  As many multiply-adds as k_unitary,
// but neither result can be written in place.
template <int S, typename C, int R>
__device__ __forceinline__ void k_full(C (&v)[R], const C B, const C F) {
    if constexpr ((1 << S) < R) {
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (!(k & (1 << S))) {
                const C x = v[k];
                v[k] = madd(B, v[k | (1 << S)], x);
                v[k | (1 << S)] = madd(F, x, v[k | (1 << S)]);
            }
    }
}
template <int S, typename C, int R> __device__ __forceinline__ void k_negate(C (&v)[R]) {
    if constexpr ((1 << S) < R) {
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (k & (1 << S)) {
                v[k].x = flip_sign(v[k].x, 1);
                v[k].y = flip_sign(v[k].y, 1);
            }
    }
}

// Value of a condition code that is the same for all of the thread's
// amplitudes.
__device__ __forceinline__ bool code_bit(uint32_t code, uint64_t base, uint32_t tb) {
    if (code == kNoQubit) return true;
    return (code & kOuterFlag) ? (base >> (code & 0x3F)) & 1 : (tb >> (code & 0x3F)) & 1;
}

// Byte offset of register element kk under slot offsets sb.
template <int LOG2R>
__device__ __forceinline__ uint32_t slot_place(int kk, uint32_t stb, const uint32_t (&sb)[LOG2R]) {
    uint32_t x = stb;
#pragma unroll
    for (int s = 0; s < LOG2R; ++s)
        if ((kk >> s) & 1) x ^= sb[s];
    return x;
}

// Steps prog[2..nprog) on the thread's amplitudes, loaded under prog[0..1].
// xb: the exchange buffer, psi's 2^T amplitudes and then (NS = 2) lambda's;
// base / tile: the tile's state offset and number.  NS = 2: psi in v, lambda
// in w; gradient sums go to the thread's own accumulators gsm[slot * threads
// + tid], in double.
template <typename C, int R, int NS>
__device__ __forceinline__ void run_steps(C (&v)[R], C (&w)[NS == 2 ? R : 1], unsigned char *xb, uint32_t xbytes,
                                          uint64_t base, uint32_t tile, const TOp *prog, int nprog, const C *coef,
                                          double *gsm) {
    constexpr int LOG2R = R == 2 ? 1 : R == 4 ? 2 : R == 8 ? 3 : R == 16 ? 4 : 5;
    using T = decltype(v[0].x);
    const uint32_t tid = threadIdx.x;
    const uint4 *steps = reinterpret_cast<const uint4 *>(prog);
    uint32_t tb, stb;                  // thread label, its place in the exchange buffer
    uint32_t sb[LOG2R];                // places of the slots' tile bits
    uint32_t slots, slot5;             // the slots' tile bits (bytes); until a label step changes them,
    uint32_t bm[LOG2R];                // the slots' labels
    auto map_to = [&](const uint4 &op, const uint4 &places) {
        slots = op.y;
        slot5 = op.z;
        tb = slot_deposit<LOG2R>(tid, slots, slot5);
        stb = swz<C>(tb) * (uint32_t)sizeof(C);
#pragma unroll
        for (int s = 0; s < LOG2R; ++s)
            sb[s] = ((s < 2 ? places.x : s < 4 ? places.y : places.z) >> (16 * (s & 1))) & 0xFFFF;
    };
    map_to(steps[0], steps[1]);
    bool labels = false;               // a label step has run since the last re-mapping
    C lam;                             // pending factor (TOP_LAM)
    lam.x = 1;
    lam.y = 0;
    // The next step, and in a layer the next unitary's coefficients, are read
    // ahead of the current one's arithmetic (past the end at the last: the
    // buffer has room).
    uint4 next = steps[2];
    for (int p = 2; p < nprog;) {
        const uint4 op = next;
        const uint32_t kind = op.x & 0xFF, a = (op.x >> 8) & 0xFF, b = (op.x >> 16) & 0xFF, nb = op.x >> 24;
        const C *m = coef + op.w;
        const uint4 *words = steps + p + 1;
        p += 1 + (kind == TOP_REMAP || kind == TOP_LAYER ? nb : 0);
        next = steps[p];
        switch (kind) {
        case TOP_REMAP: {
            if (labels) {
                labels = false;
                stb = swz<C>(tb) * (uint32_t)sizeof(C);
#pragma unroll
                for (int s = 0; s < LOG2R; ++s) sb[s] = swz<C>(bm[s]) * (uint32_t)sizeof(C);
                // changed labels are places other threads may still have to read
                __syncthreads();
            }
#pragma unroll
            for (int kk = 0; kk < R; ++kk) {
                unsigned char *x = xb + slot_place<LOG2R>(kk, stb, sb);
                *reinterpret_cast<C *>(x) = v[kk];
                if constexpr (NS == 2) *reinterpret_cast<C *>(x + xbytes) = w[kk];
            }
            map_to(op, words[0]);
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < R; ++kk) {
                const unsigned char *x = xb + slot_place<LOG2R>(kk, stb, sb);
                v[kk] = *reinterpret_cast<const C *>(x);
                if constexpr (NS == 2) w[kk] = *reinterpret_cast<const C *>(x + xbytes);
            }
            break;
        }
        case TOP_LAYER: {
            uint32_t neg = 0;   // bit S: slot S's factor changes sign
            if (b & kLayerWords) {
                const uint4 u03 = words[0], uw = words[1];   // u[0..3]; u[4] and w[0..4]
#define QK_W(S, U, W)                                                                 \
    if constexpr ((1 << S) < R)                                                       \
        neg |= ((uint32_t)__popc((tb & ((W) & 0xFFFF)) ^ (tile & (U))) & 1u) << S;
                QK_W(0, u03.x, uw.y) QK_W(1, u03.y, uw.y >> 16) QK_W(2, u03.z, uw.z) QK_W(3, u03.w, uw.z >> 16)
                QK_W(4, uw.x, uw.w)
#undef QK_W
            }
            T t = m[0].x;
            C l = m[1];
            if (b & kLayerSigns) {
#define QK_SG(X, Y)                                                              \
    if constexpr ((1 << Y) < R)                                                  \
        if ((op.y >> slot_pair(X, Y)) & 1) {                                       \
            _Pragma("unroll") for (int k = 0; k < R; ++k)                        \
                if ((k & (1 << X)) && (k & (1 << Y))) {                          \
                    v[k].x = flip_sign(v[k].x, 1);                               \
                    v[k].y = flip_sign(v[k].y, 1);                               \
                    if constexpr (NS == 2) {                                     \
                        w[k].x = flip_sign(w[k].x, 1);                           \
                        w[k].y = flip_sign(w[k].y, 1);                           \
                    }                                                            \
                }                                                                \
        }
                QK_SG(0, 1) QK_SG(0, 2) QK_SG(1, 2) QK_SG(0, 3) QK_SG(1, 3) QK_SG(2, 3)
                QK_SG(0, 4) QK_SG(1, 4) QK_SG(2, 4) QK_SG(3, 4)
#undef QK_SG
            }
            if constexpr (sizeof(C) == sizeof(double2))   // (complex64 programs have none)
                if (b & kLayerFull) {
#define QK_F(S)                                                     \
    if constexpr ((1 << S) < R)                                     \
        if ((a >> S) & 1) {                                         \
            if ((neg >> S) & 1) {                                   \
                k_negate<S>(v);                                     \
                if constexpr (NS == 2) k_negate<S>(w);              \
            }                                                       \
            k_full<S>(v, m[0], m[1]);                               \
            if constexpr (NS == 2) k_full<S>(w, m[0], m[1]);        \
            m += 2;                                                 \
        }
                    QK_F(0) QK_F(1) QK_F(2) QK_F(3) QK_F(4)
#undef QK_F
                    break;
                }
            const bool pending = b & kLayerPending;
#define QK_K(S)                                                     \
    if constexpr ((1 << S) < R)                                     \
        if ((a >> S) & 1) {                                         \
            const T ts = t;                                         \
            C ls = pending ? lam : l;                               \
            m += 2;                                                 \
            t = m[0].x;                                             \
            l = m[1];                                               \
            ls.x = flip_sign(ls.x, neg >> S);                       \
            ls.y = flip_sign(ls.y, neg >> S);                       \
            k_unitary<S>(v, ls, ts);                                \
            if constexpr (NS == 2) k_unitary<S>(w, ls, ts);         \
        }
            QK_K(0) QK_K(1) QK_K(2) QK_K(3) QK_K(4)
#undef QK_K
            if (pending) {
                lam.x = 1;
                lam.y = 0;
            }
            break;
        }
#define QK_P2(A, B)                                      \
    case TOP_PH2 + slot_pair(A, B): {                    \
        const C ph = *m;                                 \
        reg_phase2<A, B>(v, ph);                         \
        if constexpr (NS == 2) reg_phase2<A, B>(w, ph);  \
        break;                                           \
    }
        QK_P2(0, 1) QK_P2(0, 2) QK_P2(1, 2) QK_P2(0, 3) QK_P2(1, 3) QK_P2(2, 3)
        QK_P2(0, 4) QK_P2(1, 4) QK_P2(2, 4) QK_P2(3, 4)
#undef QK_P2
        case TOP_LAM: {
            // the conditions' bits as a table index: one multiply for four
            // conditions (with one each, decoded one by one, the 28-qubit QFT
            // took 24.1 ms)
            uint32_t idx = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t code = ((i < 4 ? op.y : op.z) >> (8 * (i & 3))) & 0xFF;
                const uint32_t bit = (((code & kOuterFlag) ? tile : tb) >> (code & 31)) & 1u;
                if (i < (int)nb) idx |= bit << i;
            }
            lam = cmul(lam, m[idx & 15]);
            if (nb > 4) lam = cmul(lam, m[16 + (idx >> 4)]);
            break;
        }
        case TOP_LCX: {
            if (!labels) {
                labels = true;
#pragma unroll
                for (int s = 0; s < LOG2R; ++s) bm[s] = 1u << ((s < 4 ? slots >> (8 * (s & 3)) : slot5) & 31);
            }
            if (b & kOuterFlag) {
                tb ^= (uint32_t)code_bit(b, base, tb) << a;
            } else {
                tb ^= ((tb >> b) & 1u) << a;
#pragma unroll
                for (int s = 0; s < LOG2R; ++s) bm[s] ^= ((bm[s] >> b) & 1u) << a;
            }
            break;
        }
        case TOP_PHASE: {
            const uint32_t c0 = op.y & 0xFF, c1 = (op.y >> 8) & 0xFF;   // slots
            const bool ba = c0 != kNoSlot || code_bit(a, base, tb), bb = c1 != kNoSlot || code_bit(b, base, tb);
            if (!(ba && bb)) break;
            const C ph = *m;
            switch (c0 != kNoSlot ? c0 : c1) {
            case 0: k_phase<0>(v, ph); if constexpr (NS == 2) k_phase<0>(w, ph); break;
            case 1: k_phase<1>(v, ph); if constexpr (NS == 2) k_phase<1>(w, ph); break;
            case 2: k_phase<2>(v, ph); if constexpr (NS == 2) k_phase<2>(w, ph); break;
            case 3: k_phase<3>(v, ph); if constexpr (NS == 2) k_phase<3>(w, ph); break;
            case 4: k_phase<4>(v, ph); if constexpr (NS == 2) k_phase<4>(w, ph); break;
            default: scale_regs(v, w, ph); break;
            }
            break;
        }
        case TOP_SCALE: {
            C f = *m;
            if (b) {
                scale_regs(v, w, f);
            } else {
#pragma unroll
                for (int kk = 0; kk < R; ++kk) {
                    v[kk].x *= f.x;
                    v[kk].y *= f.x;
                    if constexpr (NS == 2) w[kk].x *= f.x, w[kk].y *= f.x;
                }
            }
            break;
        }
        case TOP_GRAD: {
            if constexpr (NS == 2) {
                T g = 0, g2 = 0;
                switch (a) {   // (two states: three slots at most)
                case 0: g = reg_grad<0>(v, w, (int)b, m, &g2); break;
                case 1: g = reg_grad<1>(v, w, (int)b, m, &g2); break;
                case 2: g = reg_grad<2>(v, w, (int)b, m, &g2); break;
                }
                const uint32_t NT = blockDim.x;
                gsm[(op.y & 0xFFFF) * NT + tid] += (double)g;
                if (b == 5) gsm[(op.y >> 16) * NT + tid] += (double)g2;
            }
            break;
        }
        }
    }
}

// The CTA's gradient accumulators (ngrad slots of one double a thread) added
// to ggrad[gparams[i]].  Threads start at different entries: a slot's
// entries are in different banks.
__device__ __forceinline__ void flush_gradients(const double *gsm, int ngrad, const int32_t *gparams, double *ggrad) {
    const uint32_t NT = blockDim.x;
    for (int i = threadIdx.x; i < ngrad; i += NT) {
        double s = 0;
        for (uint32_t t = 0; t < NT; ++t) s += gsm[(uint32_t)i * NT + ((t + (uint32_t)i) & (NT - 1))];
        atomicAdd(ggrad + gparams[i], s);
    }
}

}  // namespace qk
