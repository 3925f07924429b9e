// Expectation values of Pauli sums and adjoint gradients.
//
// The reference computes no observables and no gradients; these entry points
// are the engine's own (the variational workloads: a circuit of RX/RY/RZ
// rotations and fixed gates, H = sum of Pauli strings).
//
// Adjoint sweep (forward state uncomputed gate by gate, nothing stored but
// a few checkpoints):
//   psi = U_L..U_1 |psi0>, lambda = H psi, <H> = Re <psi|lambda>
//   for k = L..1:  g[p(k)] += Im <lambda|G_k|psi>   (U_k = exp(-i theta G_k / 2))
//                  psi <- U_k^dag psi, lambda <- U_k^dag lambda
// The gradient inner product is fused into the kernel that uncomputes both
// states, so a parameterised gate costs one read and one write of each.
// Forward states are kept at evenly spaced checkpoints; when the backward
// sweep reaches one, the uncomputed state is compared with it (drift) and
// replaced by it.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include <cuda_runtime.h>

#include "qk_devplan.h"
#include "qk_device.h"
#include "qk_internal.h"
#include "qk_kernels.cuh"
#include "qk_pass_device.cuh"

namespace qk {

constexpr int kRedThreads = 256;
constexpr int kMaxGroupTerms = 64;

struct PauliGroup {
    uint64_t x;                       // X/Y part shared by the group
    int nterms;
    double coef[kMaxGroupTerms];      // real coefficient
    uint64_t z[kMaxGroupTerms];       // Z/Y part
    int ipow[kMaxGroupTerms];         // i^ipow from the Y factors (popcount(x & z) mod 4)
};

// factor(src) = sum_t coef_t i^ipow_t (-1)^popcount(src & z_t):
// (P psi)[src ^ x] = factor(src) psi[src]
__device__ __forceinline__ double2 group_factor(const PauliGroup &g, uint64_t src) {
    double re = 0, im = 0;
    for (int t = 0; t < g.nterms; ++t) {
        const double c = (__popcll(src & g.z[t]) & 1) ? -g.coef[t] : g.coef[t];
        switch (g.ipow[t] & 3) {
        case 0: re += c; break;
        case 1: im += c; break;
        case 2: re -= c; break;
        default: im -= c; break;
        }
    }
    return make_double2(re, im);
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double red[kRedThreads / 32];
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (!l) red[w] = v;
    __syncthreads();
    v = (threadIdx.x < blockDim.x / 32) ? red[threadIdx.x] : 0.0;
    if (w == 0)
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// acc += sum_j Re( conj(psi[j]) (P psi)[j] ) over one X-group:
// (P psi)[j] = factor(j ^ x) psi[j ^ x]
template <typename C>
__global__ void __launch_bounds__(kRedThreads) k_pauli_expval(const C *__restrict__ psi, uint64_t namp,
                                                              const __grid_constant__ PauliGroup g, double *acc) {
    double s = 0;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < namp; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t src = j ^ g.x;
        const C a = psi[j], b = psi[src];
        const double2 f = group_factor(g, src);
        // Re( conj(a) f b )
        const double br = (double)b.x * f.x - (double)b.y * f.y, bi = (double)b.x * f.y + (double)b.y * f.x;
        s += (double)a.x * br + (double)a.y * bi;
    }
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(acc, s);
}

// out[j] (+)= (P psi)[j] for one X-group
template <typename C>
__global__ void __launch_bounds__(kRedThreads) k_pauli_apply(C *__restrict__ out, const C *__restrict__ psi, uint64_t namp,
                                                             const __grid_constant__ PauliGroup g, int accumulate) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < namp; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t src = j ^ g.x;
        const C b = psi[src];
        const double2 f = group_factor(g, src);
        double re = (double)b.x * f.x - (double)b.y * f.y, im = (double)b.x * f.y + (double)b.y * f.x;
        if (accumulate) {
            const C o = out[j];
            re += o.x;
            im += o.y;
        }
        out[j] = mk<C>(re, im);
    }
}

// Pauli groups by tiles: all groups whose X masks lie in the tile's bits, from
// one read of the state.  One group a sweep is bound by HBM -- H = sum J Z Z +
// sum h X on 27 qubits took 28 sweeps of a 2 GiB state, 18.2 ms -- and the
// groups of a tile of 2^T amplitudes with the lowest L bits share theirs
// (T - L qubits' X terms a sweep: four sweeps there).
constexpr int kTileGroups = 24, kTileTerms = 64;
constexpr int kTileSlots = 2;   // elements a thread: 2^kTileSlots
struct PauliTile {
    PassDesc d;                            // T, L, bpos
    int ngroups;
    int16_t term0[kTileGroups + 1];        // terms of group g: term0[g] .. term0[g + 1]
    int nsimple;                           // groups of one term without Z: its coefficient (real), and
    double scoef[kTileGroups];             // the places of its partners, an XOR of byte offsets
    uint32_t splace[kTileGroups];
    uint32_t xplace[kTileGroups];          // the same of the other groups' partners
    uint64_t x[kTileGroups];               // and their X masks over the state's bits
    double coef[kTileTerms];
    uint64_t z[kTileTerms];
    uint8_t ipow[kTileTerms];
};

// out (+)= sum of the groups' P psi (out may be null), acc += Re <psi| them >
//
// The sign of term k at an amplitude is the parity of its index & z[k], a sum
// of the parities of the tile's, the thread's and the element's parts: three
// 64-bit words with a bit a term, of which only the tile's is made anew for a
// tile (a lane a term).  With the parities taken term by term, POPC bound the
// kernel (27 qubits, 53 terms: 7.6 ms).  Groups of one X string, the common
// case, have a loop of their own.
// ROUND: out's sum is rounded to C after every group, the groups of several
// terms first, as by a sweep a group (complex64 gradients keep their values
// so: with one rounding a tile they changed by 6e-8); acc is not used.
template <typename C, bool ROUND>
__global__ void __launch_bounds__(kRedThreads, 2) k_pauli_tile(C *__restrict__ out, const C *__restrict__ psi, uint64_t ntiles,
                                                            const __grid_constant__ PauliTile t, int accumulate,
                                                            double *acc) {
    extern __shared__ __align__(16) unsigned char smem_raw[];   // the tile
    const uint32_t NT = blockDim.x, N = 1u << t.d.T, tid = threadIdx.x, lane = tid & 31;
    constexpr int E = 1 << kTileSlots;
    const int nterms = t.term0[t.ngroups];
    // element u of the thread: tid + u NT; its offset is linear in u's bits
    const uint64_t off_t = tid < N ? pass_off(tid, t.d) : 0;
    uint64_t off_u[kTileSlots];
    uint64_t sg_t = 0, sg_u[kTileSlots];   // bit k: parity of the part & z[k]
#pragma unroll
    for (int b = 0; b < kTileSlots; ++b) {
        off_u[b] = (NT << b) < N ? pass_off(NT << b, t.d) : 0;
        sg_u[b] = 0;
    }
    for (int k = 0; k < nterms; ++k) {
        const uint64_t z = t.z[k];
        sg_t |= (uint64_t)(__popcll(off_t & z) & 1) << k;
#pragma unroll
        for (int b = 0; b < kTileSlots; ++b) sg_u[b] |= (uint64_t)(__popcll(off_u[b] & z) & 1) << k;
    }
    // of the lane's terms lane and lane + 32: z, and whether its constant part
    // (x & z, the sign of i^ipow) is negative
    uint64_t z0 = 0, z1 = 0;
    int c0 = 0, c1 = 0;
    for (int g = 0; g < t.ngroups; ++g)
        for (int k = t.term0[g]; k < t.term0[g + 1]; ++k) {
            const int c = (__popcll(t.x[g] & t.z[k]) & 1) ^ (t.ipow[k] >> 1);
            if (k == (int)lane) z0 = t.z[k], c0 = c;
            if (k == (int)lane + 32) z1 = t.z[k], c1 = c;
        }
    uint32_t place[E];   // (elements past a small tile's end: those of its start)
#pragma unroll
    for (int u = 0; u < E; ++u) place[u] = swz<C>((tid + u * NT) & (N - 1)) * (uint32_t)sizeof(C);
    double sum = 0;
    uint64_t off[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        off[u] = off_t;
#pragma unroll
        for (int b = 0; b < kTileSlots; ++b)
            if ((u >> b) & 1) off[u] |= off_u[b];
    }
    // a tile's amplitudes are loaded while the one before it is worked on
    C next[E];
    uint64_t base = 0;
    auto load = [&](uint64_t o) {
        base = pass_base(o, t.d);
#pragma unroll
        for (int u = 0; u < E; ++u)
            if (tid + u * NT < N) next[u] = psi[base | off[u]];
    };
    if (blockIdx.x < ntiles) load(blockIdx.x);
    for (uint64_t o = blockIdx.x; o < ntiles; o += gridDim.x) {
        const uint64_t here = base;
        C v[E];
#pragma unroll
        for (int u = 0; u < E; ++u) {
            v[u] = next[u];
            if (tid + u * NT < N) *reinterpret_cast<C *>(smem_raw + place[u]) = v[u];
        }
        __syncthreads();
        if (o + gridDim.x < ntiles) load(o + gridDim.x);
        uint64_t sg[E];
        const uint64_t sg_tile =
            (uint64_t)__ballot_sync(0xffffffffu, (__popcll(here & z1) ^ c1) & 1) << 32 |
            __ballot_sync(0xffffffffu, (__popcll(here & z0) ^ c0) & 1);
#pragma unroll
        for (int u = 0; u < E; ++u) {
            sg[u] = sg_tile ^ sg_t;
#pragma unroll
            for (int b = 0; b < kTileSlots; ++b)
                if ((u >> b) & 1) sg[u] ^= sg_u[b];
        }
        double re[E], im[E];
#pragma unroll
        for (int u = 0; u < E; ++u) {
            re[u] = im[u] = 0;
            if (ROUND && accumulate && tid + u * NT < N) {
                const C b = out[here | off[u]];
                re[u] = b.x;
                im[u] = b.y;
            }
        }
        auto rounded = [&](int u) {
            if constexpr (ROUND) {
                const C b = mk<C>(re[u], im[u]);
                re[u] = b.x;
                im[u] = b.y;
            }
        };
        // += (fr + i fi) b, the group's factor at the element
        auto add = [&](int u, const C b, double fr, double fi) {
            re[u] += fr * (double)b.x - fi * (double)b.y;
            im[u] += fr * (double)b.y + fi * (double)b.x;
        };
        for (int g = 0; g < t.ngroups; ++g) {
            const int t0 = t.term0[g], t1 = t.term0[g + 1];
            const uint32_t xp = t.xplace[g];
            double fr[E], fi[E];
#pragma unroll
            for (int u = 0; u < E; ++u) fr[u] = fi[u] = 0;
            for (int k = t0; k < t1; ++k) {
                const double c = t.coef[k];
                const bool odd = t.ipow[k] & 1;
#pragma unroll
                for (int u = 0; u < E; ++u) {
                    const uint32_t w = k < 32 ? (uint32_t)sg[u] : (uint32_t)(sg[u] >> 32);
                    const double s = __hiloint2double(__double2hiint(c) ^ (int)((w >> (k & 31)) << 31), __double2loint(c));
                    if (odd) fi[u] += s;
                    else fr[u] += s;
                }
            }
#pragma unroll
            for (int u = 0; u < E; ++u) {
                add(u, *reinterpret_cast<const C *>(smem_raw + (place[u] ^ xp)), fr[u], fi[u]);
                rounded(u);
            }
        }
#pragma unroll 4
        for (int g = 0; g < t.nsimple; ++g) {
            const double c = t.scoef[g];
            const uint32_t xp = t.splace[g];
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const C b = *reinterpret_cast<const C *>(smem_raw + (place[u] ^ xp));
                re[u] += c * (double)b.x;
                im[u] += c * (double)b.y;
                rounded(u);
            }
        }
#pragma unroll
        for (int u = 0; u < E; ++u)
            if (tid + u * NT < N) {
                sum += (double)v[u].x * re[u] + (double)v[u].y * im[u];
                if (out) {
                    C *p = out + (here | off[u]);
                    if (!ROUND && accumulate) {
                        re[u] += p->x;
                        im[u] += p->y;
                    }
                    *p = mk<C>(re[u], im[u]);
                }
            }
        __syncthreads();
    }
    if (acc) {
        sum = block_sum(sum);
        if (threadIdx.x == 0) atomicAdd(acc, sum);
    }
}

// acc += Re <a|b>
template <typename C>
__global__ void __launch_bounds__(kRedThreads) k_dot_re(const C *__restrict__ a, const C *__restrict__ b, uint64_t namp,
                                                        double *acc) {
    double s = 0;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < namp; j += (uint64_t)gridDim.x * blockDim.x)
        s += (double)a[j].x * b[j].x + (double)a[j].y * b[j].y;
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(acc, s);
}

// acc += ||a - b||^2
template <typename C>
__global__ void __launch_bounds__(kRedThreads) k_dist2(const C *__restrict__ a, const C *__restrict__ b, uint64_t namp,
                                                       double *acc) {
    double s = 0;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < namp; j += (uint64_t)gridDim.x * blockDim.x) {
        const double dx = (double)a[j].x - b[j].x, dy = (double)a[j].y - b[j].y;
        s += dx * dx + dy * dy;
    }
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(acc, s);
}

// Im(conj(l) a)
template <typename C> __device__ __forceinline__ double im_dot(C l, C a) {
    return (double)l.x * a.y - (double)l.y * a.x;
}
template <typename C> __device__ __forceinline__ double re_dot(C l, C a) {
    return (double)l.x * a.x + (double)l.y * a.y;
}

// One parameterised rotation on qubit t, backward step: gradient
// Im<lambda|G|psi> (G = X, Y or Z by gen = 1, 2, 3) and both states
// multiplied by U^dag (u).
template <typename C>
__global__ void __launch_bounds__(kRedThreads) k_adj_rot(C *__restrict__ psi, C *__restrict__ lam, uint64_t npairs, int t,
                                                         Mat2<C> u, int gen, double *gacc) {
    const uint64_t h = 1ull << t;
    double s = 0;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npairs; p += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i0 = ins0(p, t), i1 = i0 + h;
        const C a0 = psi[i0], a1 = psi[i1], l0 = lam[i0], l1 = lam[i1];
        if (gen == 1) s += im_dot(l0, a1) + im_dot(l1, a0);
        else if (gen == 2) s += re_dot(l1, a0) - re_dot(l0, a1);
        else s += im_dot(l0, a0) - im_dot(l1, a1);
        psi[i0] = cmul2(u.m[0], a0, u.m[1], a1);
        psi[i1] = cmul2(u.m[2], a0, u.m[3], a1);
        lam[i0] = cmul2(u.m[0], l0, u.m[1], l1);
        lam[i1] = cmul2(u.m[2], l0, u.m[3], l1);
    }
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(gacc, s);
}

// from qk_engine.cu
int launch_gate_op(void *state, int n, int dtype, const Op &op, cudaStream_t st);

static int cuda_err(cudaError_t e, const char *what) {
    // An allocation failure is not sticky, but it stays as the thread's last
    // error; clear it so the next launch check does not report it again.
    if (e == cudaErrorMemoryAllocation) (void)cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? QK_ERR_OOM : QK_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

static unsigned red_grid(uint64_t items) {
    const int sms = device_sms();
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + kRedThreads - 1) / kRedThreads, (uint64_t)sms * 8));
}

// Group Pauli terms by their X/Y mask.
static int group_terms(const qk_pauli_term *terms, size_t nterms, int n, std::vector<PauliGroup> &groups) {
    std::map<uint64_t, size_t> idx;
    const uint64_t all = n >= 64 ? ~0ull : ((1ull << n) - 1);
    for (size_t t = 0; t < nterms; ++t) {
        if ((terms[t].x_mask | terms[t].z_mask) & ~all)
            return fail(QK_ERR_QUBIT, "Pauli term %zu acts on a qubit >= %d", t, n);
        auto it = idx.find(terms[t].x_mask);
        if (it == idx.end() || groups[it->second].nterms == kMaxGroupTerms) {
            PauliGroup g;
            std::memset(&g, 0, sizeof g);
            g.x = terms[t].x_mask;
            groups.push_back(g);
            it = idx.insert_or_assign(terms[t].x_mask, groups.size() - 1).first;
        }
        PauliGroup &g = groups[it->second];
        g.coef[g.nterms] = terms[t].coeff;
        g.z[g.nterms] = terms[t].z_mask;
        g.ipow[g.nterms] = __builtin_popcountll(terms[t].x_mask & terms[t].z_mask) & 3;
        ++g.nterms;
    }
    return QK_OK;
}

// Tile bits of k_pauli_tile: kRedThreads threads with 2^kTileSlots elements
// each, 16 KB of complex128.
constexpr int kPauliTileBits = 8 + kTileSlots;
static_assert(1 << (kPauliTileBits - kTileSlots) == kRedThreads, "elements a thread");

// Whether <H> of a group that shares its tile with no other is faster from
// k_pauli_expval.  A tile pays for its shared-memory trip and set-up with the
// signs of many terms (27 qubits, 32 terms: 3.9 -> 1.8 ms) or, in complex128,
// with partners that a sweep reads a second time (one term, top qubit: 0.73 ->
// 0.44 ms).  States of L2's size, microseconds flat / by tile: 20 qubits, one
// term 27 / 29 to 28 / 36, 8 terms 38 / 40, 16 terms 53 / 43; 14 qubits, one
// term 25 / 27, 32 terms 36 / 46.  Above, complex64, 25 qubits: one term 111 /
// 123, two 148 / 136.
static bool flat_alone(int nterms, int n, int dtype) {
    const uint64_t bytes = (dtype == QK_C128 ? 16ull : 8ull) << n;
    if (bytes <= 1ull << 20) return true;
    if (bytes <= 16ull << 20) return nterms <= 8;
    return dtype == QK_C64 && nterms == 1;
}

// The groups whose X masks fit a tile, cut into tiles; the others stay in
// `flat` (one sweep each).  apply: for H psi, where <H> comes with the tiles.
static void tile_groups(const std::vector<PauliGroup> &groups, int n, int dtype, bool apply, std::vector<PauliTile> &tiles,
                        std::vector<const PauliGroup *> &flat) {
    const int T = std::min(n, kPauliTileBits), L = std::min(T, dtype == QK_C128 ? 3 : 4);   // 128-byte runs
    const uint64_t low = (1ull << L) - 1;
    std::vector<const PauliGroup *> left;
    for (const PauliGroup &g : groups) {
        if (__builtin_popcountll(g.x | low) > T) flat.push_back(&g);
        else left.push_back(&g);
    }
    std::stable_sort(left.begin(), left.end(), [](const PauliGroup *a, const PauliGroup *b) { return a->x < b->x; });
    while (!left.empty()) {
        uint64_t bits = low;
        std::vector<const PauliGroup *> take, rest;
        int nt = 0;
        for (const PauliGroup *g : left) {
            const bool ok = (int)take.size() < kTileGroups && nt + g->nterms <= kTileTerms &&
                            __builtin_popcountll(bits | g->x) <= T;
            (ok ? take : rest).push_back(g);
            if (ok) bits |= g->x, nt += g->nterms;
        }
        left.swap(rest);
        if (!apply && take.size() == 1 && flat_alone(take[0]->nterms, n, dtype)) {
            flat.push_back(take[0]);
            continue;
        }
        PauliTile t;
        std::memset(&t, 0, sizeof t);
        for (int q = 0; __builtin_popcountll(bits) < T; ++q) bits |= 1ull << q;
        t.d.T = T;
        for (int q = 0, k = 0; q < n; ++q)
            if ((bits >> q) & 1) t.d.bpos[k++] = q;
        while (t.d.L < T && t.d.bpos[t.d.L] == t.d.L) ++t.d.L;
        int k = 0;
        for (const PauliGroup *g : take) {
            uint32_t xl = 0;
            for (int b = 0; b < T; ++b) xl |= (uint32_t)((g->x >> t.d.bpos[b]) & 1) << b;
            const uint32_t place = tile_swizzle(xl, dtype == QK_C128) * (dtype == QK_C128 ? 16 : 8);
            if (g->nterms == 1 && !g->z[0]) {
                t.scoef[t.nsimple] = g->coef[0];
                t.splace[t.nsimple++] = place;
                continue;
            }
            t.x[t.ngroups] = g->x;
            t.xplace[t.ngroups] = place;
            t.term0[t.ngroups++] = (int16_t)k;
            for (int i = 0; i < g->nterms; ++i, ++k) {
                t.coef[k] = g->coef[i];
                t.z[k] = g->z[i];
                t.ipow[k] = (uint8_t)g->ipow[i];
            }
        }
        t.term0[t.ngroups] = (int16_t)k;
        tiles.push_back(t);
    }
}

// What a call of pauli_sum_t launched: sweeps over psi, and whether <H> was a
// sweep of its own (k_dot_re).
struct PauliSweeps {
    int sums = 0;
    bool dot = false;
    int launches() const { return std::max(1, sums) + dot; }   // (an empty sum clears out)
    // bytes of H psi on states of S bytes: psi read and out written, by every
    // further sweep out read too; the dot reads both
    double bytes(double S) const { return sums ? 2 * S + 3 * S * (sums - 1) + (dot ? 2 * S : 0) : S; }
};

// out = H psi (out may be null) and, with acc (zero before), *acc = <H>.
template <typename C>
static int pauli_sum_t(C *out, const C *psi, int n, const std::vector<PauliGroup> &groups, double *acc, cudaStream_t st,
                       PauliSweeps *sweeps = nullptr) {
    const uint64_t namp = 1ull << n;
    if (groups.empty()) {
        cudaError_t e = out ? cudaMemsetAsync(out, 0, sizeof(C) * namp, st) : cudaSuccess;
        return e == cudaSuccess ? QK_OK : cuda_err(e, "memset");
    }
    std::vector<PauliTile> tiles;
    std::vector<const PauliGroup *> flat;
    tile_groups(groups, n, sizeof(C) == sizeof(double2) ? QK_C128 : QK_C64, out != nullptr, tiles, flat);
    constexpr bool c64 = sizeof(C) == sizeof(float2);
    const bool round = c64 && out, dot = out && acc && (round || !flat.empty());   // dot: <H> from all of H psi
    if (sweeps) *sweeps = {(int)(tiles.size() + flat.size()), dot};
    const auto kernel = round ? k_pauli_tile<C, c64> : k_pauli_tile<C, false>;
    int done = 0;
    for (const PauliTile &t : tiles) {
        const unsigned threads = std::min(kRedThreads, std::max(32, (1 << t.d.T) >> kTileSlots));
        const size_t smem = sizeof(C) << t.d.T;
        int mb = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&mb, kernel, (int)threads, smem);
        if (e != cudaSuccess || mb < 1) mb = 1;
        const uint64_t ntiles = namp >> t.d.T;
        const unsigned grid = (unsigned)std::min<uint64_t>(ntiles, (uint64_t)device_sms() * mb);
        kernel<<<grid, threads, smem, st>>>(out, psi, ntiles, t, done++ > 0, dot ? nullptr : acc);
        e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_err(e, "k_pauli_tile");
    }
    for (const PauliGroup *gp : flat) {
        const PauliGroup &g = *gp;
        if (out) k_pauli_apply<C><<<red_grid(namp), kRedThreads, 0, st>>>(out, psi, namp, g, done++ > 0);
        else k_pauli_expval<C><<<red_grid(namp), kRedThreads, 0, st>>>(psi, namp, g, acc);
    }
    if (dot) k_dot_re<C><<<red_grid(namp), kRedThreads, 0, st>>>(psi, out, namp, acc);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QK_OK : cuda_err(e, "k_pauli");
}

// generator of a trainable gate: 1 X (RX), 2 Y (RY), 3 Z (RZ), 0 not trainable
static int generator(const qk_gate &g) {
    return g.kind == QK_GATE_RX ? 1 : g.kind == QK_GATE_RY ? 2 : g.kind == QK_GATE_RZ ? 3 : 0;
}

template <typename C>
static int adjoint_t(C *psi, int n, int dtype, const qk_gate *gates, size_t ng, const int32_t *pidx, size_t nparams,
                     const std::vector<PauliGroup> &groups, int ncheck, double *expval, double *grad, double *drift,
                     Workspace &ws, cudaStream_t st) {
    const uint64_t namp = 1ull << n;
    const size_t bytes = sizeof(C) * namp;
    std::vector<Op> ops(ng);
    for (size_t i = 0; i < ng; ++i) {
        int rc = lower_gate(gates[i], ops[i]);
        if (rc) return rc;
        for (int k = 0; k < ops[i].nq; ++k)
            if (ops[i].q[k] < 0 || ops[i].q[k] >= n)
                return fail(QK_ERR_QUBIT, "gate %zu: qubit %d outside a %d-qubit state", i, ops[i].q[k], n);
        if (pidx && pidx[i] >= 0) {
            if ((size_t)pidx[i] >= nparams) return fail(QK_ERR_ARG, "gate %zu: parameter %d >= %zu", i, pidx[i], nparams);
            if (!generator(gates[i])) return fail(QK_ERR_UNSUPPORTED, "gate %zu: only RX, RY, RZ are trainable", i);
        }
    }
    // checkpoints: the state before gate c for evenly spaced c
    std::vector<size_t> cpos;
    if (ncheck < 0) ncheck = 0;
    if (ncheck > 0 && ng > 1) {
        for (int k = 1; k <= ncheck; ++k) {
            size_t c = (size_t)((double)ng * k / (ncheck + 1));
            if (c > 0 && c < ng && (cpos.empty() || c > cpos.back())) cpos.push_back(c);
        }
    }
    cudaError_t e = ws.reserve(bytes * (1 + cpos.size()), (nparams + 2) * sizeof(double), 0);
    if (e != cudaSuccess) return cuda_err(e, "cudaMalloc(adjoint workspace: lambda, checkpoints)");
    C *lam = static_cast<C *>(ws.states);
    C *ck = lam + namp;
    double *dacc = ws.acc;
    int rc = QK_OK;
    const size_t nacc = nparams + 2;  // grads, expval, drift
    e = ws.events();
    if (e == cudaSuccess) e = cudaEventRecord(ws.ev0, st);
    if (e != cudaSuccess) return cuda_err(e, "sweep timing events");
    ws.last_fwd = ws.last_bwd = (int)ng;   // one launch per gate each way
    ws.last_bytes = 0;                     // not counted for the per-gate sweep
    e = cudaMemsetAsync(dacc, 0, nacc * sizeof(double), st);
    if (e != cudaSuccess) return cuda_err(e, "clear accumulators");

    // forward, saving checkpoints
    size_t nc = 0;
    for (size_t i = 0; i < ng; ++i) {
        if (nc < cpos.size() && cpos[nc] == i) {
            e = cudaMemcpyAsync(ck + nc * namp, psi, bytes, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return cuda_err(e, "checkpoint");
            ++nc;
        }
        rc = launch_gate_op(psi, n, dtype, ops[i], st);
        if (rc) return rc;
    }
    // lambda = H psi, <H> = Re<psi|lambda>
    PauliSweeps hs;
    rc = pauli_sum_t<C>(lam, psi, n, groups, dacc + nparams, st, &hs);
    if (rc) return rc;
    ws.last_other = (int)(hs.launches() + 3 * cpos.size());
    // backward
    for (size_t i = ng; i-- > 0;) {
        Op inv = ops[i];
        invert_op(inv);
        const int p = pidx ? pidx[i] : -1;
        if (p >= 0) {
            Mat2<C> u;
            // RX/RY lower to dense 2x2, RZ to a diagonal: both as dense U^dag here
            if (inv.kind == OP_DENSE1) {
                for (int k = 0; k < 4; ++k) u.m[k] = mk<C>(inv.m[2 * k], inv.m[2 * k + 1]);
            } else {
                u.m[0] = mk<C>(inv.m[0], inv.m[1]);
                u.m[1] = mk<C>(0, 0);
                u.m[2] = mk<C>(0, 0);
                u.m[3] = mk<C>(inv.m[2], inv.m[3]);
            }
            const uint64_t np = namp / 2;
            k_adj_rot<C><<<red_grid(np), kRedThreads, 0, st>>>(psi, lam, np, inv.q[0], u, generator(gates[i]), dacc + p);
            e = cudaGetLastError();
            if (e != cudaSuccess) return cuda_err(e, "k_adj_rot");
        } else {
            rc = launch_gate_op(psi, n, dtype, inv, st);
            if (!rc) rc = launch_gate_op(lam, n, dtype, inv, st);
            if (rc) return rc;
        }
        // psi now holds the state before gate i: compare with and restore from a checkpoint
        if (nc > 0 && cpos[nc - 1] == i) {
            --nc;
            k_dist2<C><<<red_grid(namp), kRedThreads, 0, st>>>(psi, ck + nc * namp, namp, dacc + nparams + 1);
            e = cudaMemcpyAsync(psi, ck + nc * namp, bytes, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return cuda_err(e, "restore checkpoint");
        }
    }
    e = cudaEventRecord(ws.ev1, st);
    if (e != cudaSuccess) return cuda_err(e, "sweep timing events");
    std::vector<double> h(nacc);
    e = cudaMemcpyAsync(h.data(), dacc, nacc * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_err(e, "read results");
    {
        float ms = 0;
        ws.last_ms = cudaEventElapsedTime(&ms, ws.ev0, ws.ev1) == cudaSuccess ? ms : -1.0;
    }
    if (grad) std::memcpy(grad, h.data(), nparams * sizeof(double));
    if (expval) *expval = h[nparams];
    if (drift) *drift = std::sqrt(h[nparams + 1]);
    return QK_OK;
}

// fused passes (qk_pass.cu)
int upload_host_plan(const HostPlan &hp, DevPlan &dp, cudaStream_t st);
int run_forward_plan(void *state, const HostPlan &hp, const DevPlan &dp, cudaStream_t st);
int run_adjoint_plan(void *psi, void *lam, int dtype, const HostPlan &hp, const DevPlan &dp, double *ggrad,
                     cudaStream_t st);

// The same sweep with fused passes: the gates are cut into segments at the
// checkpoints; each segment runs forward as fused passes and backward as
// two-state adjoint passes (inverse gates on psi and lambda, gradients taken
// inside the passes).  At a segment start psi is compared with and restored
// from the checkpoint.
template <typename C>
static int adjoint_fused_t(C *psi, int n, int dtype, const qk_gate *gates, size_t ng, const int32_t *pidx,
                           size_t nparams, const std::vector<PauliGroup> &groups, int ncheck, double *expval,
                           double *grad, double *drift, Workspace &ws, cudaStream_t st) {
    const uint64_t namp = 1ull << n;
    const size_t bytes = sizeof(C) * namp;
    std::vector<size_t> cut{0};
    if (ncheck > 0 && ng > 1)
        for (int k = 1; k <= ncheck; ++k) {
            size_t c = (size_t)((double)ng * k / (ncheck + 1));
            if (c > cut.back() && c < ng) cut.push_back(c);
        }
    cut.push_back(ng);
    const size_t nseg = cut.size() - 1;
    std::vector<HostPlan> fwd(nseg), bwd(nseg);
    // complex64 sweeps run the general programs both ways: with factored
    // forward passes the 23-qubit HEA sweep of 10 layers took 18.1 ms against
    // 17.9, its two-state passes being most of it
    const PlanOptions fo = dtype == QK_C128 ? factored_plan_options(dtype, n) : default_plan_options(dtype, n);
    const PlanOptions bo = factored_adjoint_options(dtype, n);
    // planning takes longer than the sweep of a small state: every segment's
    // two plans on threads of their own (13 qubits, 190 gates: 1.2 -> 0.4 ms;
    // 26 qubits, 924 gates: 12 -> 3 ms)
    auto plan_one = [&](size_t k) {
        const size_t sgi = k / 2, cnt = cut[sgi + 1] - cut[sgi];
        const qk_gate *g = gates + cut[sgi];
        return k % 2 ? plan_adjoint(g, cnt, pidx ? pidx + cut[sgi] : nullptr, n, bo, bwd[sgi])
                     : plan_forward(g, cnt, n, fo, fwd[sgi]);
    };
    if (ng >= 100) {
        int rc = run_tasks(2 * nseg, std::ref(plan_one));   // (no allocation for the callable)
        if (rc) return rc;
    }
    for (size_t sgi = 0; sgi < nseg; ++sgi) {
        for (size_t k = 2 * sgi; k < 2 * sgi + 2 && ng < 100; ++k) {
            int rc = plan_one(k);
            if (rc) return rc;
        }
        for (int32_t p : bwd[sgi].grad_params)
            if (p < 0 || (size_t)p >= nparams) return fail(QK_ERR_ARG, "parameter %d >= %zu", p, nparams);
    }
    const size_t nacc = nparams + 2;
    cudaError_t e = ws.reserve(bytes * nseg, nacc * sizeof(double), 2 * nseg);
    if (e != cudaSuccess) return cuda_err(e, "cudaMalloc(adjoint workspace: lambda, checkpoints)");
    C *lam = static_cast<C *>(ws.states);
    C *ck = lam + namp;
    double *dacc = ws.acc;
    for (size_t sgi = 0; sgi < nseg; ++sgi) {
        int rc = upload_host_plan(fwd[sgi], ws.plans[2 * sgi], st);
        if (!rc) rc = upload_host_plan(bwd[sgi], ws.plans[2 * sgi + 1], st);
        if (rc) return rc;
    }
    e = ws.events();
    if (e == cudaSuccess) e = cudaEventRecord(ws.ev0, st);
    if (e != cudaSuccess) return cuda_err(e, "sweep timing events");
    e = cudaMemsetAsync(dacc, 0, nacc * sizeof(double), st);
    if (e != cudaSuccess) return cuda_err(e, "clear accumulators");
    ws.last_fwd = ws.last_bwd = ws.last_other = 0;
    for (size_t sgi = 0; sgi < nseg; ++sgi) {
        ws.last_fwd += (int)fwd[sgi].passes.size();
        ws.last_bwd += (int)bwd[sgi].passes.size();
    }
    // forward
    for (size_t sgi = 0; sgi < nseg; ++sgi) {
        if (sgi > 0) {
            e = cudaMemcpyAsync(ck + (sgi - 1) * namp, psi, bytes, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return cuda_err(e, "checkpoint");
        }
        int rc = run_forward_plan(psi, fwd[sgi], ws.plans[2 * sgi], st);
        if (rc) return rc;
    }
    PauliSweeps hs;
    int rc = pauli_sum_t<C>(lam, psi, n, groups, dacc + nparams, st, &hs);
    if (rc) return rc;
    // algorithmic traffic: a forward pass reads and writes psi (2S), a
    // two-state pass psi and lambda (4S); each checkpoint copy, drift check
    // and restore 2S
    const double S = (double)bytes;
    ws.last_other = (int)(hs.launches() + 3 * (nseg - 1));
    ws.last_bytes = 2 * S * ws.last_fwd + 4 * S * ws.last_bwd + hs.bytes(S) + 3 * 2 * S * (double)(nseg - 1);
    // backward
    for (size_t sgi = nseg; sgi-- > 0;) {
        rc = run_adjoint_plan(psi, lam, dtype, bwd[sgi], ws.plans[2 * sgi + 1], dacc, st);
        if (rc) return rc;
        if (sgi > 0) {
            k_dist2<C><<<red_grid(namp), kRedThreads, 0, st>>>(psi, ck + (sgi - 1) * namp, namp, dacc + nparams + 1);
            e = cudaMemcpyAsync(psi, ck + (sgi - 1) * namp, bytes, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return cuda_err(e, "restore checkpoint");
        }
    }
    e = cudaEventRecord(ws.ev1, st);
    if (e != cudaSuccess) return cuda_err(e, "sweep timing events");
    std::vector<double> h(nacc);
    e = cudaMemcpyAsync(h.data(), dacc, nacc * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_err(e, "read results");
    {
        float ms = 0;
        ws.last_ms = cudaEventElapsedTime(&ms, ws.ev0, ws.ev1) == cudaSuccess ? ms : -1.0;
    }
    if (grad) std::memcpy(grad, h.data(), nparams * sizeof(double));
    if (expval) *expval = h[nparams];
    if (drift) *drift = std::sqrt(h[nparams + 1]);
    return QK_OK;
}

}  // namespace qk

using namespace qk;

// state accessors defined in qk_engine.cu
namespace qk {
cudaStream_t state_stream(const qk_sv *sv);
void *state_ptr(const qk_sv *sv);
int state_qubits(const qk_sv *sv);
int state_dtype(const qk_sv *sv);
Workspace &state_workspace(qk_sv *sv);
}  // namespace qk

extern "C" {

int qk_expval_pauli(qk_sv *sv, const qk_pauli_term *terms, size_t nterms, double *out) {
    if (!sv || !out || (!terms && nterms)) return fail(QK_ERR_ARG, "null argument");
    const int n = state_qubits(sv);
    std::vector<PauliGroup> groups;
    int rc = group_terms(terms, nterms, n, groups);
    if (rc) return rc;
    cudaStream_t st = state_stream(sv);
    Workspace &ws = state_workspace(sv);
    cudaError_t e = ws.reserve(0, sizeof(double), 0);
    if (e != cudaSuccess) return cuda_err(e, "cudaMalloc(accumulator)");
    double *dacc = ws.acc;
    e = cudaMemsetAsync(dacc, 0, sizeof(double), st);
    if (e != cudaSuccess) return cuda_err(e, "clear accumulator");
    rc = state_dtype(sv) == QK_C128
             ? pauli_sum_t<double2>(nullptr, (const double2 *)state_ptr(sv), n, groups, dacc, st)
             : pauli_sum_t<float2>(nullptr, (const float2 *)state_ptr(sv), n, groups, dacc, st);
    if (!rc) {
        e = cudaMemcpyAsync(out, dacc, sizeof(double), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = cuda_err(e, "read expectation");
    }
    return rc;
}

int qk_adjoint_grad(qk_sv *sv, const qk_gate *gates, size_t ngates, const int32_t *param_index, size_t nparams,
                    const qk_pauli_term *terms, size_t nterms, int checkpoints, double *expval, double *grad,
                    double *drift) {
    if (!sv || (!gates && ngates) || (!terms && nterms) || (!grad && nparams))
        return fail(QK_ERR_ARG, "null argument");
    const int n = state_qubits(sv);
    std::vector<PauliGroup> groups;
    int rc = group_terms(terms, nterms, n, groups);
    if (rc) return rc;
    if (checkpoints < 0) checkpoints = std::min<int>(8, (int)std::ceil(std::sqrt((double)ngates)));
    const int dtype = state_dtype(sv);
    cudaStream_t st = state_stream(sv);
    if (dtype == QK_C128)
        return adjoint_t<double2>((double2 *)state_ptr(sv), n, dtype, gates, ngates, param_index, nparams, groups,
                                  checkpoints, expval, grad, drift, state_workspace(sv), st);
    return adjoint_t<float2>((float2 *)state_ptr(sv), n, dtype, gates, ngates, param_index, nparams, groups,
                             checkpoints, expval, grad, drift, state_workspace(sv), st);
}

int qk_adjoint_grad_fused(qk_sv *sv, const qk_gate *gates, size_t ngates, const int32_t *param_index, size_t nparams,
                          const qk_pauli_term *terms, size_t nterms, int checkpoints, double *expval, double *grad,
                          double *drift) {
    if (!sv || (!gates && ngates) || (!terms && nterms) || (!grad && nparams))
        return fail(QK_ERR_ARG, "null argument");
    const int n = state_qubits(sv);
    std::vector<PauliGroup> groups;
    int rc = group_terms(terms, nterms, n, groups);
    if (rc) return rc;
    if (checkpoints < 0) checkpoints = std::min<int>(8, (int)std::ceil(std::sqrt((double)ngates)) / 4);
    const int dtype = state_dtype(sv);
    cudaStream_t st = state_stream(sv);
    if (dtype == QK_C128)
        return adjoint_fused_t<double2>((double2 *)state_ptr(sv), n, dtype, gates, ngates, param_index, nparams,
                                        groups, checkpoints, expval, grad, drift, state_workspace(sv), st);
    return adjoint_fused_t<float2>((float2 *)state_ptr(sv), n, dtype, gates, ngates, param_index, nparams, groups,
                                   checkpoints, expval, grad, drift, state_workspace(sv), st);
}

}  // extern "C"
