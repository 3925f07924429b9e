// Factored-pass kernel (plans of qk_factor.cpp): one CTA owns one tile of 2^T
// amplitudes at a time.  Each thread loads its amplitudes of the tile straight
// into registers, runs the pass's steps on them (qk_fpass_device.cuh) and
// stores them.  There is no staging buffer: the shared memory it takes holds
// another CTA or two, whose steps cover this one's loads better than a
// prefetched tile did (28-qubit 20-layer brick circuit, complex128: 69 ms with
// staging, 65 without).
//
// What bounds it, complex128 on that circuit: a unitary takes 143 cycles of a
// scheduler's FP64 pipe a warp (128 are the pipe's own), a re-mapping 512
// cycles of the shared-memory pipe; the two add up to about three quarters of
// the time, the rest is the latency of steps and loads that 16 warps an SM do
// not cover.  The general programs took 131 ms, this one 66 (2.2 times the
// time of its 23 passes' HBM traffic) and 70 with the worst of its rounded
// matrices in the full form.  complex64, 29 qubits: 169 -> 71 ms,
// issue bound (64 % of the slots).  A tile's offset comes from the uniform
// loop of pass_base: gathered over the lanes by two reductions it delayed the
// loads (complex64 76 ms).
#include <algorithm>
#include <cstring>

#include <cuda_runtime.h>

#include "qk_device.h"
#include "qk_internal.h"
#include "qk_kernels.cuh"
#include "qk_fpass_device.cuh"

namespace qk {

template <typename C, int R, int NS, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_fpass(C *__restrict__ s, C *__restrict__ s2, uint32_t ntiles,
                                                      const __grid_constant__ PassDesc d, const TOp *__restrict__ gprog,
                                                      const C *__restrict__ gcoef, const int32_t *__restrict__ gparams,
                                                      double *__restrict__ ggrad) {
    constexpr int LOG2R = R == 2 ? 1 : R == 4 ? 2 : R == 8 ? 3 : R == 16 ? 4 : 5;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t N = 1u << d.T, NT = blockDim.x, tid = threadIdx.x;
    // exchange buffer (at the start: its places are byte offsets), absent
    // from a pass of one mapping; program; coefficients; gradient accumulators
    TOp *prog = reinterpret_cast<TOp *>(smem_raw + (d.last ? (size_t)N * NS * sizeof(C) : 0));
    C *coef = reinterpret_cast<C *>(prog + d.nprog);
    double *gsm = reinterpret_cast<double *>(coef + d.ncoef);
    for (int i = tid; i < d.nprog; i += NT) prog[i] = gprog[d.prog0 + i];
    for (int i = tid; i < d.ncoef; i += NT) coef[i] = gcoef[d.coef0 + i];
    if constexpr (NS == 2)
        for (int i = tid; i < d.ngrad * (int)NT; i += NT) gsm[i] = 0.0;
    __syncthreads();
    auto lane_offset = [&](int p) {   // state offset of the thread under the mapping prog[p]
        const uint4 op = reinterpret_cast<const uint4 *>(prog)[p];
        return pass_off(slot_deposit<LOG2R>(tid, op.y, op.z), d);
    };
    const uint64_t g_first = lane_offset(0), g_last = lane_offset(d.last);
    for (uint32_t o = blockIdx.x; o < ntiles; o += gridDim.x) {
        const uint64_t base = pass_base(o, d);
        C v[R], w[NS == 2 ? R : 1];
        C *a[R];
        slot_addresses<LOG2R>(s + (base | g_first), d.fpos, a);
#pragma unroll
        for (int u = 0; u < R; ++u) v[u] = *a[u];
        if constexpr (NS == 2) {
            slot_addresses<LOG2R>(s2 + (base | g_first), d.fpos, a);
#pragma unroll
            for (int u = 0; u < R; ++u) w[u] = *a[u];
        }
        // every thread is past the previous tile's last exchange
        __syncthreads();
        run_steps<C, R, NS>(v, w, smem_raw, N * (uint32_t)sizeof(C), base, o, prog, d.nprog, coef, gsm);
        slot_addresses<LOG2R>(s + (base | g_last), d.lpos, a);
#pragma unroll
        for (int u = 0; u < R; ++u) *a[u] = v[u];
        if constexpr (NS == 2) {
            slot_addresses<LOG2R>(s2 + (base | g_last), d.lpos, a);
#pragma unroll
            for (int u = 0; u < R; ++u) *a[u] = w[u];
        }
    }
    if constexpr (NS == 2) {
        __syncthreads();
        flush_gradients(gsm, d.ngrad, gparams + d.grad0, ggrad);
    }
}

static int cuda_err(cudaError_t e, const char *what) {
    // (an allocation failure is not sticky but stays as the thread's last error)
    if (e == cudaErrorMemoryAllocation) (void)cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? QK_ERR_OOM : QK_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

template <typename C> struct FPassArgs {
    C *s, *s2;
    const TOp *ops;
    const C *coef;
    const int32_t *gparams;
    double *ggrad;
};

template <typename C, int R, int NS, int MAXT, int MINB>
static int launch_k(const FPassArgs<C> &a, int n, const PassDesc &d, uint32_t threads, cudaStream_t st) {
    static std::atomic<uint64_t> smem_done{0};
    const auto kernel = k_fpass<C, R, NS, MAXT, MINB>;
    // (64 bytes: steps and coefficients are read ahead)
    const size_t smem = (d.last ? (sizeof(C) << d.T) * NS : 0) + d.nprog * sizeof(TOp) + d.ncoef * sizeof(C) +
                        (NS == 2 ? d.ngrad * sizeof(double) * threads : 0) + 64;
    if (smem > (220u << 10)) return fail(QK_ERR_ARG, "pass needs %zu bytes of shared memory", smem);
    cudaError_t e = smem_limit_once(smem_done, (const void *)kernel, 220 << 10);
    if (e != cudaSuccess) return cuda_err(e, "cudaFuncSetAttribute(k_fpass)");
    int mb = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&mb, kernel, (int)threads, smem);
    if (e != cudaSuccess || mb < 1) mb = 1;
    const uint32_t ntiles = 1u << (n - d.T);
    const unsigned grid = (unsigned)std::min<uint64_t>(ntiles, (uint64_t)device_sms() * mb);
    kernel<<<grid, threads, smem, st>>>(a.s, a.s2, ntiles, d, a.ops, a.coef, a.gparams, a.ggrad);
    e = cudaGetLastError();
    return e == cudaSuccess ? QK_OK : cuda_err(e, "k_fpass launch");
}

// Up to 128 threads, the instances whose register amplitudes take 128 bytes
// or more are held to 16 (complex64 with 16 a thread 20, two states 12) warps
// an SM: with the registers of one CTA more (complex128, 96 a thread: 65 ms)
// or less (complex64, 168: 80 against 75 ms) the brick circuits run no faster.
template <typename C, int R, int NS>
static int launch_r(const FPassArgs<C> &a, int n, const PassDesc &d, cudaStream_t st) {
    constexpr int bytes = (int)sizeof(C) * R * NS;
    const uint32_t threads = (1u << d.T) / R;
    if (threads > (uint32_t)pass_max_threads<C, R, NS>() || threads == 0)
        return fail(QK_ERR_ARG, "pass of %d tile bits needs %u threads", d.T, threads);
    if constexpr (bytes >= 128)
        if (threads <= 128)
            return launch_k<C, R, NS, 128, NS == 2 ? 3 : bytes == 128 && R == 16 ? 5 : 4>(a, n, d, threads, st);
    return launch_k<C, R, NS, pass_max_threads<C, R, NS>(), 1>(a, n, d, threads, st);
}

template <typename C>
static int launch(const FPassArgs<C> &a, int n, int r, const PassDesc &d, cudaStream_t st) {
    if (!a.ops || (d.ncoef && !a.coef)) return fail(QK_ERR_ARG, "compute pass without its program in device memory");
    if (a.s2) {   // complex128 only: complex64 sweeps run the general programs
        if constexpr (sizeof(C) == sizeof(double2)) {
            switch (r) {
            case 1: return launch_r<C, 2, 2>(a, n, d, st);
            case 2: return launch_r<C, 4, 2>(a, n, d, st);
            case 3: return launch_r<C, 8, 2>(a, n, d, st);
            }
        }
        return fail(QK_ERR_ARG, "reg_bits %d unsupported for two-state passes", r);
    }
    switch (r) {
    case 1: return launch_r<C, 2, 1>(a, n, d, st);
    case 2: return launch_r<C, 4, 1>(a, n, d, st);
    case 3: return launch_r<C, 8, 1>(a, n, d, st);
    case 4: return launch_r<C, 16, 1>(a, n, d, st);
    case 5:
        if constexpr (sizeof(C) == sizeof(float2)) return launch_r<C, 32, 1>(a, n, d, st);
        break;
    }
    return fail(QK_ERR_ARG, "reg_bits %d unsupported", r);
}

int launch_factored_pass(double2 *s, double2 *s2, int n, int r, const PassDesc &d, const TOp *ops, const double2 *coef,
                         const int32_t *gparams, double *ggrad, cudaStream_t st) {
    return launch(FPassArgs<double2>{s, s2, ops, coef, gparams, ggrad}, n, r, d, st);
}
int launch_factored_pass(float2 *s, float2 *s2, int n, int r, const PassDesc &d, const TOp *ops, const float2 *coef,
                         const int32_t *gparams, double *ggrad, cudaStream_t st) {
    return launch(FPassArgs<float2>{s, s2, ops, coef, gparams, ggrad}, n, r, d, st);
}

}  // namespace qk
