// Device-resident mixed-precision Lanczos: one step = two or three kernels that read
// the step index, the vector pointers and the recurrence scalars from device
// memory, so the step is captured once as a CUDA graph and replayed.
//
// Stored vectors.  v_k = sig[k] * V_k with V_0 the normalised start vector and
// V_{k+1} = w_k (the un-normalised residual of step k), sig[k+1] = 1 / beta_k.
// The SpMV multiplies its output by sig[k], so y = H v_k and every stored
// vector has norm beta_{k-1}: no growth, no separate normalisation pass.
//   1. SpMV (fast kernel, Lanczos mode): V_{k+1} = sig_k H V_k - beta_{k-1}
//      sig_{k-1} V_{k-1} (the previous-vector term applied as each row is
//      written), plus per-block partials of Re<V_k, V_{k+1}>  =>  alpha_k =
//      sig_k * sum = <v_k, H v_k - beta_{k-1} v_{k-1}> (the modified
//      Gram-Schmidt order of Paige's Lanczos variant: equal to <v_k, H v_k> in
//      exact arithmetic, one pass over a vector fewer per step).
//      The last CTA adds the partials and sets alpha_k and a = alpha_k sig_k (a
//      kernel of its own, lz_alpha, where the grid is large).
//   2. lz_update: V_{k+1} -= a V_k; compensated |V_{k+1}|^2, and the projections on
//      the Ritz vectors held; the last CTA sets beta_k, sig_{k+1} and k += 1.
//   3. lz_orth, with Ritz vectors held: the correction along them where the
//      projections ask for it, and beta_k from the corrected vector.
// alpha/beta are also written to mapped pinned host memory; the host reads
// them a few steps behind the GPU (convergence test, selective
// reorthogonalisation trigger) without stalling the stream.
#include "fast_common.cuh"
#include "pair.cuh"
#include "solvers.hpp"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <type_traits>

namespace qkg {
using namespace fastk;
using namespace pairk;

namespace {
constexpr int kT = 256;
constexpr int kUpdGrid = 152 * 8;
// CTAs of the FP32 update and correction: each ends in block sums, a fence and an atomic, so
// fewer of them with more bytes in flight each (100 steps at L = 24: 8 CTAs an SM and 16-byte
// accesses 8.91 ms, 32-byte accesses 8.98, with 4 CTAs an SM 8.63, with 2 8.73).
constexpr int kUpdGrid32 = 152 * 4;
constexpr int kTimedSteps = 8;  // steps launched one by one with an SpMV timer before the graph takes over
constexpr int kInFlight = 6;    // steps the host lets the GPU run ahead of its checks
constexpr double kOrthTol = 3.4526698300124393e-4;  // sqrt(2^-23): FP32 semiorthogonality level

constexpr int kMaxPsi = kMaxRitzLocked;  // converged Ritz vectors held for selective reorthogonalisation
static_assert(kMaxPsi <= kMaxLzRitz, "the step's state holds a projection for every Ritz vector");

struct PsiTab {
    const float2* p[kMaxPsi];
};

// alpha from the SpMV's per-CTA partials where its grid is too large for its last
// CTA to add them: blocks sum fixed slices, the last one to finish adds their sums in
// block order; the result does not depend on which block that is.
constexpr int kAlphaBlocks = 64, kAlphaThreads = 1024;
// SpMV grids up to this add their own partials: every CTA then passes a fence and an
// atomic, 4 us on 380 CTAs (L = 18, FP64) where the kernel of its own takes 7, but 7 us on
// 1,700 (L = 20) and 15 us on 5,400 (L = 24, FP32).
constexpr int kFusedParts = 1024;
// One block for up to eight partials a thread.
inline int alpha_blocks(int nparts) { return nparts <= 8 * kAlphaThreads ? 1 : kAlphaBlocks; }
__global__ void __launch_bounds__(kAlphaThreads) lz_alpha_kernel(const double2* __restrict__ apart, int nparts, const LzDev d, double2* part2) {
    double s = 0.0;
#pragma unroll 8
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nparts; i += gridDim.x * blockDim.x) s += apart[i].x;
    s = block_sum_d(s);
    if (gridDim.x == 1) {
        if (threadIdx.x == 0) lz_set_alpha(d, s);
        return;
    }
    if (threadIdx.x == 0) part2[blockIdx.x] = make_double2(s, 0.0);
    if (!last_cta(d.arrived)) return;
    const double t = sum_partials(part2, gridDim.x);
    if (threadIdx.x == 0) lz_set_alpha(d, t);
}

// Four elements of the update w -= a v with its ||w||^2 (and, with NP Ritz vectors psi_p,
// the <psi_p, w>) contributions: compensated sums of (re, im) pairs.
template <int NP>
struct UpdAcc {
    static constexpr int NQ = NP > 0 ? NP : 1;
    u64 hi = 0, lo = 0;                                   // Re^2, Im^2 of w
    u64 rh[NQ] = {}, rl[NQ] = {}, ih[NQ] = {}, il[NQ] = {};  // the two products of Re and of Im <psi, w>
};
constexpr u64 kConj2 = 0x8000000000000000ull;  // the sign of the imaginary part
template <int NP>
__device__ __forceinline__ void upd_elem(u64& x, u64 c, u64 a2, UpdAcc<NP>& s) {
    x = fma2(a2, c, x);
    acc2(s.hi, s.lo, x, x);
}
template <int NP>
__device__ __forceinline__ void upd_psi(u64 x, u64 p, int q, UpdAcc<NP>& s) {
    const float2 f = unpk(x);
    acc2(s.rh[q], s.rl[q], p, x);
    acc2(s.ih[q], s.il[q], p ^ kConj2, pk(f.y, f.x));
}
// the two halves of a compensated pair sum added
__device__ __forceinline__ double halves(u64 hi, u64 lo) {
    const float2 h = unpk(hi), l = unpk(lo);
    float a = h.x, b = l.x;
    ff_add(a, b, h.y, l.y);
    return (double)a + (double)b;
}
// CTA sums of M values a thread, in double and in a fixed order, valid in thread 0: the values
// go through shared memory and a warp takes one of them, eight additions a lane and a tree, so
// that GB300's narrow FP64 pipe sees 13 additions a value and CTA where shuffles in every warp
// would take 45.  About as fast as float pairs throughout (100 steps at L = 24, median of ten
// processes 8.33 and 8.31 ms, 60 at L = 28 54.9 and 54.9, 100 at L = 18 3.30 and 3.30) without
// their 48 bits; a thread's own sums are brought to one pair in FP32 first (two conversions a
// value and not four: 0.2 ms at L = 24).
template <int M>
__device__ __forceinline__ void block_sums_d(double (&v)[M]) {
    __shared__ double red[M][kT], sum[M];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int m = 0; m < M; ++m) red[m][threadIdx.x] = v[m];
    __syncthreads();
    for (int m = threadIdx.x >> 5; m < M; m += kT / 32) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < kT / 32; ++i) s += red[m][lane + 32 * i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) sum[m] = s;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = sum[m];
}
struct Four {
    u64 v[4];
    __device__ __forceinline__ explicit Four(const float2* p) {
        asm("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
    }
    __device__ __forceinline__ void store(float2* p) const {
        asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3]) : "memory");
    }
};

// w -= a v in place (the SpMV applied the previous-vector term), ||w||^2 (and the
// <psi_q, w> of the NP Ritz vectors, for selective reorthogonalisation), and from them
// beta: four elements per thread and iteration with 32-byte accesses (the Krylov vectors
// and the Ritz vectors are 256-byte aligned).  ppart[q * gridDim.x + block] holds Ritz
// vector q's partial.
template <int NP>
__global__ void __launch_bounds__(kT) lz_update_t(const LzDev d, uint64_t n, const PsiTab psi, double orth_tol,
                                                  double2* __restrict__ bpart, double2* __restrict__ ppart) {
    const int k = d.st->k;
    float2* w = static_cast<float2*>(d.vtab[k + 1]);
    const float2* v = static_cast<const float2*>(d.vtab[k]);
    const float a = -(float)d.st->a;
    const u64 a2 = pk(a, a);
    UpdAcc<NP> s;
    const uint64_t n4 = n / 4, step = (uint64_t)gridDim.x * blockDim.x;
#pragma unroll 2
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n4; i += step) {
        Four x(w + 4 * i);
        const Four c(v + 4 * i);
#pragma unroll
        for (int e = 0; e < 4; ++e) upd_elem<NP>(x.v[e], c.v[e], a2, s);
        x.store(w + 4 * i);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const Four p(psi.p[q] + 4 * i);
#pragma unroll
            for (int e = 0; e < 4; ++e) upd_psi<NP>(x.v[e], p.v[e], q, s);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
        const uint64_t i = 4 * n4 + threadIdx.x;
        u64 x = reinterpret_cast<const u64*>(w)[i];
        upd_elem<NP>(x, reinterpret_cast<const u64*>(v)[i], a2, s);
        reinterpret_cast<u64*>(w)[i] = x;
#pragma unroll
        for (int q = 0; q < NP; ++q) upd_psi<NP>(x, reinterpret_cast<const u64*>(psi.p[q])[i], q, s);
    }
    double t[1 + 2 * NP];
    t[0] = halves(s.hi, s.lo);
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        t[1 + 2 * q] = halves(s.rh[q], s.rl[q]);
        t[2 + 2 * q] = halves(s.ih[q], s.il[q]);
    }
    block_sums_d(t);
    if (threadIdx.x == 0) {
        bpart[blockIdx.x] = make_double2(t[0], 0.0);
#pragma unroll
        for (int q = 0; q < NP; ++q) ppart[(size_t)q * gridDim.x + blockIdx.x] = make_double2(t[1 + 2 * q], t[2 + 2 * q]);
    }
    if (!last_cta(d.arrived)) return;
    // the last CTA: ||w||^2, c_q = <psi_q, w>.  The correction is applied only when
    // some |c_q| exceeds orth_tol ||w|| (components below the square root of the working
    // precision are harmless, Parlett & Scott 1979), so most steps skip the extra pass.
    const double w2 = sum_partials(bpart, gridDim.x);
    int orth = 0;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        double r = 0.0, m = 0.0;
        for (int j = threadIdx.x; j < gridDim.x; j += blockDim.x) {
            const double2 e = __ldcg(ppart + (size_t)q * gridDim.x + j);
            r += e.x;
            m += e.y;
        }
        r = block_sum_d(r);
        m = block_sum_d(m);
        if (threadIdx.x == 0) {
            d.st->pre[q] = r;
            d.st->pim[q] = m;
            orth |= r * r + m * m > orth_tol * orth_tol * w2 ? 1 : 0;
        }
    }
    if (threadIdx.x == 0) {
        d.st->orth = orth;
        if (!orth) lz_set_beta(d, k, w2);  // else after the correction
    }
}

// W -= sum_q c_q psi_q with c_q = <psi_q, W>, then beta from the corrected W.
template <int NP>
__global__ void __launch_bounds__(kT) lz_orth_kernel(const LzDev d, const PsiTab psi, uint64_t n, double2* __restrict__ bpart) {
    if (!d.st->orth) return;
    const int k = d.st->k;
    float2* w = static_cast<float2*>(d.vtab[k + 1]);
    u64 cr[NP], ci[NP];  // -(c, c) and (im c, -im c)
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const float r = (float)d.st->pre[q], m = (float)d.st->pim[q];
        cr[q] = pk(-r, -r);
        ci[q] = pk(m, -m);
    }
    auto take = [&](u64 x, u64 p, int q) {
        const float2 f = unpk(p);
        return fma2(ci[q], pk(f.y, f.x), fma2(cr[q], p, x));
    };
    u64 h2 = 0, l2 = 0;
    const uint64_t n4 = n / 4;
#pragma unroll 2
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n4; i += (uint64_t)gridDim.x * blockDim.x) {
        Four x(w + 4 * i);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const Four p(psi.p[q] + 4 * i);
#pragma unroll
            for (int e = 0; e < 4; ++e) x.v[e] = take(x.v[e], p.v[e], q);
        }
        x.store(w + 4 * i);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc2(h2, l2, x.v[e], x.v[e]);
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
        const uint64_t i = 4 * n4 + threadIdx.x;
        u64 x = reinterpret_cast<const u64*>(w)[i];
#pragma unroll
        for (int q = 0; q < NP; ++q) x = take(x, reinterpret_cast<const u64*>(psi.p[q])[i], q);
        reinterpret_cast<u64*>(w)[i] = x;
        acc2(h2, l2, x, x);
    }
    double s[1] = {halves(h2, l2)};
    block_sums_d(s);
    if (threadIdx.x == 0) bpart[blockIdx.x] = make_double2(s[0], 0.0);
    if (!last_cta(d.arrived)) return;
    const double w2 = sum_partials(bpart, gridDim.x);
    if (threadIdx.x == 0) {
        d.st->orth = 0;
        lz_set_beta(d, k, w2);
    }
}

// ---- FP64 ---------------------------------------------------------------------
// Per-CTA partials of ||w||^2; the last CTA adds them and sets beta_k.
__device__ __forceinline__ void finish_beta(const LzDev& d, int k, double acc, double2* bpart) {
    const double t = block_sum_d(acc);
    if (threadIdx.x == 0) bpart[blockIdx.x] = make_double2(t, 0.0);
    if (!last_cta(d.arrived)) return;
    const double w2 = sum_partials(bpart, gridDim.x);
    if (threadIdx.x == 0) lz_set_beta(d, k, w2);
}
// w -= a v in place, and beta.
// FULL: a reorthogonalisation follows, which sets beta.
template <bool FULL>
__global__ void __launch_bounds__(kT) lz64_update(const LzDev d, uint64_t n, double2* __restrict__ bpart) {
    const int k = d.st->k;
    double2* __restrict__ w = static_cast<double2*>(d.vtab[k + 1]);
    const double2* __restrict__ v = static_cast<const double2*>(d.vtab[k]);
    const double a = -d.st->a;
    double acc = 0.0;
#pragma unroll 4
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double2 x = w[i];
        const double2 c = v[i];
        x.x = fma(a, c.x, x.x);
        x.y = fma(a, c.y, x.y);
        w[i] = x;
        if (!FULL) acc = fma(x.y, x.y, fma(x.x, x.x, acc));
    }
    if (!FULL) finish_beta(d, k, acc, bpart);
}
// y = scale y - bprev vprev and Re<x, y> partials, for an SpMV that does not do it.
__global__ void lz64_post(const LzOperands* __restrict__ op, uint64_t n, double2* __restrict__ apart) {
    const LzOperands o = *op;
    const double2* __restrict__ x = static_cast<const double2*>(o.x);
    const double2* __restrict__ p = static_cast<const double2*>(o.vprev);
    double2* __restrict__ y = static_cast<double2*>(o.y);
    double acc = 0.0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double2 w = y[i];
        const double2 c = x[i];
        w.x *= o.scale;
        w.y *= o.scale;
        if (p) {
            const double2 d = p[i];
            w.x = fma(-o.bprev, d.x, w.x);
            w.y = fma(-o.bprev, d.y, w.y);
        }
        y[i] = w;
        acc = fma(c.y, w.y, fma(c.x, w.x, acc));
    }
    acc = block_sum_d(acc);
    if (threadIdx.x == 0) apart[blockIdx.x] = make_double2(acc, 0.0);
}
// coef_j = -sig_j^2 <V_j, w> from the projections' partials (column j at part[j * nparts]).
__global__ void lz64_coef(const double2* __restrict__ part, int nparts, const double* __restrict__ sig,
                          double2* __restrict__ coef) {
    const int j = blockIdx.x;
    double re = 0.0, im = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        const double2 v = part[(size_t)j * nparts + i];
        re += v.x;
        im += v.y;
    }
    re = block_sum_d(re);
    im = block_sum_d(im);
    if (threadIdx.x == 0) {
        const double f = -sig[j] * sig[j];
        coef[j] = make_double2(f * re, f * im);
    }
}
// w += sum_j coef_j V_j for the k vectors from j0 (w = V_kw); the launch that reaches
// V_{kw-1} also sets beta_{kw-1}.  Coefficients and pointers take 24 bytes of shared
// memory a vector: kSubtractMost of them a launch keep to 24 KB.
constexpr int kSubtractMost = 1024;
// vectors a run reorthogonalises against
constexpr int kMaxBasis = 4096;
__global__ void __launch_bounds__(kT) lz64_subtract(const LzDev d, int kw, int j0, int k, const double2* __restrict__ coef,
                                                    uint64_t n, double2* __restrict__ bpart) {
    void* const* vtab = d.vtab;
    extern __shared__ double2 s_c[];
    const double2** s_v = reinterpret_cast<const double2**>(s_c + k);
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
        s_c[j] = coef[j0 + j];
        s_v[j] = static_cast<const double2*>(vtab[j0 + j]);
    }
    __syncthreads();
    double2* __restrict__ w = static_cast<double2*>(vtab[kw]);
    double acc = 0.0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double2 x = w[i];
        int j = 0;
        for (; j + 4 <= k; j += 4) {  // four vectors' loads in flight
            double2 a[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) a[q] = s_v[j + q][i];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 c = s_c[j + q];
                x.x = fma(c.x, a[q].x, fma(-c.y, a[q].y, x.x));
                x.y = fma(c.x, a[q].y, fma(c.y, a[q].x, x.y));
            }
        }
        for (; j < k; ++j) {
            const double2 a = s_v[j][i], c = s_c[j];
            x.x = fma(c.x, a.x, fma(-c.y, a.y, x.x));
            x.y = fma(c.x, a.y, fma(c.y, a.x, x.y));
        }
        w[i] = x;
        acc = fma(x.y, x.y, fma(x.x, x.x, acc));
    }
    if (j0 + k == kw) finish_beta(d, kw - 1, acc, bpart);
}

using clk = std::chrono::steady_clock;
inline double secs(clk::time_point a, clk::time_point b) { return std::chrono::duration<double>(b - a).count(); }

struct Mapped {
    double* h = nullptr;
    double* d = nullptr;
    explicit Mapped(size_t n) {
        QKG_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&h), n * sizeof(double), cudaHostAllocMapped));
        QKG_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&d), h, 0));
        std::fill(h, h + n, 0.0);
    }
    ~Mapped() { if (h) cudaFreeHost(h); }
};
}  // namespace

bool lanczos_device_supported(const Hamiltonian& H) { return H.fast(); }

// Device memory of a device-resident run of maxiter steps: maxiter + 1 Krylov
// vectors, then kMaxPsi Ritz vectors psi (FP32), the Ritz vector (FP32), the
// refined Ritz vector and its residual (FP64), each vector on a 256-byte
// boundary.  The FP64 slots also stage a caller's start vector, the first two
// psi slots the reference-order copy of the eigenvector.
size_t lanczos_device_bytes(const Hamiltonian& H, int maxiter) {
    const uint64_t n = H.dim();
    const int nmax = (int)std::min<uint64_t>((uint64_t)std::max(maxiter, 0), n);
    const uint64_t stride = (n + 31) / 32 * 32;
    return (size_t)(nmax + 1 + kMaxPsi + 5) * stride * sizeof(float2);
}

LanczosOut lanczos_mixed_device(Hamiltonian& H, const LanczosOpts& o) {
    LanczosOut out;
    const uint64_t n = H.dim();
    if (n == 0) return out;
    const auto ws_lock = H.workspace_lock();
    cudaStream_t st = H.stream();
    const int nmax = (int)std::min<uint64_t>((uint64_t)std::max(o.maxiter, 0), n);
    if (nmax <= 0) return out;
    // all nmax + 1 Krylov vectors (FP32) up front: the graph addresses them through vtab
    // vectors start on 256-byte boundaries (a warp's 32 consecutive rows then
    // cover whole 128-byte lines)
    const uint64_t stride = (n + 31) / 32 * 32;
    const size_t need = lanczos_device_bytes(H, o.maxiter);
    if (H.krylov_workspace_bytes() < need) {
        H.release_workspace();  // with the FP64 vectors, which the new space need not fit beside
        size_t fr = 0, tot = 0;
        QKG_CUDA(cudaMemGetInfo(&fr, &tot));
        if (need + (512ull << 20) > fr)
            throw Error(CUDA_ERR, "out of device memory for " + std::to_string(nmax + 1) + " Krylov vectors");
    }
    // one allocation for all vectors (a cudaMalloc per vector costs more than a
    // step), kept on the Hamiltonian for the next run
    const DBuf& V = H.krylov_workspace(need);
    std::vector<void*> vptr;
    for (int i = 0; i <= nmax; ++i) vptr.push_back(V.as<float2>() + (size_t)i * stride);
    float2* const psi_p = V.as<float2>() + (size_t)(nmax + 1) * stride;
    float2* const r32_p = psi_p + (size_t)kMaxPsi * stride;
    double2* const r64_p = reinterpret_cast<double2*>(r32_p + stride);
    double2* const h64_p = r64_p + stride;
    DBuf vtab((nmax + 1) * sizeof(void*));
    QKG_CUDA(cudaMemcpy(vtab.p, vptr.data(), vptr.size() * sizeof(void*), cudaMemcpyHostToDevice));
    DBuf state(sizeof(LzState)), alpha((nmax + 2) * 8), beta((nmax + 2) * 8), sig((nmax + 2) * 8);
    DBuf apart(std::max<size_t>(1, H.lanczos_parts()) * sizeof(double2)), bpart(kUpdGrid * sizeof(double2)),
        ppart((size_t)kMaxPsi * kUpdGrid * sizeof(double2)), psitab(kMaxPsi * sizeof(float2*));
    Mapped ah(nmax + 2), bh(nmax + 2);
    DBuf part2(kAlphaBlocks * sizeof(double2)), arrived(sizeof(unsigned int));
    QKG_CUDA(cudaMemsetAsync(arrived.p, 0, sizeof(unsigned int), st));
    Workspace ws(std::max<size_t>(1 << 16, (size_t)1216 * (size_t)(nmax + 2)));
    DBuf tmp;

    float2* v0 = static_cast<float2*>(vptr[0]);
    if (o.device_start) {
        H.philox_f32(o.seed, 0, v0, st);
    } else {
        // the caller's vector is copied straight from its buffer (pinned memory takes the DMA path)
        std::vector<cd> h;
        const cd* src = o.v0_ref;
        if (!src) {
            h.resize(n);
            ref_uniform_complex(1234, n, h.data(), o.f32_stream);
            src = h.data();
        }
        QKG_CUDA(cudaMemcpyAsync(r64_p, src, n * sizeof(double2), cudaMemcpyHostToDevice, st));
        const double2* in = r64_p;
        if (H.permuted()) {
            H.to_internal_f64(r64_p, h64_p, st);
            in = h64_p;
        }
        f64_to_f32(in, v0, n, st);
        QKG_CUDA(cudaStreamSynchronize(st));
    }
    const double nr0 = std::sqrt(nrm2sq_f32(v0, n, ws, st));
    if (nr0 != 0.0) scal_f32(1.0 / nr0, v0, n, st);
    DBuf lzop(sizeof(LzOperands));
    {
        LzState s0{};
        const double one = 1.0;
        LzOperands op0;  // step 0: y = H v_0, no previous vector
        op0.x = vptr[0];
        op0.y = vptr[1];
        QKG_CUDA(cudaMemcpyAsync(state.p, &s0, sizeof(s0), cudaMemcpyHostToDevice, st));
        QKG_CUDA(cudaMemcpyAsync(sig.p, &one, sizeof(one), cudaMemcpyHostToDevice, st));
        QKG_CUDA(cudaMemcpyAsync(lzop.p, &op0, sizeof(op0), cudaMemcpyHostToDevice, st));
        QKG_CUDA(cudaStreamSynchronize(st));
    }

    LzDev dev;
    dev.st = state.as<LzState>();
    dev.alpha = alpha.as<double>();
    dev.beta = beta.as<double>();
    dev.sig = sig.as<double>();
    dev.alpha_host = ah.d;
    dev.beta_host = bh.d;
    dev.vtab = static_cast<void* const*>(vtab.p);
    dev.nmax = nmax;
    dev.op = lzop.as<LzOperands>();
    dev.arrived = arrived.as<unsigned int>();
    LanczosHooks hooks;
    hooks.op = lzop.as<LzOperands>();
    hooks.apart = apart.as<double2>();
    const int nparts = (int)H.lanczos_parts();
    const bool own_alpha = H.packed() && nparts <= kFusedParts;
    if (own_alpha) hooks.fin = dev;
    // CTAs of the update: four 16-byte elements a thread at least, up to a resident wave
    const int ug = (int)std::max<uint64_t>(1, std::min<uint64_t>(n / (8 * kT), kUpdGrid32));
    PsiTab psi{};   // converged Ritz vectors (selective reorthogonalisation)
    int npsi = 0;   // how many are held
    std::vector<double> locked;  // their Ritz values
    auto enqueue_step = [&](int np, LaunchTimer* timer) {
        if (timer) timer->start();
        H.apply_lanczos_f32(hooks, st);
        if (timer) timer->stop();
        if (!own_alpha) {
            lz_alpha_kernel<<<alpha_blocks(nparts), kAlphaThreads, 0, st>>>(apart.as<double2>(), nparts, dev, part2.as<double2>());
            QKG_LAUNCHED();
        }
        auto sel = [&](auto npc) {
            constexpr int NP = decltype(npc)::value;
            lz_update_t<NP><<<ug, kT, 0, st>>>(dev, n, psi, kOrthTol, bpart.as<double2>(), ppart.as<double2>());
            QKG_LAUNCHED();
            if constexpr (NP > 0) {
                lz_orth_kernel<NP><<<ug, kT, 0, st>>>(dev, psi, n, bpart.as<double2>());
                QKG_LAUNCHED();
            }
        };
        switch (np) {
            case 0: sel(std::integral_constant<int, 0>{}); break;
            case 1: sel(std::integral_constant<int, 1>{}); break;
            case 2: sel(std::integral_constant<int, 2>{}); break;
            case 3: sel(std::integral_constant<int, 3>{}); break;
            default: sel(std::integral_constant<int, 4>{}); break;
        }
    };
    int kernels[kMaxPsi + 1] = {};  // kernels per step graph (by Ritz vectors held), counted at capture
    auto capture = [&](int np) {
        cudaGraph_t g = nullptr;
        cudaGraphExec_t ge = nullptr;
        const uint64_t c0 = launch_count();
        QKG_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        enqueue_step(np, nullptr);
        QKG_CUDA(cudaStreamEndCapture(st, &g));
        const int64_t captured = (int64_t)(launch_count() - c0);
        add_launches(-captured);
        kernels[np] = (int)captured;  // kernels per replay
        QKG_CUDA(cudaGraphInstantiate(&ge, g, 0));
        QKG_CUDA(cudaGraphDestroy(g));
        return ge;
    };
    cudaGraphExec_t graphs[kMaxPsi + 1] = {};
    auto destroy_graphs = [&] {
        for (auto& g : graphs)
            if (g) {
                cudaGraphExecDestroy(g);
                g = nullptr;
            }
    };
    std::vector<cudaEvent_t> ev(kInFlight + 2);
    for (auto& e : ev) QKG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));

    int stop_at = -1;       // last accepted step (inclusive)
    bool converged = false;
    double e_old = 1e100;
    const double so_tol = 3.5e-4;
    LaunchTimer timer(st);
    int launched = 0, checked = 0;
    const auto t0 = clk::now();
    try {
        auto check_step = [&](int j) {  // step j has completed
            const double b = bh.h[j];
            if (b < 1e-15) { converged = true; stop_at = j; return; }
            if (j + 1 == nmax) { stop_at = j; return; }
            if (j > 0) {
                std::vector<double> a(ah.h, ah.h + j + 1), bb(bh.h, bh.h + j);
                const double e = tridiag_lowest(a.data(), bb.data(), j + 1);
                if (!o.fixed_steps && std::abs(e - e_old) < o.tol) { converged = true; stop_at = j; return; }
                e_old = e;
                if (j + 1 >= 4) {
                    // Parlett-Scott: lock the Ritz vectors of newly converged low Ritz values
                    for (double theta : ritz_to_lock(a.data(), bb.data(), j + 1, b, so_tol, locked, o.ritz_guard)) {
                        if (npsi >= kMaxPsi) break;
                        std::vector<double> s;
                        if (!tridiag_vector(a.data(), bb.data(), j + 1, theta, s)) continue;
                        // Ritz vector of T_j from v_0..v_j = sig_i V_i (sig_0 = 1, sig_{i+1} = 1/beta_i)
                        std::vector<cd> c(j + 1);
                        double sg = 1.0;
                        for (int i = 0; i <= j; ++i) {
                            c[i] = s[i] * sg;
                            sg = 1.0 / bh.h[i];
                        }
                        float2* p = psi_p + (size_t)npsi * stride;
                        QKG_CUDA(cudaMemsetAsync(p, 0, n * sizeof(float2), st));
                        mcombine_f32(reinterpret_cast<const float2* const*>(vtab.p), j + 1, c.data(), p, n, ws, st);
                        double pn = std::sqrt(nrm2sq_f32(p, n, ws, st));
                        if (!(pn > 0.0)) continue;
                        scal_f32(1.0 / pn, p, n, st);
                        if (npsi > 0) {  // orthonormal to the Ritz vectors already held (two passes)
                            const auto* pt = static_cast<const float2* const*>(psitab.p);
                            for (int pass = 0; pass < 2; ++pass) {
                                std::vector<cd> h(npsi);
                                mdot_f32(pt, npsi, p, n, h.data(), ws, st);
                                for (auto& x : h) x = -x;
                                mcombine_f32(pt, npsi, h.data(), p, n, ws, st);
                            }
                            pn = std::sqrt(nrm2sq_f32(p, n, ws, st));
                            if (pn < 0.5) continue;  // in the span of those held: the same Ritz value again
                            scal_f32(1.0 / pn, p, n, st);
                        }
                        psi.p[npsi++] = p;
                        QKG_CUDA(cudaMemcpyAsync(psitab.p, psi.p, sizeof(psi.p), cudaMemcpyHostToDevice, st));
                        locked.push_back(theta);
                    }
                }
            }
        };
        while (launched < nmax && stop_at < 0) {
            if (launched < kTimedSteps) {
                enqueue_step(npsi, &timer);
                out.t_spmv += timer.collect();  // waits for this SpMV only
                ++out.n_spmv;
            } else {
                cudaGraphExec_t& g = graphs[npsi];
                if (!g) g = capture(npsi);
                QKG_CUDA(cudaGraphLaunch(g, st));
                for (int q = 0; q < kernels[npsi]; ++q) count_launch();
            }
            if (npsi) ++out.n_selective;
            QKG_CUDA(cudaEventRecord(ev[launched % ev.size()], st));
            ++launched;
            while (checked < launched && stop_at < 0) {
                cudaEvent_t e = ev[checked % ev.size()];
                if (launched - checked < kInFlight) {
                    const cudaError_t q = cudaEventQuery(e);
                    if (q == cudaErrorNotReady) break;
                    QKG_CUDA(q);
                } else {
                    QKG_CUDA(cudaEventSynchronize(e));
                }
                check_step(checked);
                ++checked;
            }
        }
        QKG_CUDA(cudaStreamSynchronize(st));
        while (stop_at < 0 && checked < launched) check_step(checked++);
    } catch (...) {
        cudaStreamSynchronize(st);
        for (auto& e : ev) cudaEventDestroy(e);
        destroy_graphs();
        throw;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    destroy_graphs();
    out.n_ritz_locked = npsi;
    out.t_loop = secs(t0, clk::now());
    if (stop_at < 0) stop_at = launched - 1;
    out.iters = stop_at + 1;
    out.converged = converged;
    out.alphas.assign(ah.h, ah.h + stop_at + 1);
    out.betas.assign(bh.h, bh.h + stop_at);  // the last step's beta is not part of T

    // Ritz vector from the FP32 basis, then FP64 Rayleigh quotient and residual.
    const auto t1 = clk::now();
    std::vector<double> s;
    out.energy_tridiag = tridiag_ground(out.alphas.data(), out.betas.data(), (int)out.alphas.size(), s);
    std::vector<cd> c(s.size());
    double sg = 1.0;
    for (size_t i = 0; i < s.size(); ++i) {
        c[i] = s[i] * sg;
        sg = 1.0 / bh.h[i];
    }
    QKG_CUDA(cudaMemsetAsync(r32_p, 0, n * sizeof(float2), st));
    mcombine_f32(reinterpret_cast<const float2* const*>(vtab.p), (int)c.size(), c.data(), r32_p, n, ws, st);
    f32_to_f64(r32_p, r64_p, n, st);
    const double nr = std::sqrt(nrm2sq_f64(r64_p, n, ws, st));
    scal_f64(1.0 / nr, r64_p, n, st);
    H.apply_f64(r64_p, h64_p, st);
    const double E = dot_f64(r64_p, h64_p, n, ws, st).real();
    axpy_f64(-E, r64_p, h64_p, n, st);
    out.residual = std::sqrt(nrm2sq_f64(h64_p, n, ws, st));
    out.energy = E;
    out.t_refine = secs(t1, clk::now());
    if (o.want_vec) {
        cd* dst = o.evec_out;
        if (!dst) {
            out.evec.resize(n);
            dst = out.evec.data();
        }
        const double2* src = r64_p;
        if (H.permuted()) {
            double2* t2 = reinterpret_cast<double2*>(psi_p);  // psi and the FP32 Ritz slot, no longer needed
            H.to_reference_f64(r64_p, t2, st);
            src = t2;
        }
        QKG_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(double2), cudaMemcpyDeviceToHost, st));
        QKG_CUDA(cudaStreamSynchronize(st));
    }
    return out;
}

// The FP64 recurrence with its scalars on the device: the host enqueues steps up
// to kInFlight ahead and reads alpha and beta (mapped memory) behind them, so
// nothing waits for the GPU within a step.  v_k = sig_k V_k as in the mixed form.
//   SpMV (y = sig_k H V_k - beta_{k-1} v_{k-1}, Re<V_k, y> partials), alpha,
//   update (w -= alpha v_k, and its norm), with `full` the projections of w on
//   every V_j, their coefficients and the subtraction (one classical
//   Gram-Schmidt pass, and the norm), beta.
// vec(i) gives the memory of V_i; keep(j) is called with each completed step j
// in order and says whether to go on.
namespace {
struct Recurrence64 {
    Hamiltonian& H;
    uint64_t n;
    cudaStream_t st;
    int nmax;
    bool full;
    double *ah = nullptr, *bh = nullptr;  // alpha_j, beta_j on the host
    double t_spmv = 0.0;
    int n_spmv = 0;
    Recurrence64(Hamiltonian& h, int steps, bool reorth) : H(h), n(h.dim()), st(h.stream()), nmax(steps), full(reorth) {}

    // V_0 is the start vector (its norm need not be 1: sig0 = 1 / ||V_0||)
    // slot(i): the vector slot V_i lives in
    template <class Slot, class Vec, class Keep>
    void run(double sig0, Slot&& slot, Vec&& vec, Keep&& keep) {
        const int N = nmax + 2;
        const int nparts = H.packed() ? (int)H.lanczos_parts() : kUpdGrid;
        const int g = (int)std::max<uint64_t>(1, std::min<uint64_t>((n + kT - 1) / kT, kUpdGrid));
        // device scalars: state, operands, pointers, alpha, beta, sig, coefficients, partials
        auto al = [](size_t b) { return (b + 255) / 256 * 256; };
        size_t off = 0;
        auto take = [&](size_t b) { const size_t o = off; off += al(b); return o; };
        const size_t o_st = take(sizeof(LzState)), o_op = take(sizeof(LzOperands)), o_tab = take(N * sizeof(void*)),
                     o_al = take(N * 8), o_be = take(N * 8), o_sg = take(N * 8), o_co = take((size_t)N * 16),
                     o_ap = take((size_t)nparts * 16), o_bp = take((size_t)kUpdGrid * 16), o_p2 = take(kAlphaBlocks * 16),
                     o_ar = take(sizeof(unsigned int));
        Workspace& ws = H.reduction_scratch(std::max<size_t>(1 << 16, off / sizeof(double2) + 1 + (full ? mdot_f64_most_partials(std::min(N, kMaxBasis), n) : 0)));
        char* base = ws.partial.as<char>();
        auto* state = reinterpret_cast<LzState*>(base + o_st);
        auto* op = reinterpret_cast<LzOperands*>(base + o_op);
        auto** tab = reinterpret_cast<void**>(base + o_tab);
        auto *alpha = reinterpret_cast<double*>(base + o_al), *beta = reinterpret_cast<double*>(base + o_be),
             *sig = reinterpret_cast<double*>(base + o_sg);
        auto* coef = reinterpret_cast<double2*>(base + o_co);
        auto *apart = reinterpret_cast<double2*>(base + o_ap), *bpart = reinterpret_cast<double2*>(base + o_bp);
        auto* part2 = reinterpret_cast<double2*>(base + o_p2);
        auto* arrived = reinterpret_cast<unsigned int*>(base + o_ar);
        double2* ppart = reinterpret_cast<double2*>(base + off);
        const auto m = H.mapped_scalars(2 * (size_t)N);
        ah = m.host;
        bh = m.host + N;
        // initial image: state, operands, the pointers of the vectors there are, sig_0
        std::vector<void*> ptr(N, nullptr);
        std::vector<char> image(off, 0);
        int known = 0;  // pointers the device has
        auto name_vectors = [&](int need) {  // V_0 .. V_need and those allocated with them
            int i = known;
            for (; i <= nmax && (i <= need || H.has_krylov_vector(slot(i))); ++i) ptr[i] = vec(i);
            return i;
        };
        known = name_vectors(std::min(1, nmax));
        LzOperands op0;
        op0.x = ptr[0];
        op0.y = ptr[1];
        op0.scale = sig0;
        std::memcpy(image.data() + o_op, &op0, sizeof(op0));
        std::memcpy(image.data() + o_tab, ptr.data(), (size_t)known * sizeof(void*));
        std::memcpy(image.data() + o_sg, &sig0, sizeof(double));
        QKG_CUDA(cudaMemcpyAsync(base, image.data(), image.size(), cudaMemcpyHostToDevice, st));
        LzDev d;
        d.st = state;
        d.alpha = alpha;
        d.beta = beta;
        d.sig = sig;
        d.alpha_host = m.dev;
        d.beta_host = m.dev + N;
        d.vtab = tab;
        d.nmax = nmax;
        d.op = op;
        d.arrived = arrived;
        LanczosHooks hooks;
        hooks.op = op;
        hooks.apart = apart;
        const bool own_alpha = H.packed() && nparts <= kFusedParts;
        if (own_alpha) hooks.fin = d;
        struct Events {
            std::vector<cudaEvent_t> e;
            ~Events() { for (auto x : e) if (x) cudaEventDestroy(x); }
        } done{std::vector<cudaEvent_t>(kInFlight + 2, nullptr)};
        for (auto& e : done.e) QKG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        std::vector<std::unique_ptr<LaunchTimer>> timers;
        int launched = 0, checked = 0;
        bool go = true;
        auto enqueue = [&](int k) {
            // V_{k+2}, the next step's output, joins the table before a kernel names it
            if (k + 2 <= nmax && k + 2 >= known) {
                const int from = known;
                known = name_vectors(k + 2);
                QKG_CUDA(cudaMemcpyAsync(tab + from, &ptr[from], (size_t)(known - from) * sizeof(void*), cudaMemcpyHostToDevice, st));
            }
            if (k < kTimedSteps) {
                timers.push_back(std::make_unique<LaunchTimer>(st));
                timers.back()->start();
            }
            const bool fused = H.apply_lanczos_f64(hooks, st);
            if (!fused) H.apply_f64(static_cast<const double2*>(ptr[k]), static_cast<double2*>(ptr[k + 1]), st);
            if (k < kTimedSteps) timers.back()->stop();
            if (!fused) {
                lz64_post<<<kUpdGrid, kT, 0, st>>>(op, n, apart);
                QKG_LAUNCHED();
            }
            if (!own_alpha) {
                lz_alpha_kernel<<<alpha_blocks(nparts), kAlphaThreads, 0, st>>>(apart, nparts, d, part2);
                QKG_LAUNCHED();
            }
            if (full) lz64_update<true><<<g, kT, 0, st>>>(d, n, bpart);
            else lz64_update<false><<<g, kT, 0, st>>>(d, n, bpart);
            QKG_LAUNCHED();
            if (full) {
                QKG_REQUIRE(k < kMaxBasis, "Lanczos with full reorthogonalisation: at most 4096 vectors");
                const int gm = mdot_f64_chunks(k + 1, n);
                mdot_f64_partials(reinterpret_cast<const double2* const*>(tab), k + 1, static_cast<const double2*>(ptr[k + 1]),
                                  n, ppart, gm, st);
                lz64_coef<<<k + 1, kT, 0, st>>>(ppart, gm, sig, coef);
                QKG_LAUNCHED();
                for (int j0 = 0; j0 <= k; j0 += kSubtractMost) {
                    const int kk = std::min(kSubtractMost, k + 1 - j0);
                    lz64_subtract<<<g, kT, (size_t)kk * (sizeof(double2) + sizeof(void*)), st>>>(d, k + 1, j0, kk, coef, n, bpart);
                    QKG_LAUNCHED();
                }
            }
        };
        try {
            while (launched < nmax && go) {
                enqueue(launched);
                QKG_CUDA(cudaEventRecord(done.e[launched % done.e.size()], st));
                ++launched;
                while (checked < launched && go) {
                    cudaEvent_t e = done.e[checked % done.e.size()];
                    if (launched < nmax && launched - checked < kInFlight) {
                        const cudaError_t q = cudaEventQuery(e);
                        if (q == cudaErrorNotReady) break;
                        QKG_CUDA(q);
                    } else {
                        QKG_CUDA(cudaEventSynchronize(e));
                    }
                    go = keep(checked++);
                }
            }
            QKG_CUDA(cudaStreamSynchronize(st));
        } catch (...) {
            cudaStreamSynchronize(st);  // nothing of this run is in flight when its memory is reused
            throw;
        }
        for (auto& t : timers) t_spmv += t->collect();
        n_spmv = (int)timers.size();
    }
};
}  // namespace

// src/solvers/lanczos.cpp:101-202 in FP64: full reorthogonalisation, the
// reference's start vector and stopping rules.
LanczosOut lanczos_f64_device(Hamiltonian& H, const LanczosOpts& o) {
    LanczosOut out;
    const uint64_t n = H.dim();
    if (n == 0) return out;
    const auto lock = H.workspace_lock();
    cudaStream_t st = H.stream();
    const int nmax = (int)std::min<uint64_t>((uint64_t)std::max(o.maxiter, 0), n);
    const size_t vb = n * sizeof(double2);
    auto vec = [&](int i) { return H.krylov_vector((size_t)i, vb); };
    const TrimVectors trim{H};
    double2* v0 = static_cast<double2*>(vec(0));
    double2* v1 = static_cast<double2*>(vec(1));
    if (o.device_start) {
        H.philox_f64(o.seed, 0, v0, st);
    } else {
        std::vector<cd> h;
        const cd* src = o.v0_ref;
        if (!src) {
            h.resize(n);
            ref_uniform_complex(1234, n, h.data(), o.f32_stream);  // src/solvers/lanczos.cpp:115-120
            src = h.data();
        }
        QKG_CUDA(cudaMemcpyAsync(H.permuted() ? v1 : v0, src, vb, cudaMemcpyHostToDevice, st));
        if (H.permuted()) H.to_internal_f64(v1, v0, st);
        QKG_CUDA(cudaStreamSynchronize(st));
    }
    double nr0;
    {
        Workspace& ws = H.reduction_scratch(1 << 16);
        nr0 = std::sqrt(nrm2sq_f64(v0, n, ws, st));
        if (nr0 != 0.0) scal_f64(1.0 / nr0, v0, n, st);
    }
    auto& alphas = out.alphas;
    auto& betas = out.betas;
    double e_old = 1e100;
    Recurrence64 R(H, nmax, true);
    const auto t0 = clk::now();
    R.run(1.0, [](int i) { return (size_t)i; }, vec, [&](int j) {
        alphas.push_back(R.ah[j]);
        const double b = R.bh[j];
        out.iters = j + 1;
        if (b < 1e-15) {
            out.converged = true;
            return false;
        }
        if (j + 1 == nmax) return false;
        betas.push_back(b);
        if (j > 0 && !o.fixed_steps) {
            const double e = tridiag_lowest(alphas.data(), betas.data(), j + 1);
            if (std::abs(e - e_old) < o.tol) {
                out.converged = true;
                return false;
            }
            e_old = e;
        }
        return true;
    });
    out.t_loop = secs(t0, clk::now());
    out.t_spmv = R.t_spmv;
    out.n_spmv = R.n_spmv;
    std::vector<double> s;
    out.energy = tridiag_ground(alphas.data(), betas.data(), (int)alphas.size(), s);
    out.energy_tridiag = out.energy;
    out.residual = -1.0;
    if (o.want_vec) {
        // Ritz vector into the place of the first vector past the basis used
        const int m = (int)s.size();
        std::vector<cd> c(m);
        double sg = 1.0;
        for (int i = 0; i < m; ++i) {
            c[i] = s[i] * sg;
            sg = 1.0 / R.bh[i];
        }
        Workspace& ws = H.reduction_scratch(1 << 16);
        std::vector<const double2*> p(m);
        for (int i = 0; i < m; ++i) p[i] = static_cast<const double2*>(vec(i));
        DBuf tab(std::max(1, m) * sizeof(void*));
        QKG_CUDA(cudaMemcpy(tab.p, p.data(), m * sizeof(void*), cudaMemcpyHostToDevice));
        double2* ritz = static_cast<double2*>(vec(m));
        QKG_CUDA(cudaMemsetAsync(ritz, 0, vb, st));
        mcombine_f64(static_cast<const double2* const*>(tab.p), m, c.data(), ritz, n, ws, st);
        const double nr = std::sqrt(nrm2sq_f64(ritz, n, ws, st));
        if (nr != 0.0) scal_f64(1.0 / nr, ritz, n, st);
        cd* dst = o.evec_out;
        if (!dst) {
            out.evec.resize(n);
            dst = out.evec.data();
        }
        const double2* src = ritz;
        if (H.permuted()) {
            double2* t2 = static_cast<double2*>(vec(0));
            H.to_reference_f64(ritz, t2, st);
            src = t2;
        }
        QKG_CUDA(cudaMemcpyAsync(dst, src, vb, cudaMemcpyDeviceToHost, st));
        QKG_CUDA(cudaStreamSynchronize(st));
    }
    return out;
}

// The three-term recurrence without reorthogonalisation from a reference-order
// host vector (dynamics.cpp:38-56, ftlm.cpp:36-52): alphas, betas until beta <
// 1e-15 or n_steps; returns the start vector's squared norm (below min_norm^2:
// nothing recorded).
double three_term_f64(Hamiltonian& H, const cd* v_ref, int n_steps, double min_norm, std::vector<double>& alphas,
                      std::vector<double>& betas) {
    const uint64_t n = H.dim();
    const auto lock = H.workspace_lock();
    cudaStream_t st = H.stream();
    const size_t vb = n * sizeof(double2);
    const TrimVectors trim{H};
    // three vectors in turn
    auto vec = [&](int i) { return H.krylov_vector((size_t)(i % 3), vb); };
    double2* v0 = static_cast<double2*>(vec(0));
    double2* v1 = static_cast<double2*>(vec(1));
    QKG_CUDA(cudaMemcpyAsync(H.permuted() ? v1 : v0, v_ref, vb, cudaMemcpyHostToDevice, st));
    if (H.permuted()) H.to_internal_f64(v1, v0, st);
    const double norm2 = nrm2sq_f64(v0, n, H.reduction_scratch(1 << 16), st);
    const double nr = std::sqrt(norm2);
    if (nr < min_norm || n_steps <= 0) return norm2;
    Recurrence64 R(H, n_steps, false);
    R.run(nr != 0.0 ? 1.0 / nr : 1.0, [](int i) { return (size_t)(i % 3); }, vec, [&](int j) {
        alphas.push_back(R.ah[j]);
        if (R.bh[j] < 1e-15) return false;
        betas.push_back(R.bh[j]);
        return true;
    });
    return norm2;
}

}  // namespace qkg
