// Block SpMV on the packed plan (pack.hpp): y = diag(scale) H x for Rp
// interleaved vectors of several Hamiltonians in one launch.
//
// A CTA takes a run of the plan's 128-row tiles.  G lanes share a row; lane l
// holds the row's units l, l + G, ... (16 bytes: two FP32 vectors or one FP64; at
// four FP32 vectors a lane one unit of 32 bytes, loaded by one instruction), so
// that the G lanes of a row read consecutive units: whole sectors and whole
// 128-byte lines a load instruction.  A row's index work (its quads, its ranks) is
// shared by its Rp values.
//
// What bounds it (FP32, 32 vectors): the L1 data pipe and issue (246 us a launch on
// the 2^20 rows of a Heisenberg ring of 20 sites, every sector; 119 us at 12
// vectors).  Taken one after the other at 32 / 12 vectors: 310 / 154 us before, the
// sums in shared memory and not in spilled registers 262 / 140, rests of the outer
// list as shorter batches and the row's own values last 253 / 139, 32-byte accesses
// 246 / 119.
#pragma once

#include "pack.hpp"
#include "pair.cuh"

namespace qkg {
namespace blockk {
using namespace fastk;
using namespace packk;
using namespace pairk;

constexpr int kBT = 256;       // threads of a CTA
constexpr int kBatch = 3;      // outer entries loaded together
constexpr int kStrBatch = 2;   // straddling entries loaded together (the FP64 form takes its two by name)
static_assert(kStrBatch == 2);
template <int N> struct Int { static constexpr int value = N; };
constexpr int kMaxRun = 8;     // tiles of a CTA
constexpr int kMaxList = 96;   // outer (and straddling) entries of its blocks staged in shared memory

// One Hamiltonian of the batch: its rows [base, base + dim) of the block vector,
// its CTAs' range in the SpMV grid (runs of `run` tiles) and in the row grid
// (chunks of `chunk` rows).
struct Ham {
    uint64_t base, dim;
    uint32_t cta0, row_cta0;
    const uint32_t* perm;  // reference index of each internal row (null: the same)
};
// The vectors' scalars on the device.
struct BState {
    double *c_cur, *c_prev, *beta_prev, *ca, *cb, *norm2;
    double *alpha, *beta;  // [k * V + vid]
    int *active, *n_alpha, *n_beta, *kstep;
    int V, Rp, Ruser;
};
enum { FIN_INIT = 0, FIN_ALPHA = 1, FIN_BETA = 2 };

// The bookkeeping of vector vid from its sum: the norm of the start vector, step k's
// alpha or its beta.
__device__ __forceinline__ void finish_vector(const BState& st, int vid, double acc, int mode, int k) {
    if (mode == FIN_INIT) {
        st.norm2[vid] = acc;
        const double nr = sqrt(acc);
        const bool on = vid % st.Rp < st.Ruser && nr >= 1e-15;  // dynamics.cpp:27
        st.active[vid] = on;
        st.c_cur[vid] = on ? 1.0 / nr : 0.0;
        st.c_prev[vid] = 0.0;
        st.beta_prev[vid] = 0.0;
        st.n_alpha[vid] = 0;
        st.n_beta[vid] = 0;
        return;
    }
    if (mode == FIN_ALPHA) {
        if (st.active[vid]) {
            const double a = st.c_cur[vid] * acc;
            st.alpha[(size_t)k * st.V + vid] = a;
            st.n_alpha[vid] = k + 1;
            st.ca[vid] = a * st.c_cur[vid];
            st.cb[vid] = st.beta_prev[vid] * st.c_prev[vid];
        } else {
            st.ca[vid] = 0.0;
            st.cb[vid] = 0.0;
        }
        return;
    }
    if (!st.active[vid]) return;
    const double b = sqrt(acc);
    st.c_prev[vid] = st.c_cur[vid];
    if (b < 1e-15) {  // ftlm.cpp:45, dynamics.cpp:52
        st.active[vid] = 0;
        st.c_cur[vid] = 0.0;
        return;
    }
    st.beta[(size_t)k * st.V + vid] = b;
    st.n_beta[vid] = k + 1;
    st.c_cur[vid] = 1.0 / b;
    st.beta_prev[vid] = b;
}

// What the last CTA of a Hamiltonian does with its CTAs' partial sums (in the
// kernels' FUSED form; else they are left to a kernel of their own).
struct Finish {
    BState st;
    unsigned int* arrived;  // per Hamiltonian, 0 between launches
    int mode, k;
};

// the Hamiltonian whose range holds CTA c
template <class F>
__device__ __forceinline__ int find_ham(const Ham* __restrict__ hams, int n, uint32_t c, F first) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first(hams[mid]) <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// p + a * b bytes (one 32 x 32 + 64 bit multiply-add)
template <class E>
__device__ __forceinline__ const E* offset(const E* p, int a, int b) {
    return reinterpret_cast<const E*>(reinterpret_cast<const char*>(p) + (long long)a * (long long)b);
}
template <class E>
__device__ __forceinline__ E* offset(E* p, int a, int b) {
    return reinterpret_cast<E*>(reinterpret_cast<char*>(p) + (long long)a * (long long)b);
}

// A lane's values of one row: VPL complex values in units.
// FP32: pairs (re, im) packed in 64 bits.
template <class T, int VPL> struct Row;
template <int VPL> struct Row<float, VPL> {
    static constexpr int U = VPL >= 2 ? VPL / 2 : 1;  // 16-byte units (VPL = 1: half a unit)
    u64 v[VPL];
    __device__ __forceinline__ void load(const float2* p, int G) {  // p: the lane's first unit
        if constexpr (VPL == 1) {
            v[0] = *reinterpret_cast<const u64*>(p);
        } else if constexpr (VPL == 4) {
            asm("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
        } else {
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(p + 2 * j * G);
                v[2 * j] = q.x;
                v[2 * j + 1] = q.y;
            }
        }
    }
    __device__ __forceinline__ void load_if(const float2* p, int G, bool on) {
        if constexpr (VPL == 1) {
            v[0] = 0ull;
            if (on) v[0] = *reinterpret_cast<const u64*>(p);
        } else if constexpr (VPL == 4) {
            asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.b64 %0, 0;\n\tmov.b64 %1, 0;\n\tmov.b64 %2, 0;\n\tmov.b64 %3, 0;\n\t"
                "@p ld.global.v4.b64 {%0, %1, %2, %3}, [%4];\n\t}"
                : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p), "r"((uint32_t)on));
        } else {
#pragma unroll
            for (int j = 0; j < U; ++j)
                asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.b64 %0, 0;\n\tmov.b64 %1, 0;\n\t@p ld.global.v2.b64 {%0, %1}, [%2];\n\t}"
                    : "=l"(v[2 * j]), "=l"(v[2 * j + 1]) : "l"(p + 2 * j * G), "r"((uint32_t)on));
        }
    }
    __device__ __forceinline__ void store(float2* p, int G) const {
        if constexpr (VPL == 1) {
            __stcs(reinterpret_cast<u64*>(p), v[0]);
        } else if constexpr (VPL == 4) {
            asm volatile("st.global.cs.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3]) : "memory");
        } else {
#pragma unroll
            for (int j = 0; j < U; ++j)
                __stcs(reinterpret_cast<ulonglong2*>(p + 2 * j * G), make_ulonglong2(v[2 * j], v[2 * j + 1]));
        }
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = 0ull;
    }
    __device__ __forceinline__ void write(float2* p, int G) const {
        if constexpr (VPL == 1) *reinterpret_cast<u64*>(p) = v[0];
        else
#pragma unroll
            for (int j = 0; j < U; ++j) *reinterpret_cast<ulonglong2*>(p + 2 * j * G) = make_ulonglong2(v[2 * j], v[2 * j + 1]);
    }
    __device__ __forceinline__ void axpy(const float (&a)[VPL], const Row& x) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = fma2(pk(a[j], a[j]), x.v[j], v[j]);
    }
    __device__ __forceinline__ void add(float a, const Row& x) {
        const u64 aa = pk(a, a);
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = fma2(aa, x.v[j], v[j]);
    }
    __device__ __forceinline__ void add(float ar, float ai, const Row& x) {
        const u64 rr = pk(ar, ar), ii = pk(-ai, ai);
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            const float2 q = unpk(x.v[j]);
            v[j] = fma2(ii, pk(q.y, q.x), fma2(rr, x.v[j], v[j]));
        }
    }
};
template <int VPL> struct Row<double, VPL> {
    static constexpr int U = VPL;
    double2 v[VPL];
    __device__ __forceinline__ void load(const double2* p, int G) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = p[j * G];
    }
    __device__ __forceinline__ void store(double2* p, int G) const {
#pragma unroll
        for (int j = 0; j < VPL; ++j) __stcs(p + j * G, v[j]);
    }
    __device__ __forceinline__ void write(double2* p, int G) const {
#pragma unroll
        for (int j = 0; j < VPL; ++j) p[j * G] = v[j];
    }
    __device__ __forceinline__ void axpy(const double (&a)[VPL], const Row& x) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            v[j].x = fma(a[j], x.v[j].x, v[j].x);
            v[j].y = fma(a[j], x.v[j].y, v[j].y);
        }
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = make_double2(0.0, 0.0);
    }
    __device__ __forceinline__ void add(double a, const Row& x) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            v[j].x = fma(a, x.v[j].x, v[j].x);
            v[j].y = fma(a, x.v[j].y, v[j].y);
        }
    }
    __device__ __forceinline__ void add(double ar, double ai, const Row& x) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            v[j].x = fma(-ai, x.v[j].y, fma(ar, x.v[j].x, v[j].x));
            v[j].y = fma(ai, x.v[j].x, fma(ar, x.v[j].y, v[j].y));
        }
    }
};
// Vector of a lane's j-th value.
template <class T, int VPL>
__device__ __forceinline__ int vec_of(int l, int j, int G) {
    if (sizeof(T) == 4 && VPL == 4) return 4 * l + j;
    if (sizeof(T) == 4 && VPL >= 2) return 2 * (l + (j / 2) * G) + (j & 1);
    return l + j * G;
}

// Per-vector sums Re sum conj(x) y.
template <class T, int VPL> struct Dots;
template <int VPL> struct Dots<float, VPL> {
    u64 hi[VPL], lo[VPL];
    __device__ __forceinline__ void init(int j, double) { hi[j] = lo[j] = 0ull; }
    __device__ __forceinline__ void square(const Row<float, VPL>& x) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) acc2(hi[j], lo[j], x.v[j], x.v[j]);
    }
    // (hi, lo) of vector j: real and imaginary products together
    __device__ __forceinline__ double2 get(int j) const {
        const float2 h = unpk(hi[j]), l = unpk(lo[j]);
        float a = h.x, b = l.x;
        ff_add(a, b, h.y, l.y);
        double2 r;  // kept as a float pair in the two halves of one double's place
        r.x = __hiloint2double(__float_as_int(a), __float_as_int(b));
        r.y = 0.0;
        return r;
    }
};
template <int VPL> struct Dots<double, VPL> {
    double s[VPL], sc[VPL];
    __device__ __forceinline__ void init(int j, double scale) {
        s[j] = 0.0;
        sc[j] = scale;
    }
    __device__ __forceinline__ void finish(Row<double, VPL>& y, const Row<double, VPL>& x, bool dot) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            y.v[j].x *= sc[j];
            y.v[j].y *= sc[j];
            if (dot) s[j] = fma(x.v[j].y, y.v[j].y, fma(x.v[j].x, y.v[j].x, s[j]));
        }
    }
    __device__ __forceinline__ void square(const Row<double, VPL>& x) {
#pragma unroll
        for (int j = 0; j < VPL; ++j) s[j] = fma(x.v[j].y, x.v[j].y, fma(x.v[j].x, x.v[j].x, s[j]));
    }
    __device__ __forceinline__ double2 get(int j) const { return make_double2(s[j], 0.0); }
};
// The SpMV's sums and scales.  FP32: in shared memory, touched once a row (16-byte
// accesses, one per value); in registers beside the rows in flight they spilled, and
// every row wrote the spills through to L2 (Heisenberg L = 20, every sector, 32
// vectors: 310 -> 262 us a launch).
template <class T, int VPL> struct RowSums : Dots<T, VPL> {
    static constexpr int kBytes = 0;
    __device__ __forceinline__ explicit RowSums(char*) {}
};
template <int VPL> struct RowSums<float, VPL> {
    static constexpr int kBytes = kBT * VPL * 20;
    ulonglong2* s;  // (hi, lo) of the thread's j-th value at j * kBT
    float* sc;
    __device__ __forceinline__ explicit RowSums(char* mem)
        : s(reinterpret_cast<ulonglong2*>(mem) + threadIdx.x), sc(reinterpret_cast<float*>(mem + kBT * VPL * 16) + threadIdx.x * VPL) {}
    __device__ __forceinline__ void init(int j, double scale) {
        s[j * kBT] = make_ulonglong2(0ull, 0ull);
        sc[j] = (float)scale;
    }
    __device__ __forceinline__ void finish(Row<float, VPL>& y, const Row<float, VPL>& x, bool dot) {
        float f[VPL];
        if constexpr (VPL == 4) {
            const float4 f4 = *reinterpret_cast<const float4*>(sc);
            f[0] = f4.x, f[1] = f4.y, f[2] = f4.z, f[3] = f4.w;
        } else {
#pragma unroll
            for (int j = 0; j < VPL; ++j) f[j] = sc[j];
        }
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            y.v[j] = mul2(y.v[j], pk(f[j], f[j]));
            if (dot) {
                ulonglong2 a = s[j * kBT];
                acc2(a.x, a.y, x.v[j], y.v[j]);
                s[j * kBT] = a;
            }
        }
    }
    __device__ __forceinline__ double2 get(int j) const {
        Dots<float, VPL> d;
        d.hi[j] = s[j * kBT].x;
        d.lo[j] = s[j * kBT].y;
        return d.get(j);
    }
};
// Partial sums as the CTA adds them: FP32 as float pairs (a double-precision
// reduction in every CTA would cost more than its rows on the narrow FP64 pipe).
template <class T> struct Part;
template <> struct Part<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double v) { s += v; }
    __device__ __forceinline__ double pack() const { return s; }
    __device__ __forceinline__ double value() const { return s; }
};
template <> struct Part<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(double v) {
        ff_add(hi, lo, __int_as_float(__double2hiint(v)), __int_as_float(__double2loint(v)));
    }
    __device__ __forceinline__ double pack() const { return __hiloint2double(__float_as_int(hi), __float_as_int(lo)); }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
// part[v] = sum over the CTA's n_groups row groups of red[group * Rp + v], all
// threads taking part (the caller has synchronised after writing red).
template <class T>
__device__ __forceinline__ void reduce_vectors(double* red, int n_groups, int Rp, double* part) {
    const int v = threadIdx.x % Rp, s = threadIdx.x / Rp, ns = kBT / Rp;
    Part<T> a;
    if (s < ns)
        for (int g = s; g < n_groups; g += ns) a.add(red[g * Rp + v]);
    __syncthreads();
    if (s < ns) red[s * Rp + v] = a.pack();
    __syncthreads();
    int n = ns < n_groups ? ns : n_groups;
    while (n > 1) {  // halves onto each other
        const int h = (n + 1) / 2;
        if (s < n - h) {
            a.add(red[(s + h) * Rp + v]);
            red[s * Rp + v] = a.pack();
        }
        n = h;
        __syncthreads();
    }
    if ((int)threadIdx.x < Rp) part[threadIdx.x] = a.value();  // s = 0
}

// The last of a Hamiltonian's n_ctas CTAs (partials part[c * Rp + v], this CTA's
// written by its first Rp threads) adds them up, in CTA order by rows of kBT / Rp, and
// does the vectors' bookkeeping.
__device__ __forceinline__ void finish_ham(const Finish& f, int ham, uint32_t n_ctas, int Rp, const double* part, double* red) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(f.arrived + ham, 1u) == n_ctas - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) f.arrived[ham] = 0u;
    const int v = threadIdx.x % Rp, s = threadIdx.x / Rp, ns = kBT / Rp;
    double a = 0.0;
    if (s < ns) {
#pragma unroll 8
        for (uint32_t c = s; c < n_ctas; c += ns) a += __ldcg(part + (size_t)c * Rp + v);
        red[s * Rp + v] = a;
    }
    __syncthreads();
    for (int n = ns; n > 1;) {  // halves onto each other
        const int h = (n + 1) / 2;
        if (s < n - h) {
            a += red[(s + h) * Rp + v];
            red[s * Rp + v] = a;
        }
        n = h;
        __syncthreads();
    }
    if ((int)threadIdx.x < Rp) finish_vector(f.st, ham * Rp + v, a, f.mode, f.k);
}

// FUSED: the bookkeeping in the Hamiltonian's last CTA, and a tile dealt out to `parts` CTAs
// (an instantiation of its own: the code alone cost the large batches 2 %).
template <class T, int MODE, bool CPLX, int VPL, bool FUSED>
__global__ void __launch_bounds__(kBT, sizeof(T) == 4 ? 4 : 2)
    block_pack_kernel(const Params<T>* __restrict__ P, const Ham* __restrict__ hams, int n_hams, int run, int parts, int Rp,
                      const typename V2<T>::t* __restrict__ X, typename V2<T>::t* __restrict__ Y,
                      const double* __restrict__ scale, double* __restrict__ apart, const Finish fin) {
    using T2 = typename V2<T>::t;
    using R = Row<T, VPL>;
    __shared__ alignas(16) char sums_mem[RowSums<T, VPL>::kBytes > kBT * VPL * 8 ? RowSums<T, VPL>::kBytes : kBT * VPL * 8];
    double* const red = reinterpret_cast<double*>(sums_mem);  // once the rows are done
    __shared__ T s_amp[MODE == AMP_CODED ? 2 * kMaxAmps : 1];
    const int ham = find_ham(hams, n_hams, blockIdx.x, [](const Ham& h) { return h.cta0; });
    const Params<T>& p = P[ham];
    const uint32_t tile0 = FUSED ? (blockIdx.x - hams[ham].cta0) / (uint32_t)parts * (uint32_t)run
                                 : (blockIdx.x - hams[ham].cta0) * (uint32_t)run;
    const uint32_t count = min((uint32_t)run, p.n_items - tile0);
    const uint64_t base = hams[ham].base;
    if (MODE == AMP_CODED) {
        for (int i = threadIdx.x; i < 2 * p.n_amps; i += kBT) s_amp[i] = p.amps[i];
        __syncthreads();
    }
    const int G = Rp / VPL, NG = kBT / G;
    const int l = threadIdx.x % G, grp = threadIdx.x / G;
    constexpr int W0 = (sizeof(T) == 4 && VPL >= 2) ? VPL : 1;  // complex values of a unit
    RowSums<T, VPL> dots(sums_mem);
#pragma unroll
    for (int j = 0; j < VPL; ++j)
        dots.init(j, scale ? scale[(size_t)ham * Rp + vec_of<T, VPL>(l, j, G)] : 1.0);
    const T u = p.u;
    const Out<T>* const g_out = p.out;
    const Str<T>* const g_str = p.str;
    const uint2* __restrict__ tab = p.tab;
    const uint32_t* __restrict__ codes = p.codes;

    // the run's tiles and their blocks' lists
    __shared__ Item s_tile[kMaxRun];
    __shared__ uint4 s_blk[kMaxRun];
    __shared__ uint2 s_rec[kMaxRun];
    __shared__ Out<T> s_out[kMaxList];
    __shared__ Str<T> s_str[kMaxList];
    if (threadIdx.x < count) {
        const uint4 i4 = __ldg(reinterpret_cast<const uint4*>(p.items) + tile0 + threadIdx.x);
        const Item t{i4.x, i4.y, i4.z, i4.w};
        s_tile[threadIdx.x] = t;
        s_blk[threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(p.blk) + t.a);
        s_rec[threadIdx.x] = __ldg(p.tile + t.tile);
    }
    __syncthreads();
    uint32_t lo = 0, ls = 0;  // list entries of the whole run
    for (uint32_t i = 0; i < count; ++i) {
        lo += s_blk[i].y - s_blk[i].x;
        ls += s_blk[i].w - s_blk[i].z;
    }
    const bool staged = lo <= (uint32_t)kMaxList && ls <= (uint32_t)kMaxList;
    if (staged) {
        uint32_t o = 0, q = 0;
        for (uint32_t i = 0; i < count; ++i) {
            const uint4 b4 = s_blk[i];
            if (threadIdx.x < b4.y - b4.x) s_out[o + threadIdx.x] = g_out[b4.x + threadIdx.x];
            if (threadIdx.x < b4.w - b4.z) s_str[q + threadIdx.x] = g_str[b4.z + threadIdx.x];
            o += b4.y - b4.x;
            q += b4.w - b4.z;
        }
        __syncthreads();
    }
    const int rb = Rp * (int)sizeof(T2);  // bytes of a row
    const T2* __restrict__ Xh = X + base * (uint64_t)Rp + l * W0;  // the Hamiltonian's rows
    T2* __restrict__ Yh = Y + base * (uint64_t)Rp + l * W0;
    {
        uint32_t ti = 0, oo = 0, so = 0;  // the row's tile and where its lists start
        // the run's rows, or one of `parts` parts of its only tile's
        int row_lo = grp, row_hi = (int)count * kTile;
        if constexpr (FUSED)
            if (parts > 1) {
                const int lo = (int)((blockIdx.x - hams[ham].cta0) % (uint32_t)parts) * (kTile / parts);
                row_lo += lo;
                row_hi = lo + kTile / parts;
            }
        if (grp < NG)
            for (int rr = row_lo; rr < row_hi; rr += NG) {
                while (ti < (uint32_t)rr >> 7) {
                    oo += s_blk[ti].y - s_blk[ti].x;
                    so += s_blk[ti].w - s_blk[ti].z;
                    ++ti;
                }
                const Item it = s_tile[ti];
                const int r = rr & (kTile - 1);
                if (r >= (int)(it.tc & 0xFFu)) continue;
                const uint32_t lane = r & 31u, q = (uint32_t)r >> 5, tin = it.tc >> 8;
                const uint4 b4 = s_blk[ti];
                const uint2 rec = s_rec[ti];
                const uint32_t no = b4.y - b4.x, ns = b4.w - b4.z;
                const Out<T>* outl = staged ? s_out + oo : g_out + b4.x;
                const Str<T>* strl = staged ? s_str + so : g_str + b4.z;
                const uint32_t row = it.row0 + r;
                const uint32_t dc = p.diag_mode == DIAG_U8 ? (uint32_t)__ldg(static_cast<const uint8_t*>(p.dcode) + row)
                                                           : (uint32_t)__ldg(static_cast<const uint16_t*>(p.dcode) + row);
                const T2* xo = offset(Xh, (int)row, rb);
                const T2* xl = offset(Xh, (int)(it.row0 - tin * (uint32_t)kTile), rb);  // the block's rows
                auto rank_of = [](uint32_t w16) { return (int)(MODE == AMP_SIGNED ? w16 & 0x7FFFu : w16); };
                constexpr int kNone = MODE == AMP_SIGNED ? (int)kNone15 : (int)kNone16;
                // the row's index words before its values: the first quad, the straddling entries
                uint32_t first = rec.x;
                if (q > 0) first += ((rec.y & 0xFFu) + 3u) >> 2;
                if (q > 1) first += (((rec.y >> 8) & 0xFFu) + 3u) >> 2;
                if (q > 2) first += (((rec.y >> 16) & 0xFFu) + 3u) >> 2;
                const int slots = (int)((rec.y >> (8 * q)) & 0xFFu);
                uint32_t at = first * 32u + lane;
                uint2 nxt = __ldg(tab + at);
                uint32_t cn = MODE == AMP_CODED ? __ldg(codes + at) : 0u;
                uint32_t sw[kStrBatch], sc[kStrBatch];
                auto straddles = [&](uint32_t j) {
#pragma unroll
                    for (int i = 0; i < kStrBatch; ++i) {
                        sw[i] = (uint32_t)kNone;
                        sc[i] = 0u;
                        if (j + i < ns) {
                            const uint32_t as = strl[j + i].tab + tin * 32u + lane;
                            sw[i] = __ldg(reinterpret_cast<const uint16_t*>(tab + as) + q);
                            if (MODE == AMP_CODED) sc[i] = __ldg(reinterpret_cast<const uint8_t*>(codes + as) + q);
                        }
                    }
                };
                straddles(0);
                R acc;
                acc.zero();
                // outer entries, the rows of up to kBatch of them in flight; their number is the
                // warp's, so that a short rest is a shorter batch and not a chain of loads
                auto outer = [&](uint32_t k, auto batch) {
                    constexpr int N = decltype(batch)::value;
                    R v[N];
#pragma unroll
                    for (int i = 0; i < N; ++i) v[i].load(offset(xo, outl[k + i].delta, rb), G);
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        if (CPLX) acc.add(outl[k + i].ar, outl[k + i].ai, v[i]);
                        else acc.add(outl[k + i].ar, v[i]);
                    }
                };
                uint32_t k = 0;
                for (; k + kBatch <= no; k += kBatch) outer(k, Int<kBatch>{});
                if (no - k == 2) outer(k, Int<2>{});
                else if (no - k == 1) outer(k, Int<1>{});
                auto amp_add = [&](uint32_t w16, uint32_t code, T a, const R& v) {
                    if (MODE == AMP_CODED) {
                        const uint32_t c = code & 0xFFu;
                        if (CPLX) acc.add(s_amp[2 * c], s_amp[2 * c + 1], v);
                        else acc.add(s_amp[2 * c], v);
                    } else {
                        acc.add(MODE == AMP_SIGNED && (w16 & 0x8000u) ? -a : a, v);
                    }
                };
                for (int n = slots; n > 0; n -= 4) {
                    const uint2 e = nxt;
                    const uint32_t c = cn;
                    if (n > 4) {
                        at += 32u;
                        nxt = __ldg(tab + at);
                        if (MODE == AMP_CODED) cn = __ldg(codes + at);
                    }
                    if constexpr (sizeof(T) == 8) {
                        // one at a time, an empty slot ends the row: bound by the FP64 pipe, on
                        // which the empty slots' products would count like the others (2^20 rows,
                        // 32 vectors: 1.98 -> 1.78 ms)
                        unsigned long long e64 = (unsigned long long)e.y << 32 | e.x;
                        uint32_t c1 = c;
                        bool more = true;
#pragma unroll 1
                        for (int h = 0; h < 4; ++h) {
                            const uint32_t w16 = (uint32_t)e64 & 0xFFFFu;
                            const int to = rank_of(w16);
                            if (to == kNone) {
                                more = false;
                                break;
                            }
                            R v;
                            v.load(offset(xl, to, rb), G);
                            amp_add(w16, c1, u, v);
                            e64 >>= 16;
                            c1 >>= 8;
                        }
                        if (!more) break;
                    } else {
                        const uint32_t w[4] = {e.x & 0xFFFFu, e.x >> 16, e.y & 0xFFFFu, e.y >> 16};
                        if (rank_of(w[0]) == kNone) break;  // a row's entries come first
                        // the four rows' loads go out together; an empty slot reads zero
                        R v[4];
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const int to = rank_of(w[h]);
                            v[h].load_if(offset(xl, to, rb), G, to != kNone);
                        }
#pragma unroll
                        for (int h = 0; h < 4; ++h) amp_add(w[h], c >> (8 * h), u, v[h]);
                    }
                }
                for (uint32_t j = 0; j < ns; j += kStrBatch) {
                    if (j) straddles(j);
                    if constexpr (sizeof(T) == 8) {
#pragma unroll 1
                        for (uint32_t i = 0; i < (uint32_t)kStrBatch && j + i < ns; ++i) {
                            const uint32_t w16 = i ? sw[1] : sw[0];
                            const int to = rank_of(w16);
                            if (to == kNone) continue;
                            R v;
                            v.load(offset(Xh, (int)strl[j + i].off + to, rb), G);
                            amp_add(w16, i ? sc[1] : sc[0], strl[j + i].ar, v);
                        }
                    } else {
                        R v[kStrBatch];
#pragma unroll
                        for (int i = 0; i < kStrBatch; ++i) {
                            const int to = rank_of(sw[i]);
                            v[i].load_if(offset(Xh, j + i < ns ? (int)strl[j + i].off + to : 0, rb), G, to != kNone);
                        }
#pragma unroll
                        for (int i = 0; i < kStrBatch; ++i)
                            if (j + i < ns) amp_add(sw[i], sc[i], strl[j + i].ar, v[i]);
                    }
                }
                R x;
                x.load(xo, G);
                const T dr = __ldg(p.dtab + 2 * dc);
                if (p.cdiag) acc.add(dr, __ldg(p.dtab + 2 * dc + 1), x);
                else acc.add(dr, x);
                dots.finish(acc, x, apart != nullptr);
                acc.store(offset(Yh, (int)row, rb), G);
            }
    }
    if (apart) {
        double own[VPL];
#pragma unroll
        for (int j = 0; j < VPL; ++j) own[j] = dots.get(j).x;
        __syncthreads();  // red lies over the sums
        if (grp < NG)
#pragma unroll
            for (int j = 0; j < VPL; ++j) red[grp * Rp + vec_of<T, VPL>(l, j, G)] = own[j];
        __syncthreads();
        reduce_vectors<T>(red, NG, Rp, apart + (size_t)blockIdx.x * Rp);
        if constexpr (FUSED) finish_ham(fin, ham, (p.n_items + run - 1) / run * parts, Rp, apart + (size_t)hams[ham].cta0 * Rp, red);
    }
}

// w = y - ca u - cb up in place on y, and per CTA the partial ||w_v||^2 (u ==
// nullptr: only the norms of y; Up == nullptr: no previous vector).  A CTA takes
// `chunk` rows of one Hamiltonian, a lane one 16-byte unit (VPL values) of a row.
template <class T, int VPL, bool FUSED>
__global__ void __launch_bounds__(kBT)
    block_pack_update(const Ham* __restrict__ hams, int n_hams, uint32_t chunk, int Rp, typename V2<T>::t* __restrict__ Y,
                      const typename V2<T>::t* __restrict__ U, const typename V2<T>::t* __restrict__ Up,
                      const double* __restrict__ ca, const double* __restrict__ cb, double* __restrict__ part, const Finish fin) {
    using R = Row<T, VPL>;
    __shared__ double red[kBT * VPL];
    const int ham = find_ham(hams, n_hams, blockIdx.x, [](const Ham& h) { return h.row_cta0; });
    const uint32_t row0 = (blockIdx.x - hams[ham].row_cta0) * chunk;
    const uint32_t count = (uint32_t)min((unsigned long long)chunk, (unsigned long long)(hams[ham].dim - row0));
    const int G = Rp / VPL, NG = kBT / G;
    const int l = threadIdx.x % G, grp = threadIdx.x / G;
    Dots<T, VPL> dots;
    T a[VPL], b[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const size_t vid = (size_t)ham * Rp + vec_of<T, VPL>(l, j, G);
        dots.init(j, 1.0);
        a[j] = U ? -(T)ca[vid] : (T)0;
        b[j] = Up ? -(T)cb[vid] : (T)0;
    }
    const uint64_t o = (hams[ham].base + row0) * (uint64_t)Rp + l * VPL;
    if (grp < NG) {
#pragma unroll 4
        for (uint32_t r = grp; r < count; r += NG) {
            const uint64_t at = o + (uint64_t)r * Rp;
            R w;
            w.load(Y + at, G);
            if (U) {
                R u, v;
                u.load(U + at, G);
                if (Up) v.load(Up + at, G);
                w.axpy(a, u);
                if (Up) w.axpy(b, v);
                w.write(Y + at, G);
            }
            dots.square(w);
        }
#pragma unroll
        for (int j = 0; j < VPL; ++j) red[grp * Rp + vec_of<T, VPL>(l, j, G)] = dots.get(j).x;
    }
    __syncthreads();
    reduce_vectors<T>(red, NG, Rp, part + (size_t)blockIdx.x * Rp);
    if constexpr (FUSED) finish_ham(fin, ham, (uint32_t)((hams[ham].dim + chunk - 1) / chunk), Rp, part + (size_t)hams[ham].row_cta0 * Rp, red);
}

// Seeded Philox Gaussian start vectors in reference order: vector v of
// Hamiltonian h, element i of its basis' internal order (at row perm[i]), gets
// the Philox block (counter i, stream h * streams + v); padding vectors are zero.
template <class T2, bool F64>
__global__ void __launch_bounds__(kBT)
    block_pack_philox(const Ham* __restrict__ hams, int n_hams, uint32_t chunk, int Rp, int Ruser, int streams, uint64_t seed,
                      T2* __restrict__ U) {
    const int ham = find_ham(hams, n_hams, blockIdx.x, [](const Ham& h) { return h.row_cta0; });
    const uint64_t base = hams[ham].base;
    const uint32_t* __restrict__ perm = hams[ham].perm;
    const uint32_t i0 = (blockIdx.x - hams[ham].row_cta0) * chunk;
    const uint32_t count = (uint32_t)min((unsigned long long)chunk, (unsigned long long)(hams[ham].dim - i0));
    for (uint32_t e = threadIdx.x; e < count * (uint32_t)Rp; e += kBT) {
        const uint32_t i = i0 + e / Rp, v = e % Rp;
        T2 o;
        o.x = 0;
        o.y = 0;
        if ((int)v < Ruser) o = philox_cnormal<T2, F64>(seed, (uint64_t)ham * streams + v, i);
        U[(base + (perm ? perm[i] : i)) * (uint64_t)Rp + v] = o;
    }
}

// The vectors of one Hamiltonian (R contiguous FP64 vectors of n elements, one
// after the other) into its rows of the block vector; padding vectors are zero.
template <class T2>
__global__ void __launch_bounds__(kBT)
    block_pack_gather(const double2* __restrict__ src, uint64_t n, int R, int Rp, T2* __restrict__ dst) {
    __shared__ double2 t[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t r0 = blockIdx.x * 32ull;
    for (int v = w; v < Rp; v += kBT / 32)
        t[lane][v] = v < R && r0 + lane < n ? src[(uint64_t)v * n + r0 + lane] : make_double2(0.0, 0.0);
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * Rp; e += kBT) {
        const int r = e / Rp, v = e % Rp;
        if (r0 + r >= n) break;
        T2 o;
        o.x = t[r][v].x;
        o.y = t[r][v].y;
        dst[(r0 + r) * Rp + v] = o;
    }
}

}  // namespace blockk
}  // namespace qkg
