// SpMV kernels of the packed plan (pack.hpp): a tile of 128 consecutive rows is
// one warp's work (NQ = 4: lane l holds rows l, l + 32, l + 64 and l + 96) or
// four warps' (NQ = 1: 32 rows each).
//
// What bounds them.  FP32: the latency of the gathers (long-scoreboard stalls, half
// the issue slots used), so the entries are cheap to decode (a 64-bit load holds four
// ranks; a gather, its address and one packed FMA an entry), four gathers are in
// flight a warp, and the registers are held to 48 warps a SM.  Reading and writing
// vectors in the reference's order makes the lanes of a warp consecutive states:
// far flips, listed first, read one run.  L = 28 ring (40.1 M rows): 0.42 ms = 1.52
// TB/s of x and y; the kernel on the domain-wall order 0.66 ms, and 0.19 ms for each of
// the two permutation passes of an apply that this order does without.
// FP64: the integer pipe for equal magnitudes (L = 28 1.87 ms, L = 24 121 us); the FP64 pipe
// (88% busy) otherwise and in the older kernels (L = 24 197 us, and 40 of permutations).
#include "pack.hpp"
#include "pair.cuh"

#include <type_traits>

namespace qkg {
using namespace fastk;
using namespace packk;
using namespace pairk;
namespace {

// CTAs of four warps.  Resident CTAs the register allocation is held to: the
// kernels wait for gathers, so FP32 takes 48 warps a SM at 40 registers (L = 28
// ring: 32 warps 0.47 ms, 40 0.46, 48 0.42, 56 0.44) and 40 warps at 48 where signs,
// codes or the Lanczos step's terms need more (L = 28 Lanczos step 0.55 to 0.54 ms, L = 14
// Hubbard ring 0.153 to 0.148), FP64 24 warps at 80 (L = 28 ring: 16 warps 2.01 ms, 24 1.87, 32 1.93).
constexpr int kThreads = 128;
// Integer sums of four rows a lane with signs or the Lanczos step's terms: 20 warps at 96 registers
// (100 recurrence steps at L = 24: 19.1 ms with 24 warps and their spills, 18.4; 13-site Hubbard ring 151 and 150 us).
constexpr int kCtas32 = 12, kCtas32more = 10, kCtas64 = 6, kCtas64more = 5;

// ---- sums of one row -------------------------------------------------------
// FP32, real amplitudes.
struct SumF32 {
    using V = u64;  // one complex element
    u64 s;
    __device__ __forceinline__ void init() { s = 0ull; }
    __device__ __forceinline__ void add(float a, V x) { s = fma2(pk(a, a), x, s); }
    __device__ __forceinline__ void add(float ar, float ai, V x) {
        const float2 v = unpk(x);
        s = fma2(pk(ar, ar), x, s);
        s = fma2(pk(-ai, ai), pk(v.y, v.x), s);
    }
};
// FP64 on the FP64 pipe.
struct SumF64 {
    using V = double2;
    double r, i;
    __device__ __forceinline__ void init() { r = i = 0.0; }
    __device__ __forceinline__ void add(double a, V x) {
        r = fma(a, x.x, r);
        i = fma(a, x.y, i);
    }
    __device__ __forceinline__ void add(double ar, double ai, V x) {
        r = fma(-ai, x.y, fma(ar, x.x, r));
        i = fma(ai, x.x, fma(ar, x.y, i));
    }
};

// FP64 sums by integers aligned to the largest exponent met so far.  All
// amplitudes of the row have the same magnitude, so the row is that magnitude
// times a sum of +-x, and each x is its 53-bit significand shifted right by its
// exponent's distance from the largest: GB300 adds doubles at 2 a clock and SM,
// integers at 64.  The significand keeps 4 bits below its last place and 6
// above its first (up to 64 addends), so an addend loses less than 2^-56 of the
// largest one where a chain of FP64 additions rounds each partial sum to 2^-53.
// Infinities, NaN and rows whose sum, or its product with the magnitude, comes near the
// subnormal numbers (below 2^-959 for magnitudes from 2^-7 up) are left to the FP64 pipe
// (bad()), but for sums of nothing but zeros: every imaginary part of a real vector and most
// rows of a sparse one are that, and a warp that walks twice takes longer than the FP64 pipe alone (real vector, L = 24
// ring: 264 us walked twice, 237 on the FP64 pipe in the older kernels, 122 now).  What tells
// zeros from the smallest numbers is one FP32 addition an addend, on a pipe that is idle (on
// the integer pipe, two addends an OR: L = 28 1.97 against 1.94 ms); aligning the sum once
// for two addends pays for it (complex vectors without either and with both: L = 28 1.92 and
// 1.88 ms, L = 24 122 and 121 us, 13-site Hubbard ring 149 and 149, 23-site transverse-field
// ring 407 and 414).
struct IntSum {
    long long s;
    int e;
    float any;  // sum of the magnitudes of the addends' high words read as floats: 0 where those are all +-0
    // PTX shifts clamp: a distance of 64 or more leaves nothing
    static __device__ __forceinline__ u64 shift(u64 v, int d) {
        u64 r;
        asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));
        return r;
    }
    static __device__ __forceinline__ long long shift(long long v, int d) {
        long long r;
        asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));
        return r;
    }
    __device__ __forceinline__ void init() {
        s = 0;
        e = 0;
        any = 0.f;
    }
    // the x, each with its sign bit flipped by the top bit of its flip
    template <int N>
    __device__ __forceinline__ void add(const uint32_t (&flip)[N], const double (&x)[N]) {
        int em = e, ex[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            ex[k] = (int)(((uint32_t)__double2hiint(x[k]) >> 20) & 0x7FFu);
            em = max(em, ex[k]);
        }
        s = shift(s, em - e);
        e = em;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t hi = (uint32_t)__double2hiint(x[k]), lo = (uint32_t)__double2loint(x[k]);
            any += fabsf(__uint_as_float(hi));
            u64 m = ((u64)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
            m = shift(m << 4, em - ex[k]);
            const long long sg = (long long)((int)(hi ^ flip[k]) >> 31);  // 0 or -1
            s += ((long long)m ^ sg) - sg;
        }
    }
    // Whether the sum is one of zeros: with every high word +-0 the addends are below 2^32 units
    // of 2^-1074, and their sum is what s holds below the weight 2^56 of the (absent) leading ones.
    __device__ __forceinline__ bool zeros() const { return any == 0.f && (s << 8) == 0; }
    __device__ __forceinline__ bool bad(int e_min) const { return e == 0x7FF || (e < e_min && !zeros()); }
    __device__ __forceinline__ double value(double v) const { return v * __hiloint2double(e << 20, 0) * (double)s; }
};
struct SumI64 {
    using V = double2;
    IntSum r, i;
    __device__ __forceinline__ void init() {
        r.init();
        i.init();
    }
    template <int N>
    __device__ __forceinline__ void add_n(const double (&a)[N], const V* x) {  // a = +-u
        uint32_t flip[N];
        double re[N], im[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            flip[k] = (uint32_t)__double2hiint(a[k]);
            re[k] = x[k].x;
            im[k] = x[k].y;
        }
        r.add(flip, re);
        i.add(flip, im);
    }
    __device__ __forceinline__ void add(double a, V x) {
        const double a1[1] = {a};
        add_n(a1, &x);
    }
    __device__ __forceinline__ void add(double, double, V) {}  // never called: coded amplitudes go to SumF64
    __device__ __forceinline__ bool bad(int e_min) const { return r.bad(e_min) || i.bad(e_min); }
};

// a with the sign of the top bit of w applied
__device__ __forceinline__ float with_sign(float a, uint32_t w) {
    return __uint_as_float(__float_as_uint(a) ^ (w & 0x80000000u));
}
__device__ __forceinline__ double with_sign(double a, uint32_t w) {
    return __hiloint2double(__double2hiint(a) ^ (int)(w & 0x80000000u), __double2loint(a));
}

// Element i of v; on = false: zero, without a load.
template <class T> struct Elem;
template <> struct Elem<float> {
    using V = u64;
    static __device__ __forceinline__ V load(const float2* p) { return __ldg(reinterpret_cast<const u64*>(p)); }
    static __device__ __forceinline__ V load_if(const float2* p, bool on) {
        V v;
        asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.b64 %0, 0;\n\t@p ld.global.nc.b64 %0, [%1];\n\t}"
            : "=l"(v) : "l"(p), "r"((uint32_t)on));
        return v;
    }
};
template <> struct Elem<double> {
    using V = double2;
    static __device__ __forceinline__ V load(const double2* p) { return __ldg(p); }
    static __device__ __forceinline__ V load_if(const double2* p, bool on) {
        V v;
        asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\tmov.f64 %1, 0d0000000000000000;\n\t"
            "@p ld.global.nc.v2.f64 {%0, %1}, [%2];\n\t}"
            : "=d"(v.x), "=d"(v.y) : "l"(p), "r"((uint32_t)on));
        return v;
    }
};

// The off-diagonal sums of a warp's tile.  MODE: AmpMode; CPLX: complex
// amplitudes (coded).
template <class T, class Sum, int MODE, bool CPLX, int NQ>
__device__ __forceinline__ void walk(const Params<T>& p, const Item& it, uint32_t q0, const typename V2<T>::t* __restrict__ x,
                                     const T* s_amp, Sum (&acc)[NQ]) {
    using E = Elem<T>;
    using V = typename E::V;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t cnt = it.tc & 0xFFu, tin = it.tc >> 8;
    const uint4 b4 = __ldg(reinterpret_cast<const uint4*>(p.blk) + it.a);
    const uint2 t2 = __ldg(p.tile + it.tile);
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q].init();
    // outer entries: one offset and amplitude for the whole block
    const auto* xr = x + it.row0 + lane + 32u * q0;
    if (cnt >= 32u * (q0 + NQ)) {
        uint32_t k = b4.x;
        if constexpr (std::is_same<Sum, SumI64>::value) {
            for (; k + 2 <= b4.y; k += 2) {
                const Out<T> o0 = p.out[k], o1 = p.out[k + 1];
                const auto *x0 = xr + o0.delta, *x1 = xr + o1.delta;
                const T a[2] = {o0.ar, o1.ar};
                V v[NQ][2];
#pragma unroll
                for (int q = 0; q < NQ; ++q) v[q][0] = E::load(x0 + 32 * q), v[q][1] = E::load(x1 + 32 * q);
#pragma unroll
                for (int q = 0; q < NQ; ++q) acc[q].add_n(a, v[q]);
            }
        }
#pragma unroll(NQ == 4 ? 2 : 4)
        for (; k < b4.y; ++k) {
            const Out<T> o = p.out[k];
            const auto* xo = xr + o.delta;
            V v[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) v[q] = E::load(xo + 32 * q);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if (CPLX) acc[q].add(o.ar, o.ai, v[q]);
                else acc[q].add(o.ar, v[q]);
            }
        }
    } else {
        for (uint32_t k = b4.x; k < b4.y; ++k) {
            const Out<T> o = p.out[k];
            const auto* xo = xr + o.delta;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (lane + 32u * (q0 + q) < cnt) {
                    const V v = E::load(xo + 32 * q);
                    if (CPLX) acc[q].add(o.ar, o.ai, v);
                    else acc[q].add(o.ar, v);
                }
        }
    }
    // entry k of a quad: rank, whether there is one, amplitude
    auto rank_of = [&](const uint2& e, int k, bool& on) -> uint32_t {
        const uint32_t w = (k & 2) ? e.y : e.x;
        const uint32_t r = (k & 1) ? w >> 16 : w & 0xFFFFu;
        if (MODE == AMP_SIGNED) {
            on = (r & 0x7FFFu) != kNone15;
            return r & 0x7FFFu;
        }
        on = r != kNone16;
        return r;
    };
    auto add_entry = [&](const uint2& e, int k, uint32_t code, Sum& s, const V& v, T u) {
        if (MODE == AMP_CODED) {
            const uint32_t c = (code >> (8 * k)) & 0xFFu;
            if (CPLX) s.add(s_amp[2 * c], s_amp[2 * c + 1], v);
            else s.add(s_amp[2 * c], v);
        } else if (MODE == AMP_SIGNED) {
            const uint32_t w = (k & 2) ? e.y : e.x;
            s.add(with_sign(u, (k & 1) ? w : w << 16), v);
        } else {
            s.add(u, v);
        }
    };
    // inner entries, row group by row group; the next quad is loaded before this
    // one's gathers
    {
        const auto* xb = x + (it.row0 - tin * (uint32_t)kTile);
        uint32_t first = t2.x;
        if (NQ == 1) {  // the quads of the row groups before this one
            if (q0 > 0) first += ((t2.y & 0xFFu) + 3u) >> 2;
            if (q0 > 1) first += (((t2.y >> 8) & 0xFFu) + 3u) >> 2;
            if (q0 > 2) first += (((t2.y >> 16) & 0xFFu) + 3u) >> 2;
        }
        uint32_t at = first * 32u + lane;
        uint2 nxt = __ldg(p.tab + at);
        uint32_t cn = MODE == AMP_CODED ? __ldg(p.codes + at) : 0u;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            for (int n = (int)((t2.y >> (8 * (q0 + q))) & 0xFFu); n > 0; n -= 4) {
                const uint2 e = nxt;
                const uint32_t c = cn;
                at += 32u;
                nxt = __ldg(p.tab + at);
                if (MODE == AMP_CODED) cn = __ldg(p.codes + at);
                V v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    bool on;
                    const uint32_t r = rank_of(e, k, on);
                    v[k] = E::load_if(xb + r, on);
                }
                if constexpr (std::is_same<Sum, SumI64>::value) {
                    auto pair = [&](uint32_t w, const V* v2) {
                        const T a[2] = {MODE == AMP_SIGNED ? with_sign(p.u, w << 16) : p.u,
                                        MODE == AMP_SIGNED ? with_sign(p.u, w) : p.u};
                        acc[q].add_n(a, v2);
                    };
                    pair(e.x, v);
                    if (n > 2) pair(e.y, v + 2);
                    continue;
                }
                add_entry(e, 0, c, acc[q], v[0], p.u);
                add_entry(e, 1, c, acc[q], v[1], p.u);
                if (sizeof(T) == 4 || n > 2) {  // a slot costs the FP64 sums tens of instructions
                    add_entry(e, 2, c, acc[q], v[2], p.u);
                    add_entry(e, 3, c, acc[q], v[3], p.u);
                }
            }
        }
    }
    // straddling tables: one entry a row
    for (uint32_t k = b4.z; k < b4.w; ++k) {
        const Str<T> s = p.str[k];
        const uint32_t at = s.tab + tin * 32u + lane;
        const uint2 e = __ldg(p.tab + at);
        const uint32_t c = MODE == AMP_CODED ? __ldg(p.codes + at) : 0u;
        V v[NQ];
        if (NQ == 4) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                bool on;
                const uint32_t r = rank_of(e, q, on);
                v[q] = E::load_if(x + s.off + r, on);
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q) add_entry(e, q, c, acc[q], v[q], s.ar);
        } else {
            // entry q0, brought to the first place
            const uint32_t w = (q0 & 2u) ? e.y : e.x;
            const uint2 f = make_uint2((q0 & 1u) ? w >> 16 : w, 0u);
            bool on;
            const uint32_t r = rank_of(f, 0, on);
            v[0] = E::load_if(x + s.off + r, on);
            add_entry(f, 0, c >> (8u * q0), acc[0], v[0], s.ar);
        }
    }
}

template <class T>
__device__ __forceinline__ void load_amps(const Params<T>& p, T* s_amp) {
    for (int i = threadIdx.x; i < 2 * p.n_amps; i += blockDim.x) s_amp[i] = p.amps[i];
    __syncthreads();
}

template <class T>
__device__ __forceinline__ void diag_at(const Params<T>& p, uint32_t row, T& dr, T& di) {
    const uint32_t c = p.diag_mode == DIAG_U8 ? (uint32_t)__ldg(static_cast<const uint8_t*>(p.dcode) + row)
                                              : (uint32_t)__ldg(static_cast<const uint16_t*>(p.dcode) + row);
    dr = __ldg(p.dtab + 2 * c);
    di = __ldg(p.dtab + 2 * c + 1);
}

// Lanczos mode: the last CTA adds the grid's partials and sets alpha.
template <class T>
__device__ __forceinline__ void finish_alpha(const Params<T>& p) {
    if (!p.fin.st || !last_cta(p.fin.arrived)) return;
    const double t = sum_partials(p.apart, gridDim.x);
    if (threadIdx.x == 0) lz_set_alpha(p.fin, t);
}

// FP32.  LZ: the Lanczos step's form (operands from *p.lz, y = scale H x -
// bprev vprev, per-CTA partials of Re<x, y>).
template <int MODE, bool CPLX, bool LZ, int NQ>
__global__ void __launch_bounds__(kThreads, LZ || MODE != AMP_UNIFORM ? kCtas32more : kCtas32)
    pack32_kernel(const Params<float> p, const float2* __restrict__ x_in, float2* __restrict__ y_in) {
    __shared__ float s_amp[MODE == AMP_CODED ? 2 * kMaxAmps : 1];
    if (MODE == AMP_CODED) load_amps(p, s_amp);
    const float2* __restrict__ x = x_in;
    float2* __restrict__ y = y_in;
    float scale = 1.f, bprev = 0.f;
    const float2* __restrict__ vprev = nullptr;
    if (LZ) {
        const LzOperands o = *p.lz;
        x = static_cast<const float2*>(o.x);
        y = static_cast<float2*>(o.y);
        vprev = static_cast<const float2*>(o.vprev);
        scale = o.scale32;
        bprev = o.bprev32;
    }
    const uint32_t wid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    const uint32_t id = NQ == 4 ? wid : wid >> 2, q0 = NQ == 4 ? 0u : wid & 3u;
    u64 dot_hi = 0ull, dot_lo = 0ull;  // real and imaginary products apart
    if (id < p.n_items) {
        const uint4 i4 = __ldg(reinterpret_cast<const uint4*>(p.items) + id);
        const Item it{i4.x, i4.y, i4.z, i4.w};
        SumF32 acc[NQ];
        walk<float, SumF32, MODE, CPLX, NQ>(p, it, q0, x, s_amp, acc);
        const uint32_t cnt = it.tc & 0xFFu, row0 = it.row0 + lane + 32u * q0;
        uint32_t dc[NQ];
        u64 xv[NQ], pv[NQ];
        auto own = [&](int q) {  // row q's own values
            const uint32_t row = lane + 32u * (q0 + q) < cnt ? row0 + 32u * q : it.row0;
            dc[q] = p.diag_mode == DIAG_U8 ? (uint32_t)__ldg(static_cast<const uint8_t*>(p.dcode) + row)
                                           : (uint32_t)__ldg(static_cast<const uint16_t*>(p.dcode) + row);
            xv[q] = Elem<float>::load(x + row);
            pv[q] = 0ull;
            // read once a step: evict-first, so x keeps more of L2
            if (LZ && vprev) pv[q] = __ldcs(reinterpret_cast<const u64*>(vprev + row));
        };
        if (LZ)  // all in flight together (L = 28: 0.59 to 0.54 ms; without v_{k-1} it costs registers: 0.42 to 0.43)
#pragma unroll
            for (int q = 0; q < NQ; ++q) own(q);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (lane + 32u * (q0 + q) >= cnt) continue;
            if (!LZ) own(q);
            const float dr = __ldg(p.dtab + 2 * dc[q]);
            if (p.cdiag) acc[q].add(dr, __ldg(p.dtab + 2 * dc[q] + 1), xv[q]);
            else acc[q].add(dr, xv[q]);
            u64 o = acc[q].s;
            if (LZ) {
                o = mul2(o, pk(scale, scale));
                if (vprev) o = fma2(pk(-bprev, -bprev), pv[q], o);
                acc2(dot_hi, dot_lo, xv[q], o);
            }
            __stcs(reinterpret_cast<u64*>(y + row0 + 32u * q), o);
        }
    }
    if (LZ) {
        const float2 h = unpk(dot_hi), l = unpk(dot_lo);
        float hi = h.x, lo = l.x;
        ff_add(hi, lo, h.y, l.y);
        const float2 t = block_sum_ff(hi, lo);
        if (threadIdx.x == 0) p.apart[blockIdx.x] = make_double2((double)t.x + (double)t.y, 0.0);
        finish_alpha(p);
    }
}

// FP64.  EQUAL: every amplitude has the same magnitude p.u (sums of aligned
// integers).  LZ as above.
template <int MODE, bool CPLX, bool EQUAL, bool LZ, int NQ>
__global__ void __launch_bounds__(kThreads, EQUAL && NQ == 4 && (LZ || MODE == AMP_SIGNED) ? kCtas64more : kCtas64)
    pack64_kernel(const Params<double> p, const double2* __restrict__ x_in, double2* __restrict__ y_in) {
    __shared__ double s_amp[MODE == AMP_CODED ? 2 * kMaxAmps : 1];
    if (MODE == AMP_CODED) load_amps(p, s_amp);
    const double2* __restrict__ x = x_in;
    double2* __restrict__ y = y_in;
    double scale = 1.0, bprev = 0.0, dot = 0.0;
    const double2* __restrict__ vprev = nullptr;
    if (LZ) {
        const LzOperands o = *p.lz;
        x = static_cast<const double2*>(o.x);
        y = static_cast<double2*>(o.y);
        vprev = static_cast<const double2*>(o.vprev);
        scale = o.scale;
        bprev = o.bprev;
    }
    const uint32_t wid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    const uint32_t id = NQ == 4 ? wid : wid >> 2, q0 = NQ == 4 ? 0u : wid & 3u;
    if (id < p.n_items) {
        const uint4 i4 = __ldg(reinterpret_cast<const uint4*>(p.items) + id);
        const Item it{i4.x, i4.y, i4.z, i4.w};
        const uint32_t cnt = it.tc & 0xFFu;
        double orr[NQ], oi[NQ];
        bool redo = !EQUAL;
        if constexpr (EQUAL) {
            SumI64 acc[NQ];
            walk<double, SumI64, MODE, false, NQ>(p, it, q0, x, s_amp, acc);
            const double v = fabs(p.u) * 0x1p-56;
            bool bad = false;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                bad = bad || (lane + 32u * (q0 + q) < cnt && acc[q].bad(p.e_min));
                orr[q] = acc[q].r.value(v);
                oi[q] = acc[q].i.value(v);
            }
            redo = __any_sync(0xffffffffu, bad);
        }
        if (redo) {
            SumF64 acc[NQ];
            walk<double, SumF64, MODE, CPLX, NQ>(p, it, q0, x, s_amp, acc);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                orr[q] = acc[q].r;
                oi[q] = acc[q].i;
            }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (lane + 32u * (q0 + q) >= cnt) continue;
            const uint32_t row = it.row0 + lane + 32u * (q0 + q);
            double dr, di;
            diag_at(p, row, dr, di);
            const double2 xv = __ldg(x + row);
            double2 o;
            o.x = fma(dr, xv.x, orr[q]);
            o.y = fma(dr, xv.y, oi[q]);
            if (p.cdiag) {
                o.x = fma(-di, xv.y, o.x);
                o.y = fma(di, xv.x, o.y);
            }
            if (LZ) {
                o.x *= scale;
                o.y *= scale;
                if (vprev) {
                    const double2 pv = __ldcs(vprev + row);
                    o.x = fma(-bprev, pv.x, o.x);
                    o.y = fma(-bprev, pv.y, o.y);
                }
                dot = fma(xv.y, o.y, fma(xv.x, o.x, dot));
            }
            __stcs(y + row, o);
        }
    }
    if (LZ) {
        dot = block_sum_d(dot);
        if (threadIdx.x == 0) p.apart[blockIdx.x] = make_double2(dot, 0.0);
        finish_alpha(p);
    }
}

// Four warps a tile (NQ = 1) below 24 tiles a SM: one warp a tile leaves the
// SMs short of loads in flight there, and pays for itself above, where the four
// rows share the block's entries.  FP32 / FP64, one against four warps: L = 14
// 6.3 / 10.3 against 4.2 / 6.2 us, L = 20 (1,700 tiles) 10.3 / 16.5 against 7.1 /
// 13.5 us, L = 24 (21,500 tiles) 28.8 / 120.5 against 43.1 / 130.8 us.
bool split_tiles(uint32_t n_items) { return n_items < 152u * 24u; }

}  // namespace

uint32_t pack_ctas(const PackPlan& P) {
    const uint32_t n = P.n_items(), w = kThreads / 32;
    return split_tiles(n) ? n : (n + w - 1) / w;
}

namespace {
// go(mode, complex amplitudes, rows a lane) for the plan's form
template <class F>
void pick(const PackPlan& P, F&& go) {
    using std::integral_constant;
    auto rows = [&](auto mode, auto cplx) {
        if (split_tiles(P.n_items())) go(mode, cplx, integral_constant<int, 1>{});
        else go(mode, cplx, integral_constant<int, 4>{});
    };
    if (P.mode() == AMP_UNIFORM) rows(integral_constant<int, AMP_UNIFORM>{}, std::false_type{});
    else if (P.mode() == AMP_SIGNED) rows(integral_constant<int, AMP_SIGNED>{}, std::false_type{});
    else if (P.real()) rows(integral_constant<int, AMP_CODED>{}, std::false_type{});
    else rows(integral_constant<int, AMP_CODED>{}, std::true_type{});
}
}  // namespace

void pack_apply_f32(const PackPlan& P, Params<float>& p, const float2* x, float2* y, cudaStream_t s) {
    if (!p.n_items) return;
    const unsigned g = pack_ctas(P), t = kThreads;
    pick(P, [&](auto m, auto c, auto nq) {
        constexpr int M = decltype(m)::value, N = decltype(nq)::value;
        constexpr bool C = decltype(c)::value;
        if (p.lz) pack32_kernel<M, C, true, N><<<g, t, 0, s>>>(p, x, y);
        else pack32_kernel<M, C, false, N><<<g, t, 0, s>>>(p, x, y);
    });
    QKG_LAUNCHED();
}

void pack_apply_f64(const PackPlan& P, Params<double>& p, const double2* x, double2* y, cudaStream_t s) {
    if (!p.n_items) return;
    const unsigned g = pack_ctas(P), t = kThreads;
    pick(P, [&](auto m, auto c, auto nq) {
        constexpr int M = decltype(m)::value, N = decltype(nq)::value;
        constexpr bool C = decltype(c)::value;
        if constexpr (M != AMP_CODED) {
            if (P.equal_magnitude()) {
                if (p.lz) pack64_kernel<M, C, true, true, N><<<g, t, 0, s>>>(p, x, y);
                else pack64_kernel<M, C, true, false, N><<<g, t, 0, s>>>(p, x, y);
                return;
            }
        }
        if (p.lz) pack64_kernel<M, C, false, true, N><<<g, t, 0, s>>>(p, x, y);
        else pack64_kernel<M, C, false, false, N><<<g, t, 0, s>>>(p, x, y);
    });
    QKG_LAUNCHED();
}

}  // namespace qkg
