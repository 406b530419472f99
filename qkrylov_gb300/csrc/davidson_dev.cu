// Davidson in FP64 (src/solvers/davidson.cpp:86-227) with its coefficients and
// norms on the device: an iteration waits for the GPU twice, for the new rows of
// the projected matrix (with the norms of the vectors just added) and for the
// residual norms.
//
// The projected matrix keeps the entries of unchanged vectors (the reference
// recomputes all m (m + 1) / 2 dots each iteration).  The k residuals, their norms
// and the preconditioned corrections come out of one pass over V and HV; the
// residuals themselves are never stored.  A correction that vanishes against the
// basis (norm <= 1e-10, which the reference drops) is scaled to zero on the device,
// so the ones after it are not changed by it, and leaves the lists when the host
// sees its norm.
#include "fast_common.cuh"
#include "solvers.hpp"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <type_traits>

namespace qkg {
using namespace fastk;
namespace {
constexpr int kT = 256;
constexpr double kDropped = 1e-10;  // davidson.cpp:216: corrections of a smaller norm are not added

// result[j] = f * sum of column j's partials
__global__ void __launch_bounds__(kT) dav_finish(const double2* __restrict__ part, int nparts, double f, double2* __restrict__ result) {
    const int j = blockIdx.x;
    double re = 0.0, im = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        const double2 v = part[(size_t)j * nparts + i];
        re += v.x;
        im += v.y;
    }
    re = block_sum_d(re);
    im = block_sum_d(im);
    if (threadIdx.x == 0) result[j] = make_double2(f * re, f * im);
}

// t += sum_j c_j V_j (j < k); the last CTA leaves (||t||^2, 1 / ||t||, 0 where the
// norm is below kDropped) in norm.
__global__ void __launch_bounds__(kT) dav_subtract(const double2* const* __restrict__ V, int k, const double2* __restrict__ c,
                                                   double2* __restrict__ t, uint64_t n, double2* part, unsigned int* arrived,
                                                   double2* norm) {
    extern __shared__ double2 s_c[];
    const double2** s_v = reinterpret_cast<const double2**>(s_c + k);
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
        s_c[j] = c[j];
        s_v[j] = V[j];
    }
    __syncthreads();
    double acc = 0.0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double2 x = t[i];
        int j = 0;
        for (; j + 4 <= k; j += 4) {
            double2 a[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) a[q] = s_v[j + q][i];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 b = s_c[j + q];
                x.x = fma(b.x, a[q].x, fma(-b.y, a[q].y, x.x));
                x.y = fma(b.x, a[q].y, fma(b.y, a[q].x, x.y));
            }
        }
        for (; j < k; ++j) {
            const double2 a = s_v[j][i], b = s_c[j];
            x.x = fma(b.x, a.x, fma(-b.y, a.y, x.x));
            x.y = fma(b.x, a.y, fma(b.y, a.x, x.y));
        }
        t[i] = x;
        acc = fma(x.y, x.y, fma(x.x, x.x, acc));
    }
    acc = block_sum_d(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = make_double2(acc, 0.0);
    if (!last_cta(arrived)) return;
    const double s = sum_partials(part, gridDim.x);
    if (threadIdx.x == 0) {
        const double nr = sqrt(s);
        *norm = make_double2(nr, nr > kDropped ? 1.0 / nr : 0.0);
    }
}
__global__ void __launch_bounds__(kT) dav_scale(const double2* __restrict__ norm, double2* __restrict__ t, uint64_t n) {
    const double f = norm->y;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double2 x = t[i];
        // a dropped vector may hold anything: zero, not 0 * x
        x.x = f != 0.0 ? x.x * f : 0.0;
        x.y = f != 0.0 ? x.y * f : 0.0;
        t[i] = x;
    }
}

// For K Ritz pairs: r = sum_j s_j (HV_j - lambda V_j), t = r / (d - lambda) with the
// reference's clamp (davidson.cpp:171-175), and ||r||^2 in norm[k].x.
// cs[k * m + j] = s_j of pair k.  The coefficients are in shared memory: at most
// kResidualCoefs of them a pass (32 KB), so a wide basis takes its pairs in more passes.
constexpr int kResidualCoefs = 2048;
template <int K>
__global__ void __launch_bounds__(kT) dav_residual(const double2* const* __restrict__ V, const double2* const* __restrict__ HV,
                                                   int m, const double2* __restrict__ cs, const double* __restrict__ lambda,
                                                   const double2* __restrict__ diag, double2* const* __restrict__ t, uint64_t n,
                                                   double2* part, unsigned int* arrived, double2* norm) {
    extern __shared__ double2 s_c[];  // K * m coefficients
    for (int j = threadIdx.x; j < K * m; j += blockDim.x) s_c[j] = cs[j];
    __syncthreads();
    double lam[K], acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        lam[k] = lambda[k];
        acc[k] = 0.0;
    }
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        // two sums a pair, s HV and s V: the difference is taken once
        double hr[K], hi[K], vr[K], vi[K];
#pragma unroll
        for (int k = 0; k < K; ++k) hr[k] = hi[k] = vr[k] = vi[k] = 0.0;
        for (int j = 0; j < m; ++j) {
            const double2 h = HV[j][i], v = V[j][i];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const double2 c = s_c[k * m + j];
                hr[k] = fma(c.x, h.x, fma(-c.y, h.y, hr[k]));
                hi[k] = fma(c.x, h.y, fma(c.y, h.x, hi[k]));
                vr[k] = fma(c.x, v.x, fma(-c.y, v.y, vr[k]));
                vi[k] = fma(c.x, v.y, fma(c.y, v.x, vi[k]));
            }
        }
        const double2 d = diag[i];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double rr = fma(-lam[k], vr[k], hr[k]), ri = fma(-lam[k], vi[k], hi[k]);
            acc[k] = fma(ri, ri, fma(rr, rr, acc[k]));
            double dr = d.x - lam[k], di = d.y;
            if (dr * dr + di * di < 1e-20) {
                dr = (dr >= 0) ? 1e-10 : -1e-10;
                di = 0.0;
            }
            const double inv = 1.0 / (dr * dr + di * di);
            t[k][i] = make_double2((rr * dr + ri * di) * inv, (ri * dr - rr * di) * inv);
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double s = block_sum_d(acc[k]);
        if (threadIdx.x == 0) part[(size_t)k * gridDim.x + blockIdx.x] = make_double2(s, 0.0);
    }
    if (!last_cta(arrived)) return;
    for (int k = 0; k < K; ++k) {
        const double s = sum_partials(part + (size_t)k * gridDim.x, gridDim.x);
        if (threadIdx.x == 0) norm[k] = make_double2(s, 0.0);
    }
}

__global__ void dav_unit(double2* v, uint64_t i) { v[i] = make_double2(1.0, 0.0); }

// Order of the reference's seeds: std::sort of the indices by the diagonal's real
// part (davidson.cpp:111-121).  Sorting (value, index) pairs by value makes the same
// comparisons and moves, so ties fall as they do there.
std::vector<uint64_t> seed_order(const std::vector<double>& d, int n_eig) {
    const uint64_t n = d.size();
    std::vector<uint64_t> out(n_eig);
    if (n <= (1ull << 23)) {
        std::vector<std::pair<double, uint32_t>> p(n);
        for (uint64_t i = 0; i < n; ++i) p[i] = {d[i], (uint32_t)i};
        std::sort(p.begin(), p.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
        for (int i = 0; i < n_eig; ++i) out[i] = p[i].second;
    } else {  // ties by index
        std::vector<uint64_t> di(n);
        std::iota(di.begin(), di.end(), 0);
        std::partial_sort(di.begin(), di.begin() + n_eig, di.end(),
                          [&](uint64_t i, uint64_t j) { return d[i] < d[j] || (d[i] == d[j] && i < j); });
        std::copy(di.begin(), di.begin() + n_eig, out.begin());
    }
    return out;
}
}  // namespace

DavidsonOut davidson_f64(Hamiltonian& H, int n_eig, int max_sub, double tol, bool want_vecs, bool f32_stream, int max_iter) {
    DavidsonOut out;
    const uint64_t n = H.dim();
    if (n == 0) return out;
    const auto t_start = std::chrono::steady_clock::now();
    cudaStream_t st = H.stream();
    n_eig = (int)std::min<uint64_t>((uint64_t)n_eig, n);
    max_sub = std::max(max_sub, 2 * n_eig);
    QKG_REQUIRE(max_sub + n_eig <= 1024, "Davidson: subspace limited to 1024 vectors");
    const size_t vb = n * sizeof(double2);
    release_workspace_if_short(H, (size_t)(2 * (max_sub + 2 * n_eig) + 4) * vb);
    const auto lock = H.workspace_lock();
    const TrimVectors trim{H};

    // vectors by slot of the kept Krylov memory
    std::vector<int> spare;
    int slots = 0;
    auto ptr = [&](int s) { return static_cast<double2*>(H.krylov_vector((size_t)s, vb)); };
    auto get = [&] {
        if (!spare.empty()) {
            const int s = spare.back();
            spare.pop_back();
            return s;
        }
        ptr(slots);
        return slots++;
    };
    const int s_diag = get(), s_tmp = get();
    std::vector<int> V, HV, T(n_eig);  // T: where the next corrections go
    for (auto& t : T) t = get();

    // device scratch: results (read back), coefficients, pointer tables, partials
    const int cap = max_sub + 2 * n_eig + 2, KB = 4;  // KB: residuals a pass
    const int g = (int)std::max<uint64_t>(1, std::min<uint64_t>((n + kT - 1) / kT, 152ull * 8));
    const size_t n_res = (size_t)n_eig * (2 * cap + 1), n_coef = (size_t)cap + (size_t)n_eig * cap;
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    size_t off = 0;
    auto take = [&](size_t b) { const size_t o = off; off += al(b); return o; };
    const size_t o_res = take(n_res * 16), o_coef = take(n_coef * 16), o_lam = take(n_eig * 8),
                 o_tab = take((2 * (size_t)cap + n_eig) * sizeof(void*)), o_arr = take(4),
                 o_part = take(std::max((size_t)KB * g, mdot_f64_most_partials(cap, n)) * 16);
    Workspace& ws = H.reduction_scratch(std::max<size_t>(1 << 16, off / 16 + 16));
    char* base = ws.partial.as<char>();
    auto* res = reinterpret_cast<double2*>(base + o_res);
    auto* coef = reinterpret_cast<double2*>(base + o_coef);
    auto* dlam = reinterpret_cast<double*>(base + o_lam);
    auto** tabV = reinterpret_cast<double2**>(base + o_tab);
    auto** tabH = tabV + cap;
    auto** tabT = tabH + cap;
    auto* arrived = reinterpret_cast<unsigned int*>(base + o_arr);
    auto* part = reinterpret_cast<double2*>(base + o_part);
    QKG_CUDA(cudaMemsetAsync(arrived, 0, sizeof(unsigned int), st));
    const auto mapped = H.mapped_scalars(2 * n_res);  // pinned landing area of the results
    auto* hres = reinterpret_cast<double2*>(mapped.host);
    auto fetch = [&](size_t count) {
        QKG_CUDA(cudaMemcpyAsync(hres, res, count * sizeof(double2), cudaMemcpyDeviceToHost, st));
        QKG_CUDA(cudaStreamSynchronize(st));
    };
    auto name_vectors = [&] {
        std::vector<double2*> p(2 * (size_t)cap + n_eig, nullptr);
        for (size_t i = 0; i < V.size(); ++i) p[i] = ptr(V[i]);
        for (size_t i = 0; i < HV.size(); ++i) p[cap + i] = ptr(HV[i]);
        for (int i = 0; i < n_eig; ++i) p[2 * (size_t)cap + i] = ptr(T[i]);
        QKG_CUDA(cudaMemcpyAsync(tabV, p.data(), p.size() * sizeof(void*), cudaMemcpyHostToDevice, st));
    };
    const auto* dV = reinterpret_cast<const double2* const*>(tabV);
    const auto* dH = reinterpret_cast<const double2* const*>(tabH);
    auto dots = [&](const double2* const* t, int k, const double2* w, double f, double2* to) {
        const int gm = mdot_f64_chunks(k, n);
        mdot_f64_partials(t, k, w, n, part, gm, st);
        dav_finish<<<k, kT, 0, st>>>(part, gm, f, to);
        QKG_LAUNCHED();
    };

    // seeds: unit vectors at the n_eig smallest diagonal entries
    H.diagonal_f64(ptr(s_diag), st);
    {
        std::vector<cd> d(n);
        const double2* src = ptr(s_diag);
        if (H.permuted()) {
            H.to_reference_f64(src, ptr(s_tmp), st);
            src = ptr(s_tmp);
        }
        QKG_CUDA(cudaMemcpyAsync(d.data(), src, vb, cudaMemcpyDeviceToHost, st));
        QKG_CUDA(cudaStreamSynchronize(st));
        std::vector<double> key(n);
        for (uint64_t i = 0; i < n; ++i) key[i] = f32_stream ? (double)(float)d[i].real() : d[i].real();  // the FP32 engine sorts floats
        const auto di = seed_order(key, n_eig);
        for (int i = 0; i < n_eig; ++i) {
            V.push_back(get());
            HV.push_back(get());
            double2* to = ptr(H.permuted() ? s_tmp : V[i]);
            QKG_CUDA(cudaMemsetAsync(to, 0, vb, st));
            dav_unit<<<1, 1, 0, st>>>(to, di[i]);
            QKG_LAUNCHED();
            if (H.permuted()) H.to_internal_f64(to, ptr(V[i]), st);
            H.apply_f64(ptr(V[i]), ptr(HV[i]), st);
        }
        name_vectors();
    }

    std::vector<std::vector<cd>> rows;  // rows[i][j] = <V_i, HV_j>, j <= i
    int fresh = n_eig;                  // vectors without a row yet
    int added = 0;                      // the last of them that are corrections, with their norms at res[0 ..]
    std::vector<cd> Hs;
    std::vector<double> ev;
    std::vector<std::vector<cd>> evec;
    for (int iter = 0; iter < max_iter; ++iter) {
        // the new vectors' rows: row r of them at res[n_eig + r * cap]
        int m = (int)V.size();
        for (int r = 0; r < fresh; ++r) {
            const int i = m - fresh + r;
            dots(dH, i + 1, ptr(V[i]), 1.0, res + n_eig + (size_t)r * cap);  // <HV_j, V_i>
        }
        fetch((size_t)n_eig + (size_t)fresh * cap);
        {
            std::vector<int> gone;  // vanished corrections, as positions among the new vectors
            for (int r = 0; r < added; ++r)
                if (!(hres[r].x > kDropped)) gone.push_back(fresh - added + r);
            const int first = m - fresh;
            std::vector<int> keep;
            for (int r = 0; r < fresh; ++r)
                if (std::find(gone.begin(), gone.end(), r) == gone.end()) keep.push_back(r);
            for (size_t q = 0; q < keep.size(); ++q) {
                const double2* row = hres + n_eig + (size_t)keep[q] * cap;
                std::vector<cd> col;
                for (int j = 0; j < first; ++j) col.push_back(cd(row[j].x, -row[j].y));
                for (size_t p = 0; p <= q; ++p) col.push_back(cd(row[first + keep[p]].x, -row[first + keep[p]].y));
                rows.push_back(std::move(col));
            }
            for (size_t q = gone.size(); q-- > 0;) {
                const int i = first + gone[q];
                spare.push_back(V[i]);
                spare.push_back(HV[i]);
                V.erase(V.begin() + i);
                HV.erase(HV.begin() + i);
            }
            if (!gone.empty()) name_vectors();
        }
        m = (int)V.size();
        Hs.assign((size_t)m * m, 0.0);
        for (int i = 0; i < m; ++i)
            for (int j = 0; j <= i; ++j) {
                Hs[(size_t)i * m + j] = rows[i][j];
                if (i != j) Hs[(size_t)j * m + i] = std::conj(rows[i][j]);
            }
        hermitian_eig(Hs, m, ev, evec);
        // residuals, their norms, preconditioned corrections
        std::vector<cd> cs((size_t)n_eig * m);
        for (int k = 0; k < n_eig; ++k)
            for (int i = 0; i < m; ++i) cs[(size_t)k * m + i] = evec[k][i];
        QKG_CUDA(cudaMemcpyAsync(coef, cs.data(), cs.size() * sizeof(cd), cudaMemcpyHostToDevice, st));
        QKG_CUDA(cudaMemcpyAsync(dlam, ev.data(), n_eig * sizeof(double), cudaMemcpyHostToDevice, st));
        for (int k0 = 0, nk; k0 < n_eig; k0 += nk) {
            nk = std::min({KB, n_eig - k0, std::max(1, kResidualCoefs / m)});
            auto go = [&](auto kc) {
                constexpr int K = decltype(kc)::value;
                dav_residual<K><<<g, kT, (size_t)K * m * sizeof(double2), st>>>(
                    dV, dH, m, coef + (size_t)k0 * m, dlam + k0, ptr(s_diag), tabT + k0, n, part, arrived, res + k0);
                QKG_LAUNCHED();
            };
            if (nk == 1) go(std::integral_constant<int, 1>{});
            else if (nk == 2) go(std::integral_constant<int, 2>{});
            else if (nk == 3) go(std::integral_constant<int, 3>{});
            else go(std::integral_constant<int, 4>{});
        }
        fetch(n_eig);
        std::vector<int> todo;
        out.residuals.assign(n_eig, 0.0);
        for (int k = 0; k < n_eig; ++k) {
            out.residuals[k] = std::sqrt(hres[k].x);
            if (out.residuals[k] > tol) todo.push_back(k);
        }
        auto ritz = [&](const std::vector<int>& src_list, const std::vector<int>& to, int count) {  // to_k = sum_j s_kj src_j
            const int kc = std::max(1, std::min(8, 1024 / std::max(m, 1)));
            std::vector<double2*> p;
            for (int k = 0; k < count; ++k) p.push_back(ptr(to[k]));
            for (int k0 = 0; k0 < count; k0 += kc)
                mcombine_multi_f64(&src_list == &V ? dV : dH, m, cs.data() + (size_t)k0 * m, p.data() + k0,
                                   std::min(kc, count - k0), n, false, ws, st);
        };
        if (todo.empty() || iter == max_iter - 1) {
            out.iters = iter + 1;
            out.converged = todo.empty();
            out.evals.assign(ev.begin(), ev.begin() + n_eig);
            if (want_vecs) {
                ritz(V, T, n_eig);
                for (int k = 0; k < n_eig; ++k) {
                    const double2* src = ptr(T[k]);
                    if (H.permuted()) {
                        H.to_reference_f64(src, ptr(s_tmp), st);
                        src = ptr(s_tmp);
                    }
                    std::vector<cd> h(n);
                    QKG_CUDA(cudaMemcpyAsync(h.data(), src, vb, cudaMemcpyDeviceToHost, st));
                    QKG_CUDA(cudaStreamSynchronize(st));
                    out.evecs.push_back(std::move(h));
                }
            }
            QKG_CUDA(cudaStreamSynchronize(st));
            out.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
            return out;
        }
        if (V.size() + todo.size() > (size_t)max_sub) {  // restart to the Ritz vectors (:196-211)
            std::vector<int> nv, nh;
            for (int k = 0; k < n_eig; ++k) nv.push_back(get()), nh.push_back(get());
            ritz(V, nv, n_eig);
            ritz(HV, nh, n_eig);
            for (int s : V) spare.push_back(s);
            for (int s : HV) spare.push_back(s);
            V = nv;
            HV = nh;
            rows.clear();
        }
        const bool restarted = rows.empty();
        // the corrections join the basis, each orthogonalised against all before it (:213-223)
        const int kv = (int)V.size();
        for (int k : todo) {
            V.push_back(T[k]);
            HV.push_back(get());
            T[k] = get();
        }
        name_vectors();
        for (size_t q = 0; q < todo.size(); ++q) {
            const int k = kv + (int)q;
            double2* t = ptr(V[k]);
            dots(dV, k, t, -1.0, coef);
            dav_subtract<<<g, kT, (size_t)k * (sizeof(double2) + sizeof(void*)), st>>>(dV, k, coef, t, n, part, arrived, res + q);
            QKG_LAUNCHED();
            dav_scale<<<g, kT, 0, st>>>(res + q, t, n);
            QKG_LAUNCHED();
            H.apply_f64(t, ptr(HV[k]), st);
        }
        added = (int)todo.size();
        fresh = (restarted ? kv : 0) + added;  // after a restart the Ritz vectors' rows are new too
    }
    return out;
}

}  // namespace qkg
