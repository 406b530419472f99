// Host side of the packed SpMV plan (pack.hpp): the blocks and classes of the
// reference order, the terms' classification, and the tables.
#include "pack.hpp"
#include "solvers.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <map>
#include <memory>
#include <tuple>
#include <type_traits>

namespace qkg {
using namespace packk;
namespace {

inline int popc(uint64_t x) { return __builtin_popcountll(x); }

// A compiled term without variable factors: conditions, flips, parity, amplitude.
struct PTerm {
    uint64_t C, V, X, J;
    cd amp;
};

// A term's variable factors are of two kinds: (a0 = -a1) on one bit is a sign,
// so the bit joins the parity mask; a0 = 0 is a condition on its bits.  A
// parity bit that a condition pins is a constant sign.  False: another kind.
bool simplify(const HostTerm& h, PTerm& t, bool& dead) {
    t = {h.C, h.V, h.X, h.J, h.amp};
    dead = false;
    for (const DVar& v : h.vars) {
        const cd a0(v.a0r, v.a0i), a1(v.a1r, v.a1i);
        if (a0 == cd(0.0)) {  // all of sm's bits of s ^ pf set
            const uint64_t need = ~v.pf & v.sm, both = t.C & v.sm;
            if ((t.V & both) != (need & both)) { dead = true; return true; }
            t.C |= v.sm;
            t.V = (t.V & ~v.sm) | need;
            t.amp *= a1;
        } else if (a0 == -a1 && popc(v.sm) == 1) {
            // a1 where the bit of s ^ pf is 1: (-1)^bit(s) times a0 (pf = 0) or a1 (pf = 1)
            t.J ^= v.sm;
            t.amp *= (v.pf & v.sm) ? a1 : a0;
        } else {
            return false;
        }
    }
    const uint64_t pinned = t.J & t.C;
    if (popc(pinned & t.V) & 1) t.amp = -t.amp;
    t.J &= ~pinned;
    return true;
}

// parity of 16 bits without a population count (which takes Arm a trip through its vector unit)
inline uint32_t parity16(uint32_t x) {
    x ^= x >> 8;
    x ^= x >> 4;
    return (0x6996u >> (x & 15u)) & 1u;
}

int top_bit(uint64_t x) { return x ? 63 - __builtin_clzll(x) : -1; }

// Appends v to the image of a plan's tables; returns its offset (16-byte aligned).
template <class T>
size_t append(std::vector<char>& image, const std::vector<T>& v) {
    const size_t at = (image.size() + 15) / 16 * 16;
    image.resize(at + v.size() * sizeof(T));
    if (!v.empty()) std::memcpy(image.data() + at, v.data(), v.size() * sizeof(T));
    return at;
}

constexpr size_t kMaxTable = 32ull << 20;  // uint2 entries of all tables (256 MB)

// A vector whose resize leaves new elements as they are: the threads that write them touch
// their pages first.
template <class T>
struct NoInit : std::allocator<T> {
    template <class U> struct rebind { using other = NoInit<U>; };
    template <class U> void construct(U* p) { ::new (static_cast<void*>(p)) U; }
    template <class U, class A> void construct(U* p, A&& a) { ::new (static_cast<void*>(p)) U(std::forward<A>(a)); }
};
using Entries = std::vector<uint16_t, NoInit<uint16_t>>;

}  // namespace

bool PackTables::build(const Basis& B, SiteKind site, const std::vector<Term>& terms, AmpMode at_least) {
    *this = PackTables();
    dim = B.dim;
    const int nb = B.nbits;
    if (B.rank_kind != RANK_TABLE || nb > 32 || B.dim == 0 || B.dim >= (1ull << 31)) return false;
    // popcount groups in the reference encoding
    uint64_t gm[2] = {0, 0};
    for (int g = 0; g < B.ngroups; ++g) gm[g] = B.to_reference(B.gmask[g]);
    const int ng = B.ngroups;
    // --- terms
    std::vector<PTerm> list;
    for (const HostTerm& h : compile_terms(B, site, terms, true)) {
        if (h.X == 0) continue;
        PTerm t;
        bool dead;
        if (!simplify(h, t, dead)) return false;
        if (!dead) list.push_back(t);
    }
    // --- the split: the most inner bits whose largest class keeps to kClassTarget
    // rows (a block of x then fits in L1 beside its neighbours') and whose tables
    // stay below a quarter of the sector's rows (they are built for every
    // Hamiltonian), whole sites for interleaved bases
    const int unit = B.split ? 2 : 1;
    // rows of the largest class that a sector leaves, and of all of them
    auto class_rows = [&](int n_in, bool all) {
        uint64_t most = 1;
        uint64_t free_bits = (1ull << n_in) - 1;
        for (int g = 0; g < ng; ++g) {
            const int in = popc(gm[g] & ((1ull << n_in) - 1)), out = popc(gm[g]) - in;
            uint64_t m = 0;
            for (int k = 0; k <= in; ++k)
                if (B.gpop[g] - k >= 0 && B.gpop[g] - k <= out) m = all ? m + binom(in, k) : std::max(m, binom(in, k));
            most *= m;
            free_bits &= ~gm[g];
        }
        return most << popc(free_bits);
    };
    int n_in = std::min(nb, unit);
    while (n_in + unit <= nb && n_in + unit <= 16 && class_rows(n_in + unit, false) <= kClassTarget &&
           class_rows(n_in + unit, true) <= std::max<uint64_t>(4096, B.dim / 4))
        n_in += unit;
    const int n_out = nb - n_in;
    if (n_out > 22 || class_rows(n_in, false) > 0xFFFE) return false;
    const uint64_t inm = (1ull << n_in) - 1;
    // --- classes of inner configurations (by the groups' popcounts)
    const int w1 = ng > 1 ? popc(gm[1] & inm) + 1 : 1, w0 = ng > 0 ? popc(gm[0] & inm) + 1 : 1;
    const int ncls = w0 * w1;
    auto class_of_inner = [&](uint64_t b) {
        const int k0 = ng > 0 ? popc(b & gm[0]) : 0, k1 = ng > 1 ? popc(b & gm[1]) : 0;
        return k0 * w1 + k1;
    };
    auto class_of_outer = [&](uint64_t a) {  // the class that block a holds, -1: none
        const uint64_t s = a << n_in;
        int k0 = 0, k1 = 0;
        if (ng > 0) { k0 = B.gpop[0] - popc(s & gm[0]); if (k0 < 0 || k0 >= w0) return -1; }
        if (ng > 1) { k1 = B.gpop[1] - popc(s & gm[1]); if (k1 < 0 || k1 >= w1) return -1; }
        return k0 * w1 + k1;
    };
    std::vector<std::vector<uint32_t>> members(ncls);
    std::vector<uint32_t> place(1ull << n_in);  // class << 16 | rank in it
    for (uint64_t b = 0; b <= inm; ++b) {
        const int c = class_of_inner(b);
        place[b] = (uint32_t)c << 16 | (uint32_t)std::min<size_t>(members[c].size(), 0xFFFF);
        members[c].push_back((uint32_t)b);
    }
    const uint64_t n_a = 1ull << n_out;
    std::vector<uint32_t> off(n_a + 1, 0);
    std::vector<int> bcls(n_a, -1);
    std::vector<char> present(ncls, 0);
    uint64_t total = 0;
    for (uint64_t a = 0; a < n_a; ++a) {
        off[a] = (uint32_t)total;
        bcls[a] = class_of_outer(a);
        if (bcls[a] < 0) continue;
        present[bcls[a]] = 1;
        total += members[bcls[a]].size();
    }
    off[n_a] = (uint32_t)total;
    QKG_REQUIRE(total == B.dim, "packed plan: blocks do not add up to the sector");
    // --- terms by class, merged by their flips
    struct Group {
        uint64_t X;
        std::vector<PTerm> t;
    };
    std::vector<Group> inner, outer, mixed;
    auto add = [](std::vector<Group>& v, const PTerm& t) {
        for (auto& g : v)
            if (g.X == t.X) { g.t.push_back(t); return; }
        v.push_back({t.X, {t}});
    };
    for (const PTerm& t : list) {
        const uint64_t m = t.X | t.C | t.J;
        if (!(m & ~inm)) add(inner, t);
        else if (!(m & inm)) add(outer, t);
        else add(mixed, t);
    }
    // far flips first: the lanes of a warp (consecutive rows) share their high
    // bits, so their first entries mostly flip the same bond and read one run
    std::stable_sort(inner.begin(), inner.end(), [](const Group& x, const Group& y) { return top_bit(x.X) > top_bit(y.X); });
    for (const auto& g : mixed)
        if (g.t.size() > 24) return false;
    real = true;
    for (const auto* v : {&inner, &outer, &mixed})
        for (const auto& g : *v)
            for (const auto& t : g.t) real = real && t.amp.imag() == 0.0;
    auto sum_at = [](const std::vector<PTerm>& ts, uint64_t s, cd& amp) {  // amplitude of the merged terms on s
        bool any = false;
        for (const auto& t : ts)
            if ((s & t.C) == t.V) {
                const cd v = t.J && (popc(s & t.J) & 1) ? -t.amp : t.amp;
                amp = any ? amp + v : v;
                any = true;
            }
        return any;
    };
    // --- tables: a 16-bit rank and an amplitude index per entry, packed by mode at the end.
    // Each class's inner table and each straddling table is built by one thread with amplitude
    // indexes of its own; they are joined in order, so the outcome is that of one thread.
    struct Codes {
        std::vector<cd> amps;
        std::map<std::pair<uint64_t, uint64_t>, uint32_t> id;
        cd seen[4];  // the last ones looked up
        uint16_t seen_id[4];
        int n_seen = 0, next_seen = 0;
        bool too_many = false;
        uint16_t operator()(cd a) {
            for (int i = 0; i < n_seen; ++i)
                if (seen[i] == a) return seen_id[i];
            uint64_t k[2];
            const double re = a.real() + 0.0, im = a.imag() + 0.0;  // no negative zeros
            std::memcpy(k, &re, 8);
            std::memcpy(k + 1, &im, 8);
            auto it = id.find({k[0], k[1]});
            if (it == id.end()) {
                if (amps.size() >= 4096) { too_many = true; return 0; }
                it = id.emplace(std::make_pair(k[0], k[1]), (uint32_t)amps.size()).first;
                amps.push_back(cd(re, im));
            }
            seen[next_seen] = cd(re, im);
            seen_id[next_seen] = (uint16_t)it->second;
            n_seen = std::min(n_seen + 1, 4);
            next_seen = (next_seen + 1) & 3;
            return (uint16_t)it->second;
        }
    };
    // the magnitude of a set of amplitudes (-1: none), and which signs occur; one = false:
    // several magnitudes
    struct Mag {
        double mag = -1.0;
        bool plus = false, minus = false, one = true;
        void add(const std::vector<cd>& amps) {
            for (const cd& a : amps) {
                const double v = a.real();
                if (mag < 0.0) mag = std::abs(v);
                one = one && std::abs(v) == mag;
                (std::signbit(v) ? minus : plus) = true;
            }
        }
    };
    struct Built {
        Entries er, ec;  // entries: [(slot * 32 + lane) * 4 + q]
        std::vector<uint2> tile;
        Codes code;
        size_t longest = 0;  // inner entries of a row
        size_t at = 0;       // its first entry among all tables'
        bool any = false;    // whether it has entries at all
    };
    Codes code;      // of all tables
    Entries er, ec;  // entries of all tables
    // body(i) for i < n on several threads where there is work for them: a region costs some 20 us,
    // 20,000 rows tested 70 us (16 cores: 12-site Hubbard ring 5.9 to 2.1 ms, with next-nearest hops
    // 9.8 to 4.1, 20-site ring 0.86 to 0.46; one class, 14-site ring, 0.22)
    auto threads = [](size_t n, size_t work, auto&& body) {
        std::exception_ptr failed;
#pragma omp parallel for schedule(dynamic) if (n > 1 && work > 20000)
        for (long long i = 0; i < (long long)n; ++i) {
            try {
                body((size_t)i);
            } catch (...) {
#pragma omp critical(qkg_pack_plan)
                failed = std::current_exception();
            }
        }
        if (failed) std::rethrow_exception(failed);
    };
    // appends the entries of the tables that have any, in order
    auto join = [&](std::vector<Built>& built) {
        std::vector<std::vector<uint16_t>> to(built.size());  // codes, empty: the same
        size_t n = er.size();
        for (size_t t = 0; t < built.size(); ++t) {
            Built& b = built[t];
            if (!b.any) continue;
            bool same = true;
            for (size_t i = 0; i < b.code.amps.size(); ++i) {
                to[t].push_back(code(b.code.amps[i]));
                same = same && to[t][i] == i;
            }
            if (same) to[t].clear();
            b.at = n;
            n += b.er.size();
            if (n / 4 > kMaxTable || code.too_many || b.code.too_many) return false;
        }
        const size_t added = n - er.size();
        er.resize(n);
        ec.resize(n);
        threads(built.size(), added, [&](size_t t) {
            const Built& b = built[t];
            if (!b.any) return;
            std::copy(b.er.begin(), b.er.end(), er.begin() + b.at);
            if (to[t].empty()) {
                std::copy(b.ec.begin(), b.ec.end(), ec.begin() + b.at);
            } else {
                for (size_t e = 0; e < b.ec.size(); ++e) ec[b.at + e] = b.er[e] == kNone16 ? (uint16_t)0 : to[t][b.ec[e]];
            }
        });
        return true;
    };
    std::vector<uint32_t> ctile(ncls, 0);  // first inner tile of a class
    size_t longest = 0;                    // inner entries of a row
    Mag inner_mag;
    auto tiles_of = [&](int c) { return (uint32_t)((members[c].size() + kTile - 1) / kTile); };
    // emit(row, target rank, amplitude index) for the rows of class c on which the merged
    // terms ts give an entry in class c2.  A few terms have a few sums: the amplitude index is
    // looked up by which terms hold, and with which signs.
    auto each = [&](int c, int c2, const std::vector<PTerm>& ts, uint32_t flip, Codes& code_of, auto&& emit) {
        const int T = (int)ts.size();
        const bool few = T <= 5;
        int sums[1 << 10];
        if (few) std::fill(sums, sums + ((size_t)1 << (2 * T)), -1);
        uint32_t C[5], V[5], J[5];
        for (int k = 0; few && k < T; ++k) C[k] = (uint32_t)ts[k].C, V[k] = (uint32_t)ts[k].V, J[k] = (uint32_t)ts[k].J;
        const uint32_t *mem = members[c].data(), *at = place.data();
        const uint32_t n = (uint32_t)members[c].size();
        for (uint32_t r = 0; r < n; ++r) {
            const uint32_t bb = mem[r];
            cd amp;
            if (few) {
                uint32_t key = 0;
                for (int k = 0; k < T; ++k)
                    if ((bb & C[k]) == V[k]) key |= (J[k] && parity16(bb & J[k]) ? ((1u << T) | 1u) : 1u) << k;
                if (!key) continue;
                const uint32_t to = at[bb ^ flip];
                if ((to >> 16) != (uint32_t)c2) continue;
                int& id = sums[key];
                if (id < 0) {
                    sum_at(ts, bb, amp);
                    id = code_of(amp);
                }
                emit(r, (uint16_t)to, (uint16_t)id);
            } else {
                const uint32_t to = at[bb ^ flip];
                if (!sum_at(ts, bb, amp) || (to >> 16) != (uint32_t)c2) continue;
                emit(r, (uint16_t)to, code_of(amp));
            }
        }
    };
    if (inner.size() > 255) return false;
    {
        std::vector<int> list;       // the classes that occur
        std::vector<size_t> row_at;  // their first rows in the scratch below
        size_t rows = 0;
        for (int c = 0; c < ncls; ++c)
            if (present[c]) {
                list.push_back(c);
                row_at.push_back(rows);
                rows += members[c].size();
            }
        // rows: entries in group order (not initialised), and how many
        const size_t stride = inner.size();
        const std::unique_ptr<uint16_t[]> rows_r(new uint16_t[rows * stride]), rows_c(new uint16_t[rows * stride]);
        std::vector<uint16_t> rows_n(rows, 0);
        std::vector<Built> built(list.size());
        threads(list.size(), rows * inner.size(), [&](size_t n) {
            const int c = list[n];
            Built& b = built[n];
            const size_t W = members[c].size();
            uint16_t *rr = rows_r.get() + row_at[n] * stride, *rc = rows_c.get() + row_at[n] * stride, *rn = rows_n.data() + row_at[n];
            for (const auto& g : inner)
                each(c, c, g.t, (uint32_t)g.X, b.code, [stride, R = rr, A = rc, N = rn](uint32_t r, uint16_t to, uint16_t code) {
                    const size_t at = r * stride + N[r]++;
                    R[at] = to;
                    A[at] = code;
                });
            b.er.reserve((size_t)tiles_of(c) * kTile * ((stride + 7) / 8 * 4));
            b.ec.reserve((size_t)tiles_of(c) * kTile * ((stride + 7) / 8 * 4));
            for (uint32_t t = 0; t < tiles_of(c); ++t) {
                uint2 rec = make_uint2((uint32_t)(b.er.size() / kTile), 0u);
                for (uint32_t q = 0; q < 4; ++q) {
                    const size_t r0 = (size_t)t * kTile + q * 32, r1 = std::min(W, r0 + 32);
                    size_t most = 0;
                    for (size_t r = r0; r < r1; ++r) most = std::max<size_t>(most, rn[r]);
                    rec.y |= (uint32_t)most << (8 * q);
                    b.longest = std::max(b.longest, most);
                    const size_t e0 = b.er.size(), nq = (most + 3) / 4;
                    b.er.resize(e0 + nq * kTile, (uint16_t)kNone16);
                    b.ec.resize(b.er.size(), 0);
                    for (size_t r = r0; r < r1; ++r)
                        for (size_t j = 0; j < rn[r]; j += 4) {  // a quad, or the rest of the row
                            const size_t at = e0 + ((j / 4) * 32 + (r - r0)) * 4, k = std::min<size_t>(4, rn[r] - j) * 2;
                            std::memcpy(&b.er[at], &rr[r * stride + j], k);
                            std::memcpy(&b.ec[at], &rc[r * stride + j], k);
                        }
                }
                b.tile.push_back(rec);
            }
            b.any = true;
        });
        if (!join(built)) return false;
        for (size_t n = 0; n < list.size(); ++n) {
            const Built& b = built[n];
            ctile[list[n]] = (uint32_t)tile.size();
            for (uint2 rec : b.tile) tile.push_back(make_uint2(rec.x + (uint32_t)(b.at / kTile), rec.y));
            longest = std::max(longest, b.longest);
            inner_mag.add(b.code.amps);
        }
    }
    // the kernels read one quad ahead
    er.resize(er.size() + kTile, (uint16_t)kNone16);
    ec.resize(er.size(), 0);
    // --- per block: outer entries and straddling tables
    blk.assign(n_a, Blk{});
    struct O { int32_t d; cd a; };
    struct M { uint32_t tab, off; };  // tab: index in `tables` first, its entries in the end
    std::vector<O> olist;
    std::vector<M> slist;
    struct Table {
        int c, c2;
        uint32_t group, valid, neg;
        uint32_t id;  // first entry / 4 (uint2 index), kNoTable: no row of the class has an entry
    };
    constexpr uint32_t kNoTable = 0xFFFFFFFFu;
    std::vector<Table> tables;
    // by class and group, a few each: (valid, neg, c2) -> index in tables
    std::vector<std::map<std::tuple<uint32_t, uint32_t, int>, uint32_t>> known((size_t)ncls * mixed.size());
    std::vector<std::pair<uint32_t, Mag>> table_mag;                        // of each straddling table
    size_t outer_most = 0, mixed_most = 0;
    for (uint64_t a = 0; a < n_a; ++a) {
        blk[a].o0 = (uint32_t)olist.size();
        blk[a].m0 = (uint32_t)slist.size();
        if (bcls[a] >= 0) {
            const uint64_t sa = a << n_in;
            for (const auto& g : outer) {
                const uint64_t a2 = a ^ (g.X >> n_in);
                cd amp;
                if (bcls[a2] != bcls[a] || !sum_at(g.t, sa, amp)) continue;
                olist.push_back({(int32_t)((int64_t)off[a2] - (int64_t)off[a]), amp});
            }
            for (size_t gi = 0; gi < mixed.size(); ++gi) {
                const auto& g = mixed[gi];
                const uint64_t a2 = a ^ (g.X >> n_in);
                if (bcls[a2] < 0) continue;
                uint32_t valid = 0, neg = 0;
                for (size_t k = 0; k < g.t.size(); ++k)
                    if ((sa & g.t[k].C & ~inm) == (g.t[k].V & ~inm)) {
                        valid |= 1u << k;
                        const uint64_t J = g.t[k].J & ~inm;
                        if (J && (popc(sa & J) & 1)) neg |= 1u << k;
                    }
                if (!valid) continue;
                const auto [it, fresh] = known[bcls[a] * mixed.size() + gi].try_emplace({valid, neg, bcls[a2]}, (uint32_t)tables.size());
                if (fresh) tables.push_back({bcls[a], bcls[a2], (uint32_t)gi, valid, neg, kNoTable});
                slist.push_back({it->second, off[a2]});
            }
        }
        blk[a].o1 = (uint32_t)olist.size();
        blk[a].m1 = (uint32_t)slist.size();
        outer_most = std::max<size_t>(outer_most, blk[a].o1 - blk[a].o0);
        if (olist.size() > 0x7FFFFFFFull || slist.size() > 0x7FFFFFFFull) return false;
    }
    {
        size_t all = er.size();
        for (const Table& t : tables) all += (size_t)tiles_of(t.c) * kTile;
        er.reserve(std::min(all, 4 * kMaxTable));
        ec.reserve(std::min(all, 4 * kMaxTable));
    }
    // the tables, some at a time (what is built before it is joined stays below 8 M entries)
    for (size_t t0 = 0, t1; t0 < tables.size(); t0 = t1) {
        size_t rows = 0, work = 0;
        for (t1 = t0; t1 < tables.size() && rows < (8u << 20); ++t1) {
            rows += (size_t)tiles_of(tables[t1].c) * kTile;
            work += members[tables[t1].c].size() * mixed[tables[t1].group].t.size();
        }
        std::vector<Built> built(t1 - t0);
        threads(t1 - t0, work, [&](size_t n) {
            const Table& tb = tables[t0 + n];
            const Group& g = mixed[tb.group];
            Built& b = built[n];
            std::vector<PTerm> ts;
            for (size_t k = 0; k < g.t.size(); ++k)
                if (tb.valid >> k & 1) {
                    PTerm t = g.t[k];
                    t.C &= inm;
                    t.V &= inm;
                    t.J &= inm;
                    if (tb.neg >> k & 1) t.amp = -t.amp;
                    ts.push_back(t);
                }
            b.er.resize((size_t)tiles_of(tb.c) * kTile, (uint16_t)kNone16);
            b.ec.resize(b.er.size(), 0);
            bool any = false;
            each(tb.c, tb.c2, ts, (uint32_t)(g.X & inm), b.code, [&any, R = b.er.data(), A = b.ec.data()](uint32_t r, uint16_t to, uint16_t code) {
                const uint32_t t = r / kTile, i = r % kTile;
                const size_t at = (t * 32 + (i & 31)) * 4 + (i >> 5);
                R[at] = to;
                A[at] = code;
                any = true;
            });
            b.any = any;
        });
        if (!join(built)) return false;
        for (size_t n = 0; n < built.size(); ++n) {
            if (!built[n].any) continue;
            tables[t0 + n].id = (uint32_t)(built[n].at / 4);
            Mag m;
            m.add(built[n].code.amps);
            table_mag.push_back({tables[t0 + n].id, m});
        }
    }
    // the blocks' entries of tables that are there
    {
        uint32_t n = 0;
        for (uint64_t a = 0; a < n_a; ++a) {
            const uint32_t m0 = n;
            for (uint32_t k = blk[a].m0; k < blk[a].m1; ++k)
                if (tables[slist[k].tab].id != kNoTable) slist[n++] = {tables[slist[k].tab].id, slist[k].off};
            blk[a].m0 = m0;
            blk[a].m1 = n;
            mixed_most = std::max<size_t>(mixed_most, n - m0);
        }
        slist.resize(n);
    }
    amps = code.amps;
    // an empty slot adds amplitude * 0: that is nothing only for finite amplitudes, in FP32 too
    auto finite32 = [](cd a) { return std::isfinite((float)a.real()) && std::isfinite((float)a.imag()); };
    for (const cd& a : amps)
        if (!finite32(a)) return false;
    for (const auto& o : olist)
        if (!finite32(o.a)) return false;
    // --- amplitude mode: one magnitude per inner table and per straddling table?
    size_t widest = 0;
    for (int c = 0; c < ncls; ++c)
        if (present[c]) widest = std::max(widest, members[c].size());
    bool one = real && inner_mag.one, sgn = inner_mag.plus && inner_mag.minus;
    const double umag = inner_mag.mag;
    std::map<uint32_t, double> smag;  // straddling table -> its amplitude (its magnitude where signs differ)
    equal = real;
    u = umag < 0.0 ? 0.0 : (inner_mag.plus ? umag : -umag);
    for (const auto& t : table_mag) {
        one = one && t.second.one;
        sgn = sgn || (t.second.plus && t.second.minus);
    }
    sgn = sgn || at_least == AMP_SIGNED;
    if (sgn && widest > 0x7FFF) one = false;
    mode = one && at_least != AMP_CODED ? (sgn ? AMP_SIGNED : AMP_UNIFORM) : AMP_CODED;
    if (mode == AMP_CODED && amps.size() > (size_t)kMaxAmps) return false;
    if (mode != AMP_CODED) {
        if (mode == AMP_SIGNED) {
            // rank | sign << 15; amplitudes are magnitudes
            std::vector<uint16_t> bit(amps.size());
            for (size_t i = 0; i < amps.size(); ++i) bit[i] = std::signbit(amps[i].real()) ? 0x8000u : 0u;
            constexpr size_t kChunk = 1 << 14;
            threads((er.size() + kChunk - 1) / kChunk, er.size(), [&](size_t n) {
                for (size_t e = n * kChunk; e < std::min(er.size(), (n + 1) * kChunk); ++e)
                    er[e] = er[e] == kNone16 ? (uint16_t)kNone15 : (uint16_t)(er[e] | bit[ec[e]]);
            });
            u = std::max(umag, 0.0);
        }
        for (const auto& t : table_mag)
            smag[t.first] = mode == AMP_SIGNED || t.second.plus ? t.second.mag : -t.second.mag;
        double mag = umag;
        auto same = [&](double v) {
            v = std::abs(v);
            if (mag < 0.0) mag = v;
            if (v != mag) equal = false;
        };
        for (const auto& o : olist) same(o.a.real());
        for (const auto& s : smag) same(s.second);
        if (umag < 0.0) u = std::max(mag, 0.0);  // no inner entry: the common magnitude
    } else {
        equal = false;
    }
    if (longest + outer_most + mixed_most > (size_t)kMaxRowEntries || (u != 0.0 && std::abs(u) < kMinEqual)) equal = false;
    // --- items: the tiles of every block; blocks that a straddling flip of the
    // highest outer bit joins run side by side, so that the rows they gather from
    // one another are still in L2
    int pair_bit = -1;
    for (const auto& g : mixed) pair_bit = std::max(pair_bit, top_bit(g.X >> n_in));
    std::vector<uint32_t> order;
    const uint32_t pair = pair_bit >= 0 ? 1u << pair_bit : 0u;
    for (uint64_t a = 0; a < n_a; ++a) {
        if (a & pair) continue;  // comes with its partner
        if (bcls[a] >= 0) order.push_back((uint32_t)a);
        if (pair && bcls[a | pair] >= 0) order.push_back((uint32_t)a | pair);
    }
    size_t n_tiles = 0;
    for (uint32_t a : order) n_tiles += tiles_of(bcls[a]);
    items.reserve(n_tiles);
    for (uint32_t a : order) {
        const size_t W = members[bcls[a]].size();
        for (size_t t = 0; t * kTile < W; ++t)
            items.push_back({(uint32_t)(off[a] + t * kTile), a, ctile[bcls[a]] + (uint32_t)t,
                             (uint32_t)(t << 8 | std::min<size_t>(kTile, W - t * kTile))});
    }
    // --- the packed tables
    tab.resize(er.size() / 4);
    if (!er.empty()) std::memcpy(tab.data(), er.data(), er.size() * 2);
    if (mode == AMP_CODED) {
        codes.resize(er.size() / 4);
        for (size_t e = 0; e < codes.size(); ++e)
            codes[e] = (uint32_t)ec[4 * e] | (uint32_t)ec[4 * e + 1] << 8 | (uint32_t)ec[4 * e + 2] << 16 | (uint32_t)ec[4 * e + 3] << 24;
    }
    out.reserve(olist.size());
    str.reserve(slist.size());
    for (const auto& o : olist) out.push_back({o.d, 0u, o.a.real(), o.a.imag()});
    for (const auto& m : slist) {
        const double v = mode == AMP_CODED ? 0.0 : smag[m.tab];
        str.push_back({m.tab, m.off, v, 0.0});
    }
    return true;
}

void PackTables::apply_host(const cd* x, cd* y) const {
    auto in = [](bool ok) { QKG_REQUIRE(ok, "packed tables: index out of range"); };
    for (const Item& it : items) {
        const uint32_t cnt = it.tc & 0xFFu, tin = it.tc >> 8;
        in(it.a < blk.size() && it.tile < tile.size() && cnt <= (uint32_t)kTile);
        const Blk b = blk[it.a];
        in(b.o1 <= out.size() && b.m1 <= str.size() && tin * (uint64_t)kTile <= it.row0);
        for (uint32_t i = 0; i < (uint32_t)kTile; ++i) {
            const uint32_t lane = i & 31u, q = i >> 5;
            const uint64_t row = (uint64_t)it.row0 + i;
            cd s = 0.0;
            if (i < cnt)
                for (uint32_t k = b.o0; k < b.o1; ++k) {
                    const int64_t t = (int64_t)row + out[k].delta;
                    in(row < dim && t >= 0 && t < (int64_t)dim);
                    s += cd(out[k].ar, out[k].ai) * x[t];
                }
            auto entry = [&](uint64_t at, uint32_t k, uint64_t base, double amp) {
                in(at < tab.size() && k < 4);
                const uint32_t w = (k & 2u) ? tab[at].y : tab[at].x;
                uint32_t r = (k & 1u) ? w >> 16 : w & 0xFFFFu;
                cd a = amp;
                if (mode == AMP_SIGNED) {
                    if (r & 0x8000u) a = -a;
                    r &= 0x7FFFu;
                    if (r == kNone15) return;
                } else if (r == kNone16) {
                    return;
                }
                if (mode == AMP_CODED) {
                    in(at < codes.size());
                    const uint32_t c = (codes[at] >> (8 * k)) & 0xFFu;
                    in(c < amps.size());
                    a = amps[c];
                }
                in(i < cnt && base + r < dim);  // rows past the block's end have no entries
                s += a * x[base + r];
            };
            uint64_t quad = tile[it.tile].x;
            for (uint32_t g = 0; g < q; ++g) quad += (((tile[it.tile].y >> (8 * g)) & 0xFFu) + 3u) / 4u;
            const uint32_t slots = (tile[it.tile].y >> (8 * q)) & 0xFFu;
            for (uint32_t j = 0; j < slots; ++j)
                entry((quad + j / 4) * 32 + lane, j & 3u, it.row0 - tin * (uint64_t)kTile, u);
            in((quad + (slots + 3) / 4) * 32 + lane < tab.size());  // the quad read ahead
            for (uint32_t k = b.m0; k < b.m1; ++k) entry(str[k].tab + tin * 32ull + lane, q, str[k].off, str[k].ar);
            if (i < cnt) y[row] = s;
        }
    }
}

PackPlan::PackPlan(const PackTables& t)
    : real_(t.real), equal_(t.equal), mode_(t.mode), n_items_((uint32_t)t.items.size()), n_amps_((int)t.codes.size() ? (int)t.amps.size() : 0), u_(t.u) {
    std::vector<char> image;
    items_ = append(image, t.items);
    blk_ = append(image, t.blk);
    tile_ = append(image, t.tile);
    tab_ = append(image, t.tab);
    out64_ = append(image, t.out);
    str64_ = append(image, t.str);
    std::vector<Out<float>> o32;
    for (const auto& o : t.out) o32.push_back({o.delta, 0u, (float)o.ar, (float)o.ai});
    std::vector<Str<float>> s32;
    for (const auto& s : t.str) s32.push_back({s.tab, s.off, (float)s.ar, (float)s.ai});
    out32_ = append(image, o32);
    str32_ = append(image, s32);
    if (mode_ == AMP_CODED) {
        codes_ = append(image, t.codes);
        std::vector<float2> a32;
        std::vector<double2> a64;
        for (const cd& a : t.amps) {
            a32.push_back(make_float2((float)a.real(), (float)a.imag()));
            a64.push_back(make_double2(a.real(), a.imag()));
        }
        amps32_ = append(image, a32);
        amps64_ = append(image, a64);
    }
    all_.alloc(std::max<size_t>(16, image.size()));
    if (!image.empty()) QKG_CUDA(cudaMemcpy(all_.p, image.data(), image.size(), cudaMemcpyHostToDevice));
}

int packed_apply_host(const Basis& B, SiteKind site, const std::vector<Term>& terms, const double* x, double* y) {
    PackTables t;
    if (!t.build(B, site, terms)) return -1;
    t.apply_host(reinterpret_cast<const cd*>(x), reinterpret_cast<cd*>(y));
    return (int)t.mode + (t.equal ? 4 : 0) + (t.real ? 0 : 8);
}

template <class A>
void PackPlan::params(Params<A>& p) const {
    p = Params<A>{};
    const bool d = sizeof(A) == 8;
    p.items = at<Item>(items_);
    p.n_items = n_items_;
    p.blk = at<Blk>(blk_);
    p.out = at<Out<A>>(d ? out64_ : out32_);
    p.str = at<Str<A>>(d ? str64_ : str32_);
    p.tile = at<uint2>(tile_);
    p.tab = at<uint2>(tab_);
    p.codes = mode_ == AMP_CODED ? at<uint32_t>(codes_) : nullptr;
    p.amps = mode_ == AMP_CODED ? at<A>(d ? amps64_ : amps32_) : nullptr;
    p.n_amps = n_amps_;
    p.u = (A)u_;
    // u 2^-56 2^(e - 1023) is a normal number for the exponents that the integer sums keep
    p.e_min = std::max(64, u_ != 0.0 ? 57 - std::ilogb(u_) : 0);
}
template void PackPlan::params<float>(Params<float>&) const;
template void PackPlan::params<double>(Params<double>&) const;

}  // namespace qkg
