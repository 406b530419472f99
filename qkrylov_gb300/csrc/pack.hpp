// The packed SpMV plan: H on vectors in the reference's own order (ascending
// states), with every off-diagonal entry of a row listed as a 16-bit rank.
//
// States are split in the reference encoding, s = a << n_in | b.  The states of
// one outer part a are one contiguous block, and the inner parts b of a block
// are those of one class (the popcounts that the sector leaves for b), in
// ascending order, so block a of the vector is the class's list of inner parts.
// A term whose flips, conditions and signs touch inner bits only becomes an
// entry of the class's table (target rank in the same block); one that touches
// outer bits only is a uniform offset for the whole block; any other
// (straddling) term is a per-class table of target ranks in another block,
// whose offset and amplitude the block lists.  Terms with the same flips are
// merged into one entry.
#pragma once

#include "fast_common.cuh"

#include <vector>

namespace qkg {
namespace packk {

constexpr uint32_t kClassTarget = 5000;  // rows of the largest inner class aimed at
constexpr int kTile = 128;        // rows of a table tile: one warp, four rows a lane
constexpr uint32_t kNone16 = 0xFFFFu, kNone15 = 0x7FFFu;
constexpr int kMaxAmps = 256;     // distinct amplitudes of the coded form
constexpr double kMinEqual = 0x1p-900;
constexpr int kMaxRowEntries = 63;  // entries a row of the integer-aligned FP64 sum may have

// How the amplitudes of table entries are given.
//   UNIFORM: one real amplitude for every inner entry, one for each straddling
//            table; 16-bit ranks.
//   SIGNED:  the same with a sign per entry (bit 15); 15-bit ranks.
//   CODED:   an 8-bit code per entry into a list of amplitudes.
enum AmpMode : int { AMP_UNIFORM = 0, AMP_SIGNED = 1, AMP_CODED = 2 };

// One warp's rows: `count` (<= kTile) rows from row0 in block a; tile = its
// inner table tile, tc = (tile index inside the class) << 8 | count.
struct Item {
    uint32_t row0, a, tile, tc;
};
// Ranges of block a's outer entries and straddling tables.
struct Blk {
    uint32_t o0, o1, m0, m1;
};
template <class A>
struct alignas(16) Out {  // outer entry: row offset of its target, amplitude
    int32_t delta;
    uint32_t pad;
    A ar, ai;
};
template <class A>
struct alignas(16) Str {  // straddling entry: its table, its target block's offset, amplitude
    uint32_t tab, off;
    A ar, ai;
};

template <class A>
struct Params {
    const Item* items;
    uint32_t n_items;
    const Blk* blk;
    const Out<A>* out;
    const Str<A>* str;
    // inner tile: x = its first quad, byte q of y = the slots of rows q * 32 ..
    // q * 32 + 31.  Quads follow one another row group by row group, ceil(slots
    // / 4) of them each; quad k is tab[(x + k) * 32 + lane]: four 16-bit entries of
    // one row, filled from the first.
    const uint2* tile;
    const uint2* tab;       // straddling tables: the four rows lane + 32 q of a tile
    const uint32_t* codes;  // CODED: four 8-bit codes, indexed like tab
    const A* amps;          // CODED: (re, im) pairs
    int n_amps;
    A u;                    // UNIFORM / SIGNED: the inner amplitude
    int e_min;              // integer sums: exponents below are left to the FP64 pipe
    int diag_mode, cdiag;   // cdiag: the diagonal has imaginary parts
    const void* dcode;
    const A* dtab;
    const LzOperands* lz;   // Lanczos mode, as FastParams::lz
    double2* apart;
    LzDev fin;              // st set: the last CTA adds the partials and sets alpha
};

}  // namespace packk

// The tables as the host builds them.
struct PackTables {
    packk::AmpMode mode = packk::AMP_UNIFORM;
    bool real = true;
    // every entry has the same |amplitude| and rows are short enough: the FP64
    // kernel sums aligned integers (not for magnitudes below kMinEqual, 0 apart)
    bool equal = false;
    double u = 0.0;
    uint64_t dim = 0;
    std::vector<packk::Item> items;
    std::vector<packk::Blk> blk;
    std::vector<packk::Out<double>> out;
    std::vector<packk::Str<double>> str;
    std::vector<uint32_t> codes;
    std::vector<uint2> tile, tab;
    std::vector<std::complex<double>> amps;

    // False where the plan does not apply: ranks by search, states over 32 bits,
    // classes of more than 65,534 rows, more than 256 distinct amplitudes (coded
    // form), amplitudes that are not finite in FP32, tables over 256 MB, more than 24
    // straddling terms with one flip.
    // at_least: the least general amplitude form to give.
    bool build(const Basis& B, SiteKind site, const std::vector<Term>& terms,
               packk::AmpMode at_least = packk::AMP_UNIFORM);
    // The off-diagonal part of H x as the kernels walk the tables, every index
    // checked against its table (throws Error).
    void apply_host(const std::complex<double>* x, std::complex<double>* y) const;
};

// Their device copies.
class PackPlan {
public:
    explicit PackPlan(const PackTables& t);
    packk::AmpMode mode() const { return mode_; }
    bool real() const { return real_; }
    bool equal_magnitude() const { return equal_; }
    uint32_t n_items() const { return n_items_; }
    template <class A> void params(packk::Params<A>& p) const;

private:
    bool real_ = true, equal_ = false;
    packk::AmpMode mode_ = packk::AMP_UNIFORM;
    uint32_t n_items_ = 0;
    int n_amps_ = 0;
    double u_ = 0.0;
    DBuf all_;  // the tables, one after the other
    size_t items_ = 0, blk_ = 0, out32_ = 0, out64_ = 0, str32_ = 0, str64_ = 0, tile_ = 0, tab_ = 0, codes_ = 0,
           amps32_ = 0, amps64_ = 0;  // their offsets
    template <class E> const E* at(size_t off) const { return reinterpret_cast<const E*>(all_.as<char>() + off); }
};

// y = H x on reference-order vectors (x and y must not overlap).
void pack_apply_f32(const PackPlan& P, packk::Params<float>& p, const float2* x, float2* y, cudaStream_t s);
void pack_apply_f64(const PackPlan& P, packk::Params<double>& p, const double2* x, double2* y, cudaStream_t s);
// CTAs of a Lanczos-mode launch (one partial of Re<x, y> each)
uint32_t pack_ctas(const PackPlan& P);

}  // namespace qkg
