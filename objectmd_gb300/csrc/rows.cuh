// One atom's Verlet row against a cutoff, shared by the three-body kernels and
// the surrogate, with the row's hit bits.
#pragma once

#include <cmath>

#include "device_common.cuh"

namespace omdg {

// Bit s of atom i's row: entry s lies inside the cutoff of the pass that ran
// last.  The relative vector of a pair is the same number with the other sign
// from its other atom (pair_delta rounds symmetrically), so a bit of i's row
// says as well that the neighbour wrote a contribution for i: a centre pass
// writes the contributions of its hits only, and the gather reads no others.
// Before, a pass zeroed every slot of the list (16 bytes an entry, 220 MB for
// 512,000 Tersoff atoms with some 28 entries each) and the gather read them
// all back.
struct RowHits {
    unsigned* w;    // word s/32 of atom i at w[(s/32) * stride + i]: the first, and those below the row's end
    size_t stride;
    __device__ __forceinline__ unsigned& word(int i, int s) const { return w[(size_t)(s >> 5) * stride + i]; }
};

// The force and energy (x, y, z, e) that centre i's terms give to entry s of
// its row lie in the neighbour's row, at the entry that is i there: the gather
// reads its own row, with nothing to look up first.  (Where they lay at the
// centre's own entry each read waited for the entry and its reverse slot, two
// more sectors.  Centre pass, kick with the gather, us: 512,000 Tersoff atoms
// 48.1 + 42.0 and 49.7 + 32.9; 194,184 Stillinger-Weber atoms 56.3 + 34.9 and
// 61.6 + 27.0; 512,000 surrogate atoms' forces 108.8 + 44.9 and 112.9 + 34.9.)
struct SlotRows {
    float4* slot;
    const unsigned* nbr;
    const int* rev;
    int hshift, maxnb;
    __device__ __forceinline__ float4& at(int j, int r) const { return slot[nbr_at(j, r, hshift, maxnb)]; }
    __device__ __forceinline__ void put(int i, int s, const float4& v) const {
        const size_t a = nbr_at(i, s, hshift, maxnb);
        at(nbr_index(__ldg(nbr + a)), __ldg(rev + a)) = v;
    }
};

// The smallest FP32 number whose square root rounds to rc or above, or rc2 if
// that is less: r2 < r2_below(rc, rc2) is r2 < rc2 && sqrtf(r2) < rc (the
// square root is correctly rounded on both sides), without the root.
inline float r2_below(float rc, float rc2) {
    if (!(rc > 0.f)) return 0.f;
    float t = rc * rc;
    while (std::sqrt(t) >= rc) t = std::nextafter(t, 0.f);
    while (std::sqrt(t) < rc) t = std::nextafter(t, INFINITY);
    return std::fmin(t, rc2);
}

// Calls hit(k, j, rev, d, r2) for the k-th entry of row i, atom j, with r2 < t2
// (d = x_i - x_j) and, when one type is asked for (type >= 0), of that type;
// returns their number.  KEEP: the hit bits are stored.  REV: rev is the entry
// of j's row that is i.  The loads of four entries are in flight at a time.
template <bool KEEP, bool REV, class Hit>
__device__ __forceinline__ int scan_row(int i, int m, const PosPack& pi, const ShiftF& L, float t2, int type,
                                        const PosPack* __restrict__ pack, const unsigned* __restrict__ nbr,
                                        const int* __restrict__ rev, int hshift, int maxnb, const RowHits& hits,
                                        Hit&& hit) {
    int nc = 0;
    int w0 = 0;
    do {
        const int end = min(m, w0 + 32);
        unsigned bits = 0u;
        for (int s0 = w0; s0 < end; s0 += 4) {
            unsigned e[4];
            int r[4];
            PosPack pj[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const size_t at = nbr_at(i, min(s0 + k, end - 1), hshift, maxnb);
                e[k] = __ldg(nbr + at);
                r[k] = REV ? __ldg(rev + at) : 0;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) ldg256(pack + nbr_index(e[k]), pj[k].hi, pj[k].lo);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float3 d = pair_delta(pi.hi, pi.lo, pj[k].hi, pj[k].lo, e[k], L);
                const float r2 = fmaf(d.z, d.z, fmaf(d.y, d.y, d.x * d.x));
                if (s0 + k < end && r2 < t2 && (type < 0 || pack_type(pj[k].hi) == type)) {
                    bits |= 1u << (s0 + k - w0);
                    hit(nc, nbr_index(e[k]), r[k], d, r2);
                    nc++;
                }
            }
        }
        if (KEEP) hits.word(i, w0) = bits;
        w0 += 32;
    } while (w0 < m);
    return nc;
}

// A row that takes no part: no hits.
__device__ __forceinline__ void no_hits(int i, int m, const RowHits& hits) {
    int w0 = 0;
    do {
        hits.word(i, w0) = 0u;
        w0 += 32;
    } while (w0 < m);
}

RowHits row_hits(const Context* c);  // threebody.cu
SlotRows slot_rows(const Context* c);

}  // namespace omdg
