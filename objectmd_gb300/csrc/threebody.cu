// Three-body potentials, owner-computes in two passes over the full Verlet
// list (no atomics, deterministic):
//
//   pass A  for atom i: every term centred on i -- the two-body halves of
//           i's pairs and the triplets (SW, sw.cpp:166-236) or bonds
//           (Tersoff) whose centre is i.  The force and energy a term gives
//           to i accumulate in registers; what it gives to a neighbour j is
//           written to i's slot in j's row of a per-slot buffer (rows.cuh).
//   pass B  for atom i: own part + the slots of i's own row's hits.
//
// Pass A has two forms: a thread a centre with the neighbours in registers,
// and eight lanes a centre with up to TB_MAXN neighbours in shared memory.
// The second takes the centres that do not fit the first (queued), and every
// centre of a system too small to fill the chip with one thread each.
//
// FP32 arithmetic on relative vectors from the FP64 positions, Kahan sums in
// pass B.  Per-atom energies follow the reference: each pair half to each
// atom, V3/3 to each triplet member (sw.cpp:182-233); Tersoff: 1/2 V_ij to i.
#include <cmath>

#include "integrate_dev.cuh"

namespace omdg {

constexpr int TB_MAXN = 24;  // neighbours within the cutoff one atom can hold

// Below this many atoms a SM every centre takes eight lanes.  Thread and lane
// form, us with some 5 of launch: Tersoff 512 atoms 16.5, 13.7; 8,000 16.4,
// 15.1; 13,824 16.6, 21.1; SW 512 19.0, 11.6; 32,768 24.8, 17.8; 64,000 28.1,
// 26.2; 140,608 39.0, 42.7.
constexpr int TERS_LANE_PER_SM = 64;
constexpr int SW_LANE_PER_SM = 400;
constexpr int TB_BLOCK = 128;  // thread-a-centre kernels
constexpr int TB_LANES = 8;    // lanes a centre in the other form
constexpr int TB_LBLOCK = 64;
constexpr int TB_LGROUPS = TB_LBLOCK / TB_LANES;

// One group's centre in the lane form: its place in the block's warp.
struct LaneGroup {
    int lane, shift;
    unsigned mask;
    __device__ __forceinline__ LaneGroup()
        : lane(threadIdx.x & (TB_LANES - 1)), shift(threadIdx.x & 31 & ~(TB_LANES - 1)),
          mask(((1u << TB_LANES) - 1u) << shift) {}
    __device__ __forceinline__ float sum(float v) const {
#pragma unroll
        for (int o = TB_LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
        return v;
    }
};

// The neighbours of centre i inside the cutoff, in row order: vectors to them
// with their squared distance in v[], list slots in sl[]; returns their number
// (those past TB_MAXN are reported and get a zero slot).  A queued centre's
// row was scanned before (hits.w holds at least its hits); the others' bits
// are stored here.
template <bool QUEUED>
__device__ __forceinline__ int lanes_collect(const LaneGroup& g, int i, int m, const PosPack& pi, const ShiftF& L,
                                             float t2, int type, const PosPack* __restrict__ pack,
                                             const unsigned* __restrict__ nbr, int hshift, int maxnb,
                                             const RowHits& hits, const SlotRows& slot, float4* v, int* sl,
                                             unsigned* status) {
    int nc = 0;
    int w0 = 0;
    do {
        const unsigned want = QUEUED ? hits.word(i, w0) : 0xffffffffu;
        float4 d[4];
        unsigned bits = 0u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int b = j * TB_LANES + g.lane;
            bool in = false;
            if (w0 + b < m && ((want >> b) & 1u)) {
                const unsigned e = __ldg(nbr + nbr_at(i, w0 + b, hshift, maxnb));
                PosPack pj;
                ldg256(pack + nbr_index(e), pj.hi, pj.lo);
                const float3 x = pair_delta(pi.hi, pi.lo, pj.hi, pj.lo, e, L);
                d[j] = make_float4(-x.x, -x.y, -x.z, fmaf(x.z, x.z, fmaf(x.y, x.y, x.x * x.x)));
                in = d[j].w < t2 && (type < 0 || pack_type(pj.hi) == type);
            }
            bits |= ((__ballot_sync(g.mask, in) >> g.shift) & ((1u << TB_LANES) - 1u)) << (j * TB_LANES);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int b = j * TB_LANES + g.lane;
            if (!((bits >> b) & 1u)) continue;
            const int k = nc + __popc(bits & ((1u << b) - 1u));
            if (k < TB_MAXN) {
                v[k] = d[j];
                sl[k] = w0 + b;
            } else {
                slot.put(i, w0 + b, make_float4(0.f, 0.f, 0.f, 0.f));
                atomicOr(status, ERR_NBR_OVERFLOW);
            }
        }
        nc += __popc(bits);
        if (!QUEUED && g.lane == 0) hits.word(i, w0) = bits;
        w0 += 32;
    } while (w0 < m);
    __syncwarp(g.mask);
    return nc;
}

struct SWDev {
    int n, hshift, maxnb, single_type, ta;
    ShiftF L;
    float rc, t2;  // t2: r2 < t2 is "inside the cutoff" (r2_below); r == rc is outside, where 1/(r - rc) is infinite
    float A, B, p, q, sigma, eps;
    float c1, c2, c3, c4, c5, c6, c7, c8, c9, c10;
    int usezbl;
    float sx0, sx1, sa0, sa1, sa2, sa3;
    float zc, ze0, ze1, ze2, ze3;
    int first;
    int ip, iq;  // p and q as integers when they are (then r^-p by multiplication), else -1
};

// r^-k for a small non-negative integer k, from ir = 1/r
__device__ __forceinline__ float inv_ipow(float ir, int k) {
    float res = 1.0f, b = ir;
    while (k > 0) {
        if (k & 1) res *= b;
        b *= b;
        k >>= 1;
    }
    return res;
}

// One half of a pair at distance r; ir = 1/r, ira = 1/(r - rc).
__device__ __forceinline__ void sw_two_body(const SWDev& p, float r, float ir, float ira, float& fr, float& half_e) {
    if (p.usezbl && r < p.sx0) {
        // sw.cpp:118-146
        const float f0 = 0.1818f * expf(-p.ze0 * r), f1 = 0.5099f * expf(-p.ze1 * r);
        const float f2 = 0.2802f * expf(-p.ze2 * r), f3 = 0.02817f * expf(-p.ze3 * r);
        const float fpot = (f0 + f1 + f2 + f3) * p.zc * ir;
        fr = ((ir + p.ze0) * f0 + (ir + p.ze1) * f1 + (ir + p.ze2) * f2 + (ir + p.ze3) * f3) * p.zc * (ir * ir);
        half_e = 0.5f * fpot;
    } else if (p.usezbl && r < p.sx1) {
        // sw.cpp:148-164 (force factor applied with the opposite sign)
        const float f = p.sa1 + p.sa2 * r + p.sa3 * r * r;
        fr = -f;
        half_e = 0.5f * (p.sa0 + f * r);
    } else {
        // sw.cpp:166-189
        const float rp = p.ip >= 0 ? inv_ipow(ir, p.ip) : powf(r, -p.p);
        const float rq = p.iq >= 0 ? inv_ipow(ir, p.iq) : powf(r, -p.q);
        const float fex = expf(p.sigma * ira);
        fr = (p.c1 * rp - p.c2 * rq + (p.c3 * rp - p.c4 * rq) * ira * ira * r) * fex * (ir * ir);
        half_e = 0.5f * (p.c5 * rp - p.c6 * rq) * fex;
    }
}

// A neighbour's own quantities: from (vector, squared distance) to (unit
// vector, exp(c7/(r - rc))), with what its triplet sums are scaled by, and its
// two-body half added to the centre.
__device__ __forceinline__ void sw_neighbour(const SWDev& p, float4& v, float2& k, float& ax, float& ay, float& az,
                                             float& ae) {
    const float r = sqrtf(v.w), ir = 1.0f / r, ira = 1.0f / (r - p.rc), fira = p.c7 * ira;
    float fr, he;
    sw_two_body(p, r, ir, ira, fr, he);
    ax -= v.x * fr;
    ay -= v.y * fr;
    az -= v.z * fr;
    ae += he;
    v = make_float4(v.x * ir, v.y * ir, v.z * ir, expf(fira));
    k = make_float2(fira * ira, ir);
}

// The triplets of neighbour a (unit vector and factor ua) with b, summed over
// b != a (sw.cpp:191-236): with w = e_b (cos - c10), the sums of w (cos -
// c10), w cos and w u_b give the energy and the force of all of a's triplets
// (sw_share), twelve instructions an ordered pair where one evaluated whole
// took some sixty an unordered one.
struct SWSums {
    float s = 0.f, t = 0.f, x = 0.f, y = 0.f, z = 0.f;
    __device__ __forceinline__ void add(const SWDev& p, const float4& ua, const float4& ub, bool self) {
        const float c = fmaf(ua.z, ub.z, fmaf(ua.y, ub.y, ua.x * ub.x));
        const float dc = c - p.c10, w = self ? 0.f : ub.w * dc;
        s = fmaf(w, dc, s);
        t = fmaf(w, c, t);
        x = fmaf(w, ub.x, x);
        y = fmaf(w, ub.y, y);
        z = fmaf(w, ub.z, z);
    }
};

// What the triplets give to neighbour a: the force, and a third of their
// energy (sw.cpp:225-233).  Every triplet is in the sums of two neighbours.
__device__ __forceinline__ float4 sw_share(const SWDev& p, const float4& ua, const float2& k, const SWSums& q) {
    const float e = p.c8 * ua.w * q.s, g = p.c9 * ua.w * k.y, f = fmaf(k.x, e, g * q.t);
    return make_float4(fmaf(ua.x, f, -g * q.x), fmaf(ua.y, f, -g * q.y), fmaf(ua.z, f, -g * q.z), e * (1.0f / 3.0f));
}

constexpr int SW_REG = 8;  // in-cutoff neighbours the register path holds (diamond: 4 + thermal second shell)

__device__ __forceinline__ void sw_store(const SWDev& p, int i, float ax, float ay, float az, float ae,
                                         float* __restrict__ fx, float* __restrict__ fy, float* __restrict__ fz,
                                         float* __restrict__ pe) {
    if (p.first) {
        fx[i] = ax;
        fy[i] = ay;
        fz[i] = az;
        pe[i] = ae;
    } else {
        fx[i] += ax;
        fy[i] += ay;
        fz[i] += az;
        pe[i] += ae;
    }
}

// Pass A of SW, a thread a centre of up to SW_REG in-cutoff neighbours;
// centres with more are queued.  The scan only collects the neighbours in
// shared memory, so that the two-body term runs once for each of them with
// most of the warp in it, and not at every row entry that any lane has a hit
// at; the triplets then read them from registers.  194,184 atoms with some 7.5
// neighbours each, both passes: 148 -> 61.6 us at five blocks a SM (two whole
// waves; six leave an L1 of 64 KB to the gather: 70.0).
__global__ void __launch_bounds__(TB_BLOCK, 5) k_sw_a(SWDev p, const PosPack* __restrict__ pack,
                                                     const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                                     RowHits hits, SlotRows slot, float* __restrict__ fx,
                                                     float* __restrict__ fy, float* __restrict__ fz,
                                                     float* __restrict__ pe, int* __restrict__ wide) {
    constexpr int K = SW_REG;
    __shared__ float4 sv[K][TB_BLOCK];
    __shared__ float2 sk[K][TB_BLOCK];
    __shared__ int2 ss[K][TB_BLOCK];  // neighbour, the entry of its row that is i
    const int t = threadIdx.x;
    const int i = blockIdx.x * TB_BLOCK + t;
    if (i >= p.n) return;
    const PosPack pi = pack[i];
    const int m = nnb[i];
    int nc = 0;
    if (p.single_type || pack_type(pi.hi) == p.ta) {
        nc = scan_row<true, true>(i, m, pi, p.L, p.t2, p.single_type ? -1 : p.ta, pack, nbr, slot.rev, p.hshift, p.maxnb, hits,
                            [&](int k, int j, int r, const float3& d, float r2) {
                                if (k < K) sv[k][t] = make_float4(-d.x, -d.y, -d.z, r2), ss[k][t] = make_int2(j, r);
                            });
        if (nc > K) {
            wide[1 + atomicAdd(wide, 1)] = i;
            return;
        }
    } else {
        no_hits(i, m, hits);
    }
    float ax = 0.f, ay = 0.f, az = 0.f, ae = 0.f;
#pragma unroll 1
    for (int a = 0; a < nc; a++) {
        float4 v = sv[a][t];
        float2 k;
        sw_neighbour(p, v, k, ax, ay, az, ae);
        sv[a][t] = v;
        sk[a][t] = k;
    }
    float4 u[K];
#pragma unroll
    for (int b = 0; b < K; b++) u[b] = b < nc ? sv[b][t] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int a = 0; a < nc; a++) {
        const float4 ua = sv[a][t];
        SWSums q;
#pragma unroll
        for (int b = 0; b < K / 2; b++) q.add(p, ua, u[b], a == b);
        if (nc > K / 2) {
#pragma unroll
            for (int b = K / 2; b < K; b++) q.add(p, ua, u[b], a == b);
        }
        const float4 f = sw_share(p, ua, sk[a][t], q);
        slot.at(ss[a][t].x, ss[a][t].y) = f;
        ax -= f.x;
        ay -= f.y;
        az -= f.z;
        ae = fmaf(0.5f, f.w, ae);
    }
    sw_store(p, i, ax, ay, az, ae, fx, fy, fz, pe);
}

// Pass A of SW, eight lanes a centre: the queued centres (wide[0] of them,
// indices from wide[1]), or all of them (then the ones past the register path
// are still counted).  A lane owns a neighbour, with all of its triplets.
template <bool QUEUED>
__global__ void __launch_bounds__(TB_LBLOCK) k_sw_lanes(SWDev p, const PosPack* __restrict__ pack,
                                                       const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                                       int* __restrict__ wide, RowHits hits,
                                                       SlotRows slot, float* __restrict__ fx,
                                                       float* __restrict__ fy, float* __restrict__ fz,
                                                       float* __restrict__ pe, unsigned* status) {
    __shared__ float4 gv[TB_LGROUPS][TB_MAXN];
    __shared__ int gs[TB_LGROUPS][TB_MAXN];
    const LaneGroup g;
    float4* v = gv[threadIdx.x / TB_LANES];
    int* sl = gs[threadIdx.x / TB_LANES];
    const int total = QUEUED ? wide[0] : p.n;
    for (int c = blockIdx.x * TB_LGROUPS + threadIdx.x / TB_LANES; c < total; c += gridDim.x * TB_LGROUPS) {
        const int i = QUEUED ? wide[1 + c] : c;
        const PosPack pi = pack[i];
        const int m = nnb[i];
        int nc = 0;
        if (p.single_type || pack_type(pi.hi) == p.ta) {
            nc = lanes_collect<QUEUED>(g, i, m, pi, p.L, p.t2, p.single_type ? -1 : p.ta, pack, nbr, p.hshift,
                                       p.maxnb, hits, slot, v, sl, status);
            if (!QUEUED && nc > SW_REG && g.lane == 0) wide[1 + atomicAdd(wide, 1)] = i;
            nc = min(nc, TB_MAXN);
        } else if (!QUEUED && g.lane == 0) {
            no_hits(i, m, hits);
        }
        float ax = 0.f, ay = 0.f, az = 0.f, ae = 0.f;
        float2 k[TB_MAXN / TB_LANES];
#pragma unroll
        for (int j = 0; j < TB_MAXN / TB_LANES; j++) {
            const int a = j * TB_LANES + g.lane;
            if (a < nc) sw_neighbour(p, v[a], k[j], ax, ay, az, ae);
        }
        __syncwarp(g.mask);
#pragma unroll
        for (int j = 0; j < TB_MAXN / TB_LANES; j++) {
            const int a = j * TB_LANES + g.lane;
            if (a >= nc) continue;
            const float4 ua = v[a];
            SWSums q;
            for (int b = 0; b < nc; b++) q.add(p, ua, v[b], a == b);
            const float4 f = sw_share(p, ua, k[j], q);
            slot.put(i, sl[a], f);
            ax -= f.x;
            ay -= f.y;
            az -= f.z;
            ae = fmaf(0.5f, f.w, ae);
        }
        __syncwarp(g.mask);  // the group's neighbours are read: the next centre may overwrite them
        ax = g.sum(ax);
        ay = g.sum(ay);
        az = g.sum(az);
        ae = g.sum(ae);
        if (g.lane == 0) sw_store(p, i, ax, ay, az, ae, fx, fy, fz, pe);
    }
}

// Gathers what every neighbour's pass A left for i; clears no state.
__global__ void __launch_bounds__(128) k_slot_gather(int n, SlotArgs a, float* __restrict__ fx,
                                                     float* __restrict__ fy, float* __restrict__ fz,
                                                     float* __restrict__ pe, float* __restrict__ vir) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float gx = fx[i], gy = fy[i], gz = fz[i], ge = pe[i];
    slot_sum(a, i, gx, gy, gz, ge);
    fx[i] = gx;
    fy[i] = gy;
    fz[i] = gz;
    pe[i] = ge;
    if (a.zero_virial) vir[i] = 0.f;
}

// ------------------------------------------------------------------ Tersoff
struct TersDev {
    int n, hshift, maxnb, single_type, ta;
    ShiftF L;
    const ShiftF* rep_L;  // replica mode: periodic lengths of each replica (else null)
    const int* rep_of;
    float A, B, l1, l2, l3c, beta, nn, c2, d2, h, R, D;
    float t2;  // r2 < t2: inside the cutoff (r2_below)
    int first;
};

// b = (1 + (beta zeta)^n)^(-1/2n) and db/dzeta.  In a close collision the
// exp(lambda3^3 (r_ij - r_ik)^3) factor makes zeta large enough for
// (beta zeta)^n to overflow FP32; there b is its limit (beta zeta)^(-1/2)
// (relative difference (beta zeta)^(-n) / 2n < 1e-26 for n ln(beta zeta) > 60).
__device__ __forceinline__ void ters_bond_order(const TersDev& p, float zeta, float& b, float& db) {
    if (!(zeta > 0.f)) {
        b = 1.f;
        db = 0.f;
        return;
    }
    // hardware logarithm and exponential: n ln(beta zeta) is off by ~1e-5
    // absolute, which moves b by ~2e-7 relative (the 1/2n power damps it)
    const float x = p.beta * zeta;
    const float nlx = p.nn * __logf(x);
    if (nlx > 60.f) {
        b = rsqrtf(x);
        db = -0.5f * b / zeta;
        return;
    }
    const float bn = __expf(nlx);
    b = exp2f((-0.5f / p.nn) * __log2f(1.f + bn));  // (1 + bn)^(-1/2n), |exponent| < 2: ~3e-7 relative
    db = __fdividef(-0.5f * b * bn, (1.f + bn) * zeta);
}

__device__ __forceinline__ float ters_fc(const TersDev& p, float r, float& dfc) {
    if (r < p.R - p.D) {
        dfc = 0.f;
        return 1.f;
    }
    if (r < p.R + p.D) {
        float sn, cs;
        sincospif(0.5f * (r - p.R) / p.D, &sn, &cs);  // sin, cos of pi (r-R) / (2D)
        dfc = -0.78539816339744831f / p.D * cs;  // -pi/(4D) cos
        return 0.5f - 0.5f * sn;
    }
    dfc = 0.f;
    return 0.f;
}

// f(b) for the in-cutoff neighbours b < nc, fully unrolled over K (the arrays
// f touches stay in registers)
template <int K, class F>
__device__ __forceinline__ void for_nbrs(int nc, F&& f) {
#pragma unroll
    for (int b = 0; b < K; b++)
        if (b < nc) f(b);
}

// a b + c d with one product rounded by itself
__device__ __forceinline__ float fma2(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }

// The arithmetic of a bond that both forms share.  Every product and sum is
// written as the instruction it is, so that the forms round alike whatever the
// compiler contracts (test_tersoff_forms_have_the_same_bits).
struct TersTriplet {
    float c, g, dg, ex, dex;  // cos, g and dg/dcos, exp(l3^3 (r_ij - r_ik)^3) and its derivative by r_ij
    __device__ __forceinline__ TersTriplet(const TersDev& p, float g0, float ax, float ay, float az, float ra, float bx,
                                           float by, float bz, float rb) {
        c = fmaf(az, bz, fma2(ax, bx, ay, by));
        const float hc = __fsub_rn(p.h, c);
        const float rden = __fdividef(1.f, fmaf(hc, hc, p.d2));
        g = fmaf(-p.c2, rden, g0);
        dg = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(-2.f, p.c2), hc), rden), rden);
        const float dr = __fsub_rn(ra, rb);
        const float l = __fmul_rn(p.l3c, dr);
        ex = __expf(__fmul_rn(__fmul_rn(l, dr), dr));
        dex = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(3.f, p.l3c), dr), dr), ex);
    }
};

// V_ij = f_c (f_R - b f_A) of a bond and its derivatives by r_ij and zeta
struct TersBond {
    float v, dr, dz;
    __device__ __forceinline__ TersBond(const TersDev& p, float r, float fc, float dfc, float zeta) {
        const float fR = __fmul_rn(p.A, __expf(__fmul_rn(-p.l1, r))), fA = __fmul_rn(p.B, __expf(__fmul_rn(-p.l2, r)));
        float b, db;
        ters_bond_order(p, zeta, b, db);
        const float att = fmaf(-b, fA, fR);
        v = __fmul_rn(fc, att);
        dr = fma2(dfc, att, fc, fma2(__fmul_rn(b, p.l2), fA, -p.l1, fR));
        dz = __fmul_rn(__fmul_rn(-fc, fA), db);
    }
};

// The bonds centred on one atom, for its nc <= K in-cutoff neighbours in
// registers (unit vectors u from the centre, distances r).  Per neighbour the
// cutoff f_c(r), f_c'(r) and 1/r are evaluated once; per triplet (a, b) the
// angular and radial factors once, in the zeta sweep, with what the x_k
// gradient needs kept for its sweep.
template <int K>
__device__ __forceinline__ void ters_bonds(const TersDev& p, const int nc, const float (&ux)[K],
                                           const float (&uy)[K], const float (&uz)[K], const float (&rr)[K],
                                           float (&skx)[K], float (&sky)[K], float (&skz)[K], float& fix,
                                           float& fiy, float& fiz, float& ei, float& wi) {
    float fc[K], dfc[K], ir[K];
    for_nbrs<K>(nc, [&](int b) {
        fc[b] = ters_fc(p, rr[b], dfc[b]);
        ir[b] = 1.0f / rr[b];
        skx[b] = sky[b] = skz[b] = 0.f;
    });
    const float g0 = 1.f + p.c2 / p.d2;
    for_nbrs<K>(nc, [&](int a) {
        const float rij = rr[a];
        const float ex_ = ux[a], ey_ = uy[a], ez_ = uz[a];
        // zeta_ij and its gradient w.r.t. x_j; per k the x_k coefficients
        float zeta = 0.f, gjx = 0.f, gjy = 0.f, gjz = 0.f;
        float ck[K], cc[K], cs[K];
        for_nbrs<K>(nc, [&](int b) {
            if (b == a) return;
            const TersTriplet t(p, g0, ex_, ey_, ez_, rij, ux[b], uy[b], uz[b], rr[b]);
            const float fg = __fmul_rn(fc[b], t.g), fd = __fmul_rn(__fmul_rn(fc[b], t.dg), t.ex);
            zeta = fmaf(fg, t.ex, zeta);
            const float cj = __fmul_rn(fd, ir[a]), cu = __fmul_rn(fg, t.dex);
            gjx = __fadd_rn(gjx, fma2(cu, ex_, cj, fmaf(-t.c, ex_, ux[b])));
            gjy = __fadd_rn(gjy, fma2(cu, ey_, cj, fmaf(-t.c, ey_, uy[b])));
            gjz = __fadd_rn(gjz, fma2(cu, ez_, cj, fmaf(-t.c, ez_, uz[b])));
            ck[b] = fma2(__fmul_rn(dfc[b], t.g), t.ex, -fg, t.dex);
            cc[b] = __fmul_rn(fd, ir[b]);
            cs[b] = t.c;
        });
        const TersBond v(p, rij, fc[a], dfc[a], zeta);
        // gradient of 1/2 V_ij: x_j part
        const float sjx = 0.5f * fma2(v.dr, ex_, v.dz, gjx);
        const float sjy = 0.5f * fma2(v.dr, ey_, v.dz, gjy);
        const float sjz = 0.5f * fma2(v.dr, ez_, v.dz, gjz);
        fix = __fadd_rn(fix, sjx);  // the x_i gradient is minus the sum of the others
        fiy = __fadd_rn(fiy, sjy);
        fiz = __fadd_rn(fiz, sjz);
        const float s = 0.5f * v.dz;
        // x_k parts
        for_nbrs<K>(nc, [&](int b) {
            if (b == a) return;
            const float kx = fma2(ck[b], ux[b], cc[b], fmaf(-cs[b], ux[b], ex_));
            const float ky = fma2(ck[b], uy[b], cc[b], fmaf(-cs[b], uy[b], ey_));
            const float kz = fma2(ck[b], uz[b], cc[b], fmaf(-cs[b], uz[b], ez_));
            fix = fmaf(s, kx, fix);
            fiy = fmaf(s, ky, fiy);
            fiz = fmaf(s, kz, fiz);
            // force on k = -gradient
            skx[b] = fmaf(-s, kx, skx[b]);
            sky[b] = fmaf(-s, ky, sky[b]);
            skz[b] = fmaf(-s, kz, skz[b]);
        });
        skx[a] = __fsub_rn(skx[a], sjx);
        sky[a] = __fsub_rn(sky[a], sjy);
        skz[a] = __fsub_rn(skz[a], sjz);
        ei = __fadd_rn(ei, 0.5f * v.v);
        wi = fmaf(0.5f * v.dr, rij, wi);
    });
}

__device__ __forceinline__ void ters_store(const TersDev& p, int i, float fix, float fiy, float fiz, float ei,
                                           float wi, float* __restrict__ fx, float* __restrict__ fy,
                                           float* __restrict__ fz, float* __restrict__ pe, float* __restrict__ vir) {
    if (p.first) {
        fx[i] = fix;
        fy[i] = fiy;
        fz[i] = fiz;
        pe[i] = ei;
        vir[i] = wi;
    } else {
        fx[i] += fix;
        fy[i] += fiy;
        fz[i] += fiz;
        pe[i] += ei;
        vir[i] += wi;
    }
}

constexpr int TERS_REG = 4;  // in-cutoff neighbours the register path holds (diamond: 4)

// A masked pass (mask[i] != 0: the centre is evaluated) finds the hit bits of
// the pass that made the mask, and leaves them.
template <bool MASKED>
__device__ __forceinline__ void ters_reg_centre(const TersDev& p, int i, const PosPack* __restrict__ pack,
                                                const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                                const RowHits& hits, const SlotRows& slot,
                                                float* __restrict__ fx, float* __restrict__ fy,
                                                float* __restrict__ fz, float* __restrict__ pe,
                                                float* __restrict__ vir, int* __restrict__ wide) {
    __shared__ float4 sv[TERS_REG][TB_BLOCK];
    __shared__ int2 ss[TERS_REG][TB_BLOCK];  // neighbour, the entry of its row that is i
    const int t = threadIdx.x;
    const PosPack pi = pack[i];
    const ShiftF L = p.rep_L ? p.rep_L[p.rep_of[i]] : p.L;
    const int m = nnb[i];
    int nc = 0;
    if (p.single_type || pack_type(pi.hi) == p.ta) {
        nc = scan_row<!MASKED, true>(i, m, pi, L, p.t2, p.single_type ? -1 : p.ta, pack, nbr, slot.rev, p.hshift, p.maxnb, hits,
                               [&](int k, int j, int r, const float3& d, float r2) {
                                   if (k < TERS_REG)
                                       sv[k][t] = make_float4(-d.x, -d.y, -d.z, r2), ss[k][t] = make_int2(j, r);
                               });
        if (nc > TERS_REG) {  // queued, so its warp does not wait on it
            wide[1 + atomicAdd(wide, 1)] = i;
            return;
        }
    } else if (!MASKED) {
        no_hits(i, m, hits);
    }
    float ux[TERS_REG], uy[TERS_REG], uz[TERS_REG], rr[TERS_REG];
#pragma unroll
    for (int k = 0; k < TERS_REG; k++) {
        ux[k] = uy[k] = uz[k] = rr[k] = 0.f;
        if (k >= nc) continue;
        const float4 v = sv[k][t];
        rr[k] = sqrtf(v.w);
        const float ri = 1.0f / rr[k];
        ux[k] = __fmul_rn(v.x, ri);
        uy[k] = __fmul_rn(v.y, ri);
        uz[k] = __fmul_rn(v.z, ri);
    }
    float fix = 0.f, fiy = 0.f, fiz = 0.f, ei = 0.f, wi = 0.f;
    float skx[TERS_REG], sky[TERS_REG], skz[TERS_REG];
    ters_bonds<TERS_REG>(p, nc, ux, uy, uz, rr, skx, sky, skz, fix, fiy, fiz, ei, wi);
#pragma unroll
    for (int a = 0; a < TERS_REG; a++)
        if (a < nc) slot.at(ss[a][t].x, ss[a][t].y) = make_float4(skx[a], sky[a], skz[a], 0.f);
    ters_store(p, i, fix, fiy, fiz, ei, wi, fx, fy, fz, pe, vir);
}

// One thread per centre.  Launched with fewer threads than centres (the
// persistent form: one resident grid over the flattened atoms of every
// replica), each thread strides over the centres.
// 72 registers and an L1 of 160 KB: 512,000 atoms take 50.4, 49.7, 53.1 and 69.4
// us (with the queue's pass) at six, seven, eight and ten blocks a SM.
constexpr int TERS_CTAS_PER_SM = 7;

template <bool PERSISTENT, bool MASKED>
__global__ void __launch_bounds__(TB_BLOCK, TERS_CTAS_PER_SM) k_tersoff_a(
    TersDev p, const PosPack* __restrict__ pack, const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
    RowHits hits, SlotRows slot, float* __restrict__ fx, float* __restrict__ fy, float* __restrict__ fz,
    float* __restrict__ pe, float* __restrict__ vir, int* __restrict__ wide, const int* __restrict__ mask,
    const int* __restrict__ nmask) {
    if (MASKED && nmask && *nmask == 0) return;  // a mask with no centre in it
    int i = blockIdx.x * TB_BLOCK + threadIdx.x;
    if (PERSISTENT) {
        for (; i < p.n; i += gridDim.x * TB_BLOCK)
            if (!MASKED || mask[i])
                ters_reg_centre<MASKED>(p, i, pack, nbr, nnb, hits, slot, fx, fy, fz, pe, vir, wide);
    } else {
        if (i < p.n && (!MASKED || mask[i]))
            ters_reg_centre<MASKED>(p, i, pack, nbr, nnb, hits, slot, fx, fy, fz, pe, vir, wide);
    }
}

// The bonds of one centre in the lane form, NJ neighbours a lane: the slots are
// written, and lane 0 to 4 return the centre's sums.  wide: more neighbours than
// the register path holds, a centre that only this form takes; of two products
// that are added the other one is then the one rounded by itself, in gjx and in
// the neighbour's part.  Neither order is nearer to the exact sum; a collision
// amplifies the difference, so they stay as trajectories have them.  With one neighbour a lane (a small box, where the chain of
// one centre is all the time there is) the gradients of all bonds are kept, and
// added up once at the end: centre pass of 512 atoms 11.9 -> 11.3 us with some 5
// of launch.
template <int NJ>
__device__ __forceinline__ float ters_lanes_bonds(const TersDev& p, const LaneGroup& g, int i, int nc, bool wide,
                                                  float g0, const float4* u, float4* f, float4* x, float2* ve,
                                                  const int* sl, const SlotRows& slot) {
    int2 to[NJ];  // the slots that the neighbours' forces go to, loaded beside the bonds
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int k = j * TB_LANES + g.lane;
        if (k >= nc) continue;
        const size_t at = nbr_at(i, sl[k], p.hshift, p.maxnb);
        to[j] = make_int2(nbr_index(__ldg(slot.nbr + at)), __ldg(slot.rev + at));
    }
    float sjx[NJ], sjy[NJ], sjz[NJ], dz[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int a = j * TB_LANES + g.lane;
        if (a >= nc) continue;
        const float4 ua = u[a], fa = f[a];
        float zeta = 0.f, gjx = 0.f, gjy = 0.f, gjz = 0.f;
#pragma unroll (NJ == 1 ? 4 : 1)
        for (int b = 0; b < nc; b++) {
            if (b == a) continue;
            const float4 ub = u[b];
            const float fb = f[b].x;
            const TersTriplet t(p, g0, ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w);
            const float fg = __fmul_rn(fb, t.g);
            zeta = fmaf(fg, t.ex, zeta);
            const float cj = __fmul_rn(__fmul_rn(__fmul_rn(fb, t.dg), t.ex), fa.z), cu = __fmul_rn(fg, t.dex);
            const float px = fmaf(-t.c, ua.x, ub.x);
            gjx = __fadd_rn(gjx, wide ? fma2(cj, px, cu, ua.x) : fma2(cu, ua.x, cj, px));
            gjy = __fadd_rn(gjy, fma2(cu, ua.y, cj, fmaf(-t.c, ua.y, ub.y)));
            gjz = __fadd_rn(gjz, fma2(cu, ua.z, cj, fmaf(-t.c, ua.z, ub.z)));
        }
        const TersBond v(p, ua.w, fa.x, fa.y, zeta);
        sjx[j] = 0.5f * (wide ? fma2(v.dz, gjx, v.dr, ua.x) : fma2(v.dr, ua.x, v.dz, gjx));
        sjy[j] = 0.5f * (wide ? fma2(v.dz, gjy, v.dr, ua.y) : fma2(v.dr, ua.y, v.dz, gjy));
        sjz[j] = 0.5f * (wide ? fma2(v.dz, gjz, v.dr, ua.z) : fma2(v.dr, ua.z, v.dz, gjz));
        dz[j] = 0.5f * v.dz;
        ve[a] = make_float2(v.v, v.dr);
    }
    __syncwarp(g.mask);
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int a = j * TB_LANES + g.lane;
        if (a < nc) f[a].w = dz[j];
    }
    __syncwarp(g.mask);
    float skx[NJ], sky[NJ], skz[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++) skx[j] = sky[j] = skz[j] = 0.f;
    float own = 0.f;  // lane 0 to 4: the centre's x, y, z, energy and virial, in the register path's order
    const auto add = [&](int a, float s, const float4* row) {
        if (g.lane < 3) {
            const float* xc = &row[0].x + g.lane;
            own = __fadd_rn(own, xc[4 * a]);  // the x_i gradient is minus the sum of the others
            for (int b = 0; b < nc; b++)
                if (b != a) own = fmaf(s, xc[4 * b], own);
        } else if (g.lane == 3) {
            own = __fadd_rn(own, 0.5f * ve[a].x);
        } else if (g.lane == 4) {
            own = fmaf(0.5f * ve[a].y, u[a].w, own);
        }
    };
#pragma unroll (NJ == 1 ? 2 : 1)
    for (int a = 0; a < nc; a++) {
        float4* const row = NJ == 1 ? x + a * TB_LANES : x;
        const float4 ua = u[a];
        const float s = f[a].w;
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int k = j * TB_LANES + g.lane;
            if (k >= nc) continue;
            if (k == a) {
                row[k] = make_float4(sjx[j], sjy[j], sjz[j], 0.f);
                skx[j] -= sjx[j];
                sky[j] -= sjy[j];
                skz[j] -= sjz[j];
                continue;
            }
            const float4 uk = u[k], fk = f[k];
            const TersTriplet t(p, g0, ua.x, ua.y, ua.z, ua.w, uk.x, uk.y, uk.z, uk.w);
            const float fg = __fmul_rn(fk.x, t.g);
            const float ck = fma2(__fmul_rn(fk.y, t.g), t.ex, -fg, t.dex);
            const float cc = __fmul_rn(__fmul_rn(__fmul_rn(fk.x, t.dg), t.ex), fk.z);
            const float kx = fma2(ck, uk.x, cc, fmaf(-t.c, uk.x, ua.x));
            const float ky = fma2(ck, uk.y, cc, fmaf(-t.c, uk.y, ua.y));
            const float kz = fma2(ck, uk.z, cc, fmaf(-t.c, uk.z, ua.z));
            row[k] = make_float4(kx, ky, kz, 0.f);
            // force on k = -gradient
            skx[j] = fmaf(-s, kx, skx[j]);
            sky[j] = fmaf(-s, ky, sky[j]);
            skz[j] = fmaf(-s, kz, skz[j]);
        }
        if (NJ > 1) {
            __syncwarp(g.mask);
            add(a, s, row);
            __syncwarp(g.mask);
        }
    }
    if (NJ == 1) {
        __syncwarp(g.mask);
        for (int a = 0; a < nc; a++) add(a, f[a].w, x + a * TB_LANES);
    }
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int k = j * TB_LANES + g.lane;
        if (k < nc) slot.at(to[j].x, to[j].y) = make_float4(skx[j], sky[j], skz[j], 0.f);
    }
    return own;
}

// Eight lanes a centre: the queued centres (wide[0] of them, indices from
// wide[1]), or all of them (then the ones past the register path are still
// counted).  A lane owns a neighbour: its bond's zeta and gradient first, then
// what each bond in turn gives to it as its third atom, for which the factors
// of the triplet are evaluated again (some 30 instructions).  The centre's sums
// are taken bond by bond in the register path's order, from the same
// instructions (TersTriplet, TersBond): both forms give the same bits, and a
// trajectory does not depend on which took a centre.  The queue was one thread a centre over local
// arrays, a chain of some 190,000 cycles: 0.7 % of the 1.47 M
// atoms of the impact ensemble, both passes 199 -> 141 us.
template <bool QUEUED>
__global__ void __launch_bounds__(TB_LBLOCK) k_tersoff_lanes(
    TersDev p, const PosPack* __restrict__ pack, const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
    int* __restrict__ wide, RowHits hits, SlotRows slot, float* __restrict__ fx, float* __restrict__ fy,
    float* __restrict__ fz, float* __restrict__ pe, float* __restrict__ vir, unsigned* status) {
    __shared__ float4 gu[TB_LGROUPS][TB_MAXN];  // vector and squared distance, then unit vector and distance
    __shared__ float4 gf[TB_LGROUPS][TB_MAXN];  // f_c, f_c', 1/r, half the bond's dV/dzeta
    __shared__ float4 gx[TB_LGROUPS][QUEUED ? TB_MAXN : TB_LANES * TB_LANES];  // the bonds' gradients by the neighbours
    __shared__ float2 ge[TB_LGROUPS][TB_MAXN];  // a bond's energy and its derivative by r
    __shared__ int gs[TB_LGROUPS][TB_MAXN];
    const LaneGroup g;
    float4* u = gu[threadIdx.x / TB_LANES];
    float4* f = gf[threadIdx.x / TB_LANES];
    float4* x = gx[threadIdx.x / TB_LANES];
    float2* ve = ge[threadIdx.x / TB_LANES];
    int* sl = gs[threadIdx.x / TB_LANES];
    const float g0 = 1.f + p.c2 / p.d2;
    const int total = QUEUED ? wide[0] : p.n;
    for (int c0 = blockIdx.x * TB_LGROUPS + threadIdx.x / TB_LANES; c0 < total; c0 += gridDim.x * TB_LGROUPS) {
        const int i = QUEUED ? wide[1 + c0] : c0;
        const PosPack pi = pack[i];
        const ShiftF L = p.rep_L ? p.rep_L[p.rep_of[i]] : p.L;
        const int m = nnb[i];
        int nc = 0;
        if (p.single_type || pack_type(pi.hi) == p.ta) {
            nc = lanes_collect<QUEUED>(g, i, m, pi, L, p.t2, p.single_type ? -1 : p.ta, pack, nbr, p.hshift,
                                       p.maxnb, hits, slot, u, sl, status);
            if (!QUEUED && nc > TERS_REG && g.lane == 0) wide[1 + atomicAdd(wide, 1)] = i;
            nc = min(nc, TB_MAXN);
        } else if (!QUEUED && g.lane == 0) {
            no_hits(i, m, hits);
        }
        for (int a = g.lane; a < nc; a += TB_LANES) {
            const float4 v = u[a];
            const float r = sqrtf(v.w), ri = 1.0f / r;
            float dfc;
            const float fc = ters_fc(p, r, dfc);
            u[a] = make_float4(v.x * ri, v.y * ri, v.z * ri, r);
            f[a] = make_float4(fc, dfc, ri, 0.f);
        }
        __syncwarp(g.mask);
        const float own = !QUEUED && nc <= TB_LANES
                              ? ters_lanes_bonds<1>(p, g, i, nc, nc > TERS_REG, g0, u, f, x, ve, sl, slot)
                              : ters_lanes_bonds<TB_MAXN / TB_LANES>(p, g, i, nc, true, g0, u, f, x, ve, sl, slot);
        __syncwarp(g.mask);  // the group's neighbours are read: the next centre may overwrite them
        if (g.lane < 5) {
            float* out = g.lane == 0 ? fx : g.lane == 1 ? fy : g.lane == 2 ? fz : g.lane == 3 ? pe : vir;
            out[i] = p.first ? own : out[i] + own;
        }
    }
}

// ------------------------------------------------------------------ ZBL pair
struct ZBLDev {
    int n, hshift, maxnb, ta, tb;
    ShiftF L;
    const ShiftF* rep_L;  // replica mode (else null)
    const int* rep_of;
    float rc, rsw, zc, ze0, ze1, ze2, ze3;
    int first;
};

// Universal ZBL screened Coulomb (sw.cpp:118-146 form), multiplied by a
// smooth switch S(r) that goes from 1 at rsw to 0 at rc.
__global__ void __launch_bounds__(128) k_zbl(ZBLDev p, const PosPack* __restrict__ pack,
                                             const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                             float* __restrict__ fx, float* __restrict__ fy, float* __restrict__ fz,
                                             float* __restrict__ pe, float* __restrict__ vir) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const PosPack pi = pack[i];
    const int ti = pack_type(pi.hi);
    const ShiftF L = p.rep_L ? p.rep_L[p.rep_of[i]] : p.L;
    float ax = 0.f, ay = 0.f, az = 0.f, ae = 0.f, av = 0.f;
    if (ti == p.ta || ti == p.tb) {
        const int m = nnb[i];
        for (int s = 0; s < m; s++) {
            const unsigned e = nbr[nbr_at(i, s, p.hshift, p.maxnb)];
            const PosPack pj = pack[nbr_index(e)];
            const int tj = pack_type(pj.hi);
            if (!((ti == p.ta && tj == p.tb) || (ti == p.tb && tj == p.ta))) continue;
            const float3 d = pair_delta(pi.hi, pi.lo, pj.hi, pj.lo, e, L);
            const float r2 = fmaf(d.z, d.z, fmaf(d.y, d.y, d.x * d.x));
            const float r = sqrtf(r2);
            if (!(r < p.rc)) continue;
            const float rinv = 1.f / r;
            const float f0 = 0.1818f * expf(-p.ze0 * r), f1 = 0.5099f * expf(-p.ze1 * r);
            const float f2 = 0.2802f * expf(-p.ze2 * r), f3 = 0.02817f * expf(-p.ze3 * r);
            const float phi = (f0 + f1 + f2 + f3) * p.zc * rinv;
            const float dphi = -((rinv + p.ze0) * f0 + (rinv + p.ze1) * f1 + (rinv + p.ze2) * f2 +
                                 (rinv + p.ze3) * f3) * p.zc * rinv;
            float S = 1.f, dS = 0.f;
            if (r > p.rsw) {
                const float t = (r - p.rsw) / (p.rc - p.rsw);
                S = 1.f - t * t * t * (10.f - 15.f * t + 6.f * t * t);
                dS = -30.f * t * t * (1.f - t) * (1.f - t) / (p.rc - p.rsw);
            }
            const float v = phi * S;
            const float dv = dphi * S + phi * dS;
            const float fr = -dv * rinv;
            ax += d.x * fr;
            ay += d.y * fr;
            az += d.z * fr;
            ae += 0.5f * v;
            av += fr * r2;
        }
    }
    if (p.first) {
        fx[i] = ax;
        fy[i] = ay;
        fz[i] = az;
        pe[i] = ae;
        vir[i] = av;
    } else {
        fx[i] += ax;
        fy[i] += ay;
        fz[i] += az;
        pe[i] += ae;
        vir[i] += av;
    }
}

// ------------------------------------------------------------------ host
int threebody_prepare(Context* c) { return OMDG_OK; }

RowHits row_hits(const Context* c) { return RowHits{c->row_hits, (size_t)c->cap}; }

SlotRows slot_rows(const Context* c) {
    return SlotRows{c->slot_buf, reinterpret_cast<const unsigned*>(c->nbr), c->rev, c->nbr_hshift, c->maxnb};
}

SlotArgs slot_args(const Context* c, bool zero_virial) {
    return SlotArgs{c->nbr_hshift, c->maxnb, c->nnb, c->slot_buf, row_hits(c), zero_virial ? 1 : 0};
}

// All centres in the lane form?
static bool all_by_lanes(const Context* c, int per_sm) { return c->n < per_sm * c->num_sms; }

// Blocks of the queue's pass: its length is on the device, so one resident
// set of groups that stride over it.
static unsigned queue_blocks(const Context* c) { return 8u * (unsigned)c->num_sms; }

// In a step the last gather before the kick joins it (forces_compute decides).
int gather_slots(Context* c, bool zero_virial) {
    if (c->defer_gather) {
        c->gather_deferred = true;
        c->gather_zero_virial = zero_virial;
        return OMDG_OK;
    }
    prof_begin(c, "slot_gather");
    k_slot_gather<<<grid_for(c->n, 128), 128, 0, c->stream>>>(c->n, slot_args(c, zero_virial), c->fx, c->fy, c->fz,
                                                              c->pe, c->vir);
    prof_end(c);
    c->launches++;
    return check_cuda(c, cudaGetLastError(), "slot gather");
}

// The queue of wide centres is empty: cleared by the step's kick_drift for the
// first pass of a step, here for every other pass.
static void clear_wide(Context* c) {
    if (!c->wide_cleared) cudaMemsetAsync(c->ters_wide, 0, sizeof(int), c->stream);
    c->wide_cleared = false;
}

int sw_launch(Context* c, Potential& pot, bool first) {
    if (!c->rev || !c->slot_buf) return set_error(c, OMDG_ESTATE, "three-body buffers missing");
    const SWParams& s = pot.sw;
    SWDev p;
    p.n = c->n;
    p.hshift = c->nbr_hshift;
    p.maxnb = c->maxnb;
    p.single_type = c->ntypes == 1;
    p.ta = pot.ta;
    p.L = make_shift(c->box);
    p.rc = (float)s.rc;
    p.t2 = r2_below(p.rc, (float)(s.rc * s.rc));
    p.A = (float)s.A;
    p.B = (float)s.B;
    p.p = (float)s.p;
    p.q = (float)s.q;
    p.ip = (s.p >= 0 && s.p <= 16 && s.p == std::floor(s.p)) ? (int)s.p : -1;
    p.iq = (s.q >= 0 && s.q <= 16 && s.q == std::floor(s.q)) ? (int)s.q : -1;
    p.sigma = (float)s.sigma;
    p.eps = (float)s.eps;
    p.c1 = (float)s.c1;
    p.c2 = (float)s.c2;
    p.c3 = (float)s.c3;
    p.c4 = (float)s.c4;
    p.c5 = (float)s.c5;
    p.c6 = (float)s.c6;
    p.c7 = (float)s.c7;
    p.c8 = (float)s.c8;
    p.c9 = (float)s.c9;
    p.c10 = (float)s.c10;
    p.usezbl = s.usezbl;
    p.sx0 = (float)s.sx0;
    p.sx1 = (float)s.sx1;
    p.sa0 = (float)s.sa0;
    p.sa1 = (float)s.sa1;
    p.sa2 = (float)s.sa2;
    p.sa3 = (float)s.sa3;
    p.zc = (float)s.zc;
    p.ze0 = (float)s.ze0;
    p.ze1 = (float)s.ze1;
    p.ze2 = (float)s.ze2;
    p.ze3 = (float)s.ze3;
    p.first = first ? 1 : 0;
    prof_begin(c, "sw_centre");
    clear_wide(c);
    const unsigned* nbr = reinterpret_cast<const unsigned*>(c->nbr);
    if (all_by_lanes(c, SW_LANE_PER_SM)) {
        k_sw_lanes<false><<<grid_for(c->n, TB_LGROUPS), TB_LBLOCK, 0, c->stream>>>(
            p, c->pack, nbr, c->nnb, c->ters_wide, row_hits(c), slot_rows(c), c->fx, c->fy, c->fz, c->pe, c->d_status);
    } else {
        k_sw_a<<<grid_for(c->n, TB_BLOCK), TB_BLOCK, 0, c->stream>>>(p, c->pack, nbr, c->nnb, row_hits(c), slot_rows(c),
                                                                     c->fx, c->fy, c->fz, c->pe, c->ters_wide);
        k_sw_lanes<true><<<queue_blocks(c), TB_LBLOCK, 0, c->stream>>>(p, c->pack, nbr, c->nnb, c->ters_wide,
                                                                       row_hits(c), slot_rows(c), c->fx, c->fy, c->fz,
                                                                       c->pe, c->d_status);
        c->launches++;
    }
    prof_end(c);
    c->launches++;
    int rc = check_cuda(c, cudaGetLastError(), "sw");
    if (rc) return rc;
    return gather_slots(c, first);
}

int tersoff_launch(Context* c, Potential& pot, bool first) {
    int rc = tersoff_centre(c, pot, first, nullptr);
    if (rc) return rc;
    return gather_slots(c, false);
}

float tersoff_t2(const TersoffParams& t) {
    const float rc = (float)(t.R + t.D);
    return r2_below(rc, rc * rc * 1.0001f);
}

// Pass A of Tersoff: bond gradients of every centre (or of the centres with
// mask[i] != 0) into the slot buffer; the caller gathers.
int tersoff_centre(Context* c, Potential& pot, bool first, const int* mask, const int* mask_count) {
    if (!c->rev || !c->slot_buf) return set_error(c, OMDG_ESTATE, "three-body buffers missing");
    const TersoffParams& t = pot.ters;
    TersDev p;
    p.n = c->n;
    p.hshift = c->nbr_hshift;
    p.maxnb = c->maxnb;
    p.single_type = c->ntypes == 1;
    p.ta = pot.ta;
    p.L = make_shift(c->box);
    p.rep_L = c->nrep > 0 ? static_cast<const ShiftF*>(c->d_rep_shift) : nullptr;
    p.rep_of = c->d_rep_of;
    p.A = (float)t.A;
    p.B = (float)t.B;
    p.l1 = (float)t.lambda1;
    p.l2 = (float)t.lambda2;
    p.l3c = (float)(t.lambda3 * t.lambda3 * t.lambda3);
    p.beta = (float)t.beta;
    p.nn = (float)t.n;
    p.c2 = (float)(t.c * t.c);
    p.d2 = (float)(t.d * t.d);
    p.h = (float)t.h;
    p.R = (float)t.R;
    p.D = (float)t.D;
    p.t2 = tersoff_t2(t);
    p.first = first ? 1 : 0;
    prof_begin(c, mask ? "tersoff_fallback" : "tersoff_centre");
    clear_wide(c);
    const unsigned* nbr = reinterpret_cast<const unsigned*>(c->nbr);
    const RowHits hits = row_hits(c);
    if (!mask && all_by_lanes(c, TERS_LANE_PER_SM)) {
        k_tersoff_lanes<false><<<grid_for(c->n, TB_LGROUPS), TB_LBLOCK, 0, c->stream>>>(
            p, c->pack, nbr, c->nnb, c->ters_wide, hits, slot_rows(c), c->fx, c->fy, c->fz, c->pe, c->vir,
            c->d_status);
    } else {
        // a masked pass (the surrogate's fallback, usually for no centre at
        // all) takes the strided form: one resident grid, each block gone
        // after reading the count
        const unsigned all = grid_for(c->n, TB_BLOCK);
        const unsigned resident = std::min(all, (unsigned)(TERS_CTAS_PER_SM * c->num_sms));
        auto pass = mask ? k_tersoff_a<true, true> : c->tb_persistent ? k_tersoff_a<true, false> : k_tersoff_a<false, false>;
        pass<<<mask || c->tb_persistent ? resident : all, TB_BLOCK, 0, c->stream>>>(
            p, c->pack, nbr, c->nnb, hits, slot_rows(c), c->fx, c->fy, c->fz, c->pe, c->vir, c->ters_wide, mask,
            mask_count);
        k_tersoff_lanes<true><<<queue_blocks(c), TB_LBLOCK, 0, c->stream>>>(p, c->pack, nbr, c->nnb, c->ters_wide,
                                                                            hits, slot_rows(c), c->fx, c->fy, c->fz,
                                                                            c->pe, c->vir, c->d_status);
        c->launches++;
    }
    prof_end(c);
    c->launches++;
    return check_cuda(c, cudaGetLastError(), "tersoff");
}

int zbl_launch(Context* c, Potential& pot, bool first) {
    const ZBLParams& z = pot.zbl;
    ZBLDev p;
    p.n = c->n;
    p.hshift = c->nbr_hshift;
    p.maxnb = c->maxnb;
    p.ta = pot.ta;
    p.tb = pot.tb;
    p.L = make_shift(c->box);
    p.rep_L = c->nrep > 0 ? static_cast<const ShiftF*>(c->d_rep_shift) : nullptr;
    p.rep_of = c->d_rep_of;
    p.rc = (float)z.rc;
    p.rsw = (float)(z.rc - z.width);
    p.zc = (float)z.zc;
    p.ze0 = (float)z.ze0;
    p.ze1 = (float)z.ze1;
    p.ze2 = (float)z.ze2;
    p.ze3 = (float)z.ze3;
    p.first = first ? 1 : 0;
    prof_begin(c, "zbl");
    k_zbl<<<grid_for(c->n, 128), 128, 0, c->stream>>>(p, c->pack, reinterpret_cast<const unsigned*>(c->nbr), c->nnb,
                                                       c->fx, c->fy, c->fz, c->pe, c->vir);
    prof_end(c);
    c->launches++;
    return check_cuda(c, cudaGetLastError(), "zbl");
}

}  // namespace omdg
