// Tabulated pair potential (TForcePair, tpair.h:38-71): fr = -phi'(r)/r for
// r < rc (strict), ReturnForce on the owner side (forcekernel.h:92-110).
// Two precisions: FP32 on the mixed-precision relative vector (LANES threads
// per atom, Kahan partials combined by a TwoSum shuffle tree), and an FP64
// path (positions, table and accumulation in FP64) for the plain FP64
// Lennard-Jones configuration.
#include "device_common.cuh"

namespace omdg {

struct PairParams {
    int n;
    int hshift, maxnb;
    ShiftF L;
    double L64[3];
    DevTable phi;
    float rc, rc2;
    double rc64;
    int ta, tb, all_types;
    int first;
    const ShiftF* rep_L;  // replica mode: periodic lengths of each replica (else null)
    const int* rep_of;
};

__device__ __forceinline__ bool types_match(int a, int b, int ta, int tb) {
    return (a == ta && b == tb) || (a == tb && b == ta);
}

template <int LANES>
__device__ __forceinline__ void lanes_twosum(float& s, float& c) {
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) {
        float s2 = __shfl_xor_sync(0xffffffffu, s, off);
        float c2 = __shfl_xor_sync(0xffffffffu, c, off);
        float t = __fadd_rn(s, s2);
        float bp = __fsub_rn(t, s);
        float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(s2, bp));
        c = __fsub_rn(__fadd_rn(c, c2), e);
        s = t;
    }
}

// One lane's share of the row of atom ii (entries lane, lane + LANES, ...).
template <int LANES>
__device__ __forceinline__ void pair32_sum(const PairParams& p, const PosPack* __restrict__ pack,
                                           const unsigned* __restrict__ nbr, int ii, const PosPack& pi, int ti, int m,
                                           int lane, Kahan& ax, Kahan& ay, Kahan& az, Kahan& ae, float& av,
                                           unsigned* status) {
    const ShiftF L = p.rep_L ? p.rep_L[p.rep_of[ii]] : p.L;
    for (int s = lane; s < m; s += LANES) {
        unsigned e = __ldg(&nbr[nbr_at(ii, s, p.hshift, p.maxnb)]);
        int j = nbr_index(e);
        const float4* pj = reinterpret_cast<const float4*>(pack + j);
        const float4 hj = __ldg(pj);  // the type word first: most rows of a mixed system skip here
        if (!p.all_types && !types_match(ti, pack_type(hj), p.ta, p.tb)) continue;
        const float4 lj = __ldg(pj + 1);
        float3 d = pair_delta(pi.hi, pi.lo, hj, lj, e, L);
        float r2 = fmaf(d.z, d.z, fmaf(d.y, d.y, d.x * d.x));
        if (r2 >= p.rc2) continue;
        float rinv = rsqrtf(r2);
        float r = r2 * rinv;
        if (!(r < p.rc)) continue;
        float ph, dph;
        tab_read(p.phi, p.phi.coef, r, rinv, ph, dph, status);
        float fr = -dph * rinv;
        ax.add(d.x * fr);
        ay.add(d.y * fr);
        az.add(d.z * fr);
        ae.add(0.5f * ph);
        av = fmaf(fr, r2, av);
    }
    lanes_twosum<LANES>(ax.s, ax.c);
    lanes_twosum<LANES>(ay.s, ay.c);
    lanes_twosum<LANES>(az.s, az.c);
    lanes_twosum<LANES>(ae.s, ae.c);
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) av += __shfl_xor_sync(0xffffffffu, av, off);
}

__device__ __forceinline__ void pair32_store(const PairParams& p, int i, int m, const Kahan& ax, const Kahan& ay,
                                             const Kahan& az, const Kahan& ae, float av, float* __restrict__ fx,
                                             float* __restrict__ fy, float* __restrict__ fz, float* __restrict__ pe,
                                             float* __restrict__ vir) {
    const float vfx = __fsub_rn(ax.s, ax.c), vfy = __fsub_rn(ay.s, ay.c), vfz = __fsub_rn(az.s, az.c);
    const float ve = __fsub_rn(ae.s, ae.c);
    if (p.first) {
        fx[i] = vfx;
        fy[i] = vfy;
        fz[i] = vfz;
        pe[i] = ve;
        vir[i] = av;
    } else if (m) {
        fx[i] += vfx;
        fy[i] += vfy;
        fz[i] += vfz;
        pe[i] += ve;
        vir[i] += av;
    }
}

// A typed pair: the row of an atom of type ta or tb that holds an atom of the
// other type (the rows' type masks; most rows of a mixed system, a Si atom
// with no Ar near, have none).
__device__ __forceinline__ bool pair32_wanted(const PairParams& p, int ti, unsigned mask) {
    const unsigned want_a = 1u << (p.tb & 31), want_b = 1u << (p.ta & 31);
    return (mask & ((ti == p.ta ? want_a : 0u) | (ti == p.tb ? want_b : 0u))) != 0u;
}

template <int LANES>
__global__ void __launch_bounds__(512) k_pair32(PairParams p, const PosPack* __restrict__ pack,
                                                const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                                float* __restrict__ fx, float* __restrict__ fy,
                                                float* __restrict__ fz, float* __restrict__ pe,
                                                float* __restrict__ vir, unsigned* status,
                                                const unsigned* __restrict__ nbmask) {
    const int lane = threadIdx.x & (LANES - 1);
    const int per_block = blockDim.x / LANES;
    for (int base = blockIdx.x * per_block; base < p.n; base += gridDim.x * per_block) {
        int i = base + threadIdx.x / LANES;
        bool valid = i < p.n;
        int ii = valid ? i : p.n - 1;
        PosPack pi = pack[ii];
        int ti = pack_type(pi.hi);
        const bool any = valid && (p.all_types || pair32_wanted(p, ti, nbmask[ii]));
        const int m = any ? nnb[ii] : 0;
        Kahan ax, ay, az, ae;
        float av = 0.f;
        pair32_sum<LANES>(p, pack, nbr, ii, pi, ti, m, lane, ax, ay, az, ae, av, status);
        if (lane == 0 && valid) pair32_store(p, i, m, ax, ay, az, ae, av, fx, fy, fz, pe, vir);
    }
}

// The typed pair where the chip is full: a warp looks at 32 atoms with one
// coalesced load each (type, mask), compacts those with a partner, and takes
// them 32 / LANES at a time.  In the impact ensemble (1.47 M atoms, 256 Ar
// atoms) LANES threads for every atom read every pack to find three thousand
// rows: 122 us, now 20.
template <int LANES>
__global__ void __launch_bounds__(256) k_pair32_typed(PairParams p, const PosPack* __restrict__ pack,
                                                      const int* __restrict__ type,
                                                      const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                                      float* __restrict__ fx, float* __restrict__ fy,
                                                      float* __restrict__ fz, float* __restrict__ pe,
                                                      float* __restrict__ vir, unsigned* status,
                                                      const unsigned* __restrict__ nbmask) {
    __shared__ int s_act[256];
    const int t = blockIdx.x * blockDim.x + threadIdx.x, wl = threadIdx.x & 31;
    const bool any = t < p.n && pair32_wanted(p, type[t], nbmask[t]);
    const unsigned act = __ballot_sync(0xffffffffu, any);
    int* const mine = s_act + (threadIdx.x & ~31);
    if (any) mine[__popc(act & ((1u << wl) - 1u))] = t;
    if (p.first && t < p.n && !any) fx[t] = fy[t] = fz[t] = pe[t] = vir[t] = 0.f;
    __syncwarp();
    const int lane = threadIdx.x & (LANES - 1), count = __popc(act);
    for (int k = 0; k < count; k += 32 / LANES) {
        const bool valid = k + wl / LANES < count;
        const int i = mine[valid ? k + wl / LANES : 0];
        const PosPack pi = pack[i];
        const int m = valid ? nnb[i] : 0;
        Kahan ax, ay, az, ae;
        float av = 0.f;
        pair32_sum<LANES>(p, pack, nbr, i, pi, pack_type(pi.hi), m, lane, ax, ay, az, ae, av, status);
        if (lane == 0 && valid) pair32_store(p, i, m, ax, ay, az, ae, av, fx, fy, fz, pe, vir);
    }
}

// FP64 end to end.  The FP64 pipe (one warp instruction in about 18 cycles of
// an SM) sets the time, so the pass counts FP64 instructions: about 30 a pair.
//   - the centre minus the image's length is formed once per centre and picked
//     by the entry's image bits (integer selects cost nothing here);
//   - 1/r comes from the hardware's reciprocal-square-root estimate and one
//     third-order step (Householder's for y^-2 = r^2: y + y e (1/2 + 3/8 e),
//     e = 1 - r^2 y^2, leaves the estimate's error cubed, below an ulp), r =
//     r^2 / r takes one Newton step to half an ulp, and the force factor a
//     product where the reference divides;
//   - the knot index comes from FP32, which near a knot may name the segment
//     next door: the offset from the knot then is negative or a whole segment,
//     one integer comparison, and the index is put right out of line;
//   - value and slope share their Horner steps.
// Reads below the first knot, with the reference's edge rules, go through
// tab_read64 out of line.  The IEEE sequences (root, two divisions, separate
// adds and products) took about 110 FP64 instructions a pair: 4,000 LJ argon
// atoms 66 us, now 33.  Against quad precision the forces are as far off as
// theirs (1.3-1.4e-15 of the norm).
__device__ __noinline__ void tab_read64_slow(const DevTable& t, double r, double* v, double* dv, unsigned* status) {
    tab_read64(t, r, *v, *dv, status);
}

// The knot next to k, and the offset from it; d: the offset from knot k.
__device__ __noinline__ int knot64_next(const DevTable& t, double rval, int k, double* d) {
    k = min(k + (__double_as_longlong(*d) < 0 ? -1 : 1), t.n - 2);
    *d = fma(-(double)k, t.dr64, rval);
    return k;
}

// double to float by the bits (truncated; normal, positive, in float's range)
__device__ __forceinline__ float d2f_bits(double d) {
    const int hi = __double2hiint(d), lo = __double2loint(d);
    return __int_as_float(__funnelshift_l(lo, hi - 0x38000000, 3));
}

constexpr int P64_BLOCK = 32;  // one warp a block: the pipe is shared evenly (4,000 atoms: 30.9 us, 33.7 at 128)

// LANES lanes per atom take every LANES-th row entry, and the lanes' FP64
// sums meet in a fixed xor tree.
template <int LANES>
__global__ void __launch_bounds__(P64_BLOCK) k_pair64(PairParams p, const double* __restrict__ x,
                                                const double* __restrict__ y, const double* __restrict__ z,
                                                const int* __restrict__ type, const unsigned* __restrict__ nbr,
                                                const int* __restrict__ nnb, double* __restrict__ f64,
                                                float* __restrict__ pe, float* __restrict__ vir, unsigned* status) {
    const int lane = threadIdx.x & (LANES - 1);
    const int at = blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
    const bool valid = at < p.n;
    const int i = valid ? at : p.n - 1;
    const int ti = type[i];
    const double xi = x[i], yi = y[i], zi = z[i];
    const double xm = xi - p.L64[0], xp = xi + p.L64[0], ym = yi - p.L64[1], yp = yi + p.L64[1], zm = zi - p.L64[2],
                 zp = zi + p.L64[2];
    double ax = 0, ay = 0, az = 0, ae = 0, av = 0;
    const bool any = valid && (p.all_types || ti == p.ta || ti == p.tb);
    const int m = any ? nnb[i] : 0;
    const long long rc_bits = __double_as_longlong(p.rc64);
    const unsigned long long dr_bits = (unsigned long long)__double_as_longlong(p.phi.dr64);
    for (int s = lane; s < m; s += LANES) {
        const unsigned e = __ldg(&nbr[nbr_at(i, s, p.hshift, p.maxnb)]);
        const int j = nbr_index(e);
        if (!p.all_types && !types_match(ti, type[j], p.ta, p.tb)) continue;
        const int sx = nbr_sx(e), sy = nbr_sy(e), sz = nbr_sz(e);
        const double dx = (sx == 0 ? xi : (sx > 0 ? xm : xp)) - x[j];
        const double dy = (sy == 0 ? yi : (sy > 0 ? ym : yp)) - y[j];
        const double dz = (sz == 0 ? zi : (sz > 0 ? zm : zp)) - z[j];
        const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
        double w;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(w) : "d"(r2));
        const double err = fma(-(r2 * w), w, 1.0);
        double rinv = fma(fma(0.375, err, 0.5), w * err, w);
        double r = r2 * rinv;
        r = fma(fma(-r, r, r2), 0.5 * rinv, r);  // the root to half an ulp, as the reference's
        const bool tiny = __double_as_longlong(r2) < 0x3D70000000000000ll;  // r below 2^-20: the estimate may not hold
        if (tiny) {
            r = __dsqrt_rn(r2);
            rinv = 1.0 / r;
        }
        if (!(__double_as_longlong(r) < rc_bits)) continue;  // r < rc, on the bits of non-negative doubles
        const double rval = r - p.phi.off64;
        double ph, dph;
        // at or below the first knot, or a table so long that FP32 may miss its knot by one
        if (tiny || __double_as_longlong(rval) < (1ll << 52) || p.phi.n > (1 << 16)) {
            tab_read64_slow(p.phi, r, &ph, &dph, status);
        } else {
            int k = min((int)(d2f_bits(rval) * p.phi.inv_dr), p.phi.n - 2);
            double d = fma(-f2d_exact((float)k), p.phi.dr64, rval);
            if ((unsigned long long)__double_as_longlong(d) >= dr_bits) k = knot64_next(p.phi, rval, k, &d);
            const double4_32a cf = p.phi.coef64[k];
            const double u = fma(d, cf.x, cf.y), h = fma(d, u, cf.z);
            ph = fma(d, h, cf.w);
            dph = fma(d, fma(d, cf.x, u), h);
            if (p.phi.rmult) {
                ph *= rinv;
                dph = (dph - ph) * rinv;
            }
        }
        const double fr = -dph * rinv;
        ax = fma(dx, fr, ax);
        ay = fma(dy, fr, ay);
        az = fma(dz, fr, az);
        ae = fma(0.5, ph, ae);
        av = fma(fr, r2, av);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
        ae += __shfl_xor_sync(0xffffffffu, ae, o);
        av += __shfl_xor_sync(0xffffffffu, av, o);
    }
    if (lane != 0 || !valid) return;
    if (p.first) {
        f64[3 * (size_t)i + 0] = ax;
        f64[3 * (size_t)i + 1] = ay;
        f64[3 * (size_t)i + 2] = az;
        pe[i] = (float)ae;
        vir[i] = (float)av;
        f64[3 * (size_t)p.n + i] = ae;
    } else if (m) {
        f64[3 * (size_t)i + 0] += ax;
        f64[3 * (size_t)i + 1] += ay;
        f64[3 * (size_t)i + 2] += az;
        pe[i] += (float)ae;
        vir[i] += (float)av;
        f64[3 * (size_t)p.n + i] += ae;
    }
}

template <int LANES>
static void launch64(Context* c, const PairParams& p) {
    k_pair64<LANES><<<grid_for(c->n, P64_BLOCK / LANES), P64_BLOCK, 0, c->stream>>>(
        p, c->x, c->y, c->z, c->type, reinterpret_cast<const unsigned*>(c->nbr), c->nnb, c->f64, c->pe, c->vir,
        c->d_status);
}

// Few lanes an atom waste the least on ragged rows and on the sums' exchange,
// many shorten the dependent chain where the chip is not full (a warp alone
// takes about 2 us per row entry).  LJ argon, 79 entries, us with 8 / 16 / 32
// lanes: 500 atoms 27.4 / 18.6 / 13.8, 1,372 27.4 / 19.1 / 18.8, 2,048 28.4 /
// 21.5 / 24.4, 2,916 29.0 / 26.6 / 31.4, 4,000 33.1 / 33.6 / 41.0, 16,384 103 / 111 /
// 140.  (8 and 16 meet between 3,000 and 4,000 atoms, where they are within 8 %.)
static void launch64(Context* c, const PairParams& p) {
    if (c->n >= 20 * c->num_sms) launch64<8>(c, p);
    else if (c->n >= 8 * c->num_sms) launch64<16>(c, p);
    else launch64<32>(c, p);
}

constexpr int PAIR_TYPED_PER_SM = 256;  // atoms per SM from which typed pairs compact their rows

template <int LANES>
static void launch32(Context* c, const PairParams& p, int block) {
    // below this a warp per 32 atoms would not fill the chip
    if (!p.all_types && c->n >= PAIR_TYPED_PER_SM * c->num_sms) {
        k_pair32_typed<LANES><<<grid_for(c->n, 256), 256, 0, c->stream>>>(
            p, c->pack, c->type, reinterpret_cast<const unsigned*>(c->nbr), c->nnb, c->fx, c->fy, c->fz, c->pe,
            c->vir, c->d_status, c->nbmask);
        return;
    }
    int per_block = block / LANES;
    k_pair32<LANES><<<grid_for(c->n, per_block), block, 0, c->stream>>>(
        p, c->pack, reinterpret_cast<const unsigned*>(c->nbr), c->nnb, c->fx, c->fy, c->fz, c->pe, c->vir,
        c->d_status, c->nbmask);
}

int pair_launch(Context* c, Potential& pot, bool first) {
    PairParams p;
    p.n = c->n;
    p.hshift = c->nbr_hshift;
    p.maxnb = c->maxnb;
    p.L = make_shift(c->box);
    for (int d = 0; d < 3; d++) p.L64[d] = c->box.L[d];
    p.phi = pot.dt[0];
    p.rc64 = pot.t0.max_range();
    p.rc = (float)p.rc64;
    p.rc2 = p.rc * p.rc * 1.0001f;
    p.ta = pot.ta;
    p.tb = pot.tb;
    p.all_types = c->ntypes == 1 ? 1 : 0;
    p.first = first ? 1 : 0;
    p.rep_L = c->nrep > 0 ? static_cast<const ShiftF*>(c->d_rep_shift) : nullptr;
    p.rep_of = c->nrep > 0 ? c->d_rep_of : nullptr;
    if (pot.fp64 && c->nrep > 0) return set_error(c, OMDG_EINVAL, "replica mode has no FP64 pair kernel");
    int block = c->pair_block;
    if (pot.fp64) {
        prof_begin(c, "pair64");
        launch64(c, p);
    } else {
        prof_begin(c, "pair32");
        switch (c->pair_lanes) {
            case 1: launch32<1>(c, p, block); break;
            case 2: launch32<2>(c, p, block); break;
            case 4: launch32<4>(c, p, block); break;
            case 8: launch32<8>(c, p, block); break;
            case 16: launch32<16>(c, p, block); break;
            default: launch32<32>(c, p, block); break;
        }
    }
    prof_end(c);
    c->launches++;
    return check_cuda(c, cudaGetLastError(), "pair");
}

}  // namespace omdg
