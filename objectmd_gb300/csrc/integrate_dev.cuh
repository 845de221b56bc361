// Device side of the integrator shared by the kick kernel (integrate.cu) and
// the force kernels that take the second half-kick into their epilogue
// (eam_fast.cu): the step state, the kick parameters, and the energy ledger's
// block partials and last-block finalisation.
#pragma once

#include "rows.cuh"

namespace omdg {

struct StepState {
    long long step;      // RunKernel Step (system.cpp:979)
    int row;             // ledger row within the current omdg_step call
    int rebuild;         // rebuild request for the next list build
    double lambda;       // velocity factor to apply before the next kick
    int rebuild_every;   // >0: rebuild when step % rebuild_every == 0
    int nrebuild;        // list builds taken by the graph's conditional node
    double dt;               // TimeStep (DynamicTimeStep changes it here, between steps)
    double hdtm[MAX_TYPES];  // (dt/2) / m per type, refreshed with dt
    double elapsed;          // ElapsedTime (system.cpp:979)
    double sqrmaxv;          // SqrMaxVelocity of the last measurement (system.cpp:1075-1094)
    int src_first;           // EnergySource: the first call inside the window only arms it
    int src_scale;           // EnergySource: scale velocities at the next PreIntegration
    int halted;              // a rebuild overflowed its rows: later rebuilds are skipped until omdg_sync recovers
    int rebuild_all;         // replica mode: the request covers every replica (periodic rebuild, state upload)
    int building;            // small boxes: this step's rebuild kernels run (k_sort_small)
};

struct IntParams {
    int n;
    double org[3], P[3];
    float half_skin2;       // (skin/2)^2
    int use_f64;
    double Q[3];            // P - org: the pack coordinate is X = x + Q
    float Qh[3], Ql[3];     // Q as an FP32 pair (pack_coord)
    float mh[MAX_TYPES], ml[MAX_TYPES];  // mass per type as an FP32 pair
    int range_on;                        // RangeLimiter (RangeLimiter.h:33-54)
    unsigned range_group;                // group bits it acts on
    double range_lo[3], range_hi[3];     // box -/+ border
    int need_vmax;                       // measure SqrMaxVelocity (DynamicTimeStep)
};

struct FinParams {
    int natoms;
    int ledger_cap;
    int count_step;       // 1: this is a RunKernel step (advance Step)
    const int* ghosts;    // reference compatibility: periodic images added to the atom count (or null)
    unsigned* status;     // ERR_NONFINITE when a total is NaN or infinite
    unsigned* ticket;     // blocks done (the last one resets it)
    double tau, inv_tau;  // thermostat (tau <= 0: off)
    double kin_set;       // kinetic energy of an atom at Tset: Tset / (2/3/k_B) (unit.h:66-104)
    int need_vmax;        // SqrMaxVelocity from the block partials
    int dyn_update;       // DynamicTimeStep period (0: off; DynamicTimeStep.h:58-70)
    int dyn_apply;        // this measurement precedes a step's PreIntegration
    double dyn_maxpath, dyn_maxdt;
    double mass[MAX_TYPES];
    int src_on;                 // EnergySource (EnergySource.h:103-133)
    double src_start, src_stop;
};

// Block partials: sum m v^2, sum potential, sum virial as FP32 pairs, and
// the block's largest squared speed as the bit pattern of a non-negative
// double (integer order is value order): two float4 per block.
struct BlockPartial {
    float4 ke, wv;  // (k.hi, k.lo, e.hi, e.lo), (w.hi, w.lo, vmax bits low, high)
};

__device__ __forceinline__ unsigned long long vmax_bits(const float4& wv) {
    return ((unsigned long long)__float_as_uint(wv.w) << 32) | __float_as_uint(wv.z);
}

// sqrt(1 + a (b / k - 1)) as N / sqrt(N k) with N = k + a (b - k): one root's
// estimate and a third-order step (Householder; the estimate is good to 2^-20)
// in place of a division, a root and what lies between them (2,660 cycles from
// the sums to the factor in one thread, 2,050 now: FP64 latency).  Outside the estimate's safe range
// the plain form.
__device__ __forceinline__ double thermo_factor(double a, double b, double k) {
    const double N = fma(a, b - k, k), M = N * k;
    if (!(M > 1e-280 && M < 1e280)) return sqrt(1. + a * (b / k - 1.));
    double w;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(w) : "d"(M));
    const double err = fma(-(M * w), w, 1.0);
    return N * fma(fma(0.375, err, 0.5), w * err, w);
}

// A block's sums of the three ledger terms of its T threads, and the largest
// squared speed, in shared memory: one warp for each sum adds T / 32 terms a
// lane and then a fixed xor tree (450 instructions for 256 threads; a tree in
// every warp took 1,800).  Ends with a barrier.
template <int T>
struct LedgerSums {
    F2 terms[3][T], sums[3];
    unsigned long long vmax[T / 32];
    // what the last block reads of the step's state, and what follows from it
    int slot, row, rebuild, dyn, thermo;
    long long step;
    double elapsed, dt, a, b;

    __device__ __forceinline__ void add(F2 k, F2 e, F2 w, unsigned long long vm, int need_vmax) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        terms[0][threadIdx.x] = k;
        terms[1][threadIdx.x] = e;
        terms[2][threadIdx.x] = w;
        if (need_vmax) {
            for (int o = 16; o > 0; o >>= 1) vm = max(vm, __shfl_xor_sync(0xffffffffu, vm, o));
            if (lane == 0) vmax[warp] = vm;
        }
        __syncthreads();
        if (warp < 3) {
            F2 q = terms[warp][lane];
#pragma unroll 8
            for (int j = 1; j < T / 32; j++) q = f2_add(q, terms[warp][32 * j + lane]);
            for (int o = 16; o > 0; o >>= 1) q = f2_add(q, f2_shfl_xor(q, o));
            if (lane == 0) sums[warp] = q;
        }
        __syncthreads();
    }
    __device__ __forceinline__ unsigned long long largest(int need_vmax) const {
        unsigned long long v = 0ull;
        if (need_vmax)
            for (int q = 0; q < T / 32; q++) v = max(v, vmax[q]);
        return v;
    }
    // By one thread, ahead of the sums: the state's loads and what follows from
    // them alone.
    __device__ __forceinline__ void prepare(const FinParams& p, const StepState* st) {
        step = st->step;
        row = st->row;
        slot = row % p.ledger_cap;  // ring buffer between host reads
        elapsed = st->elapsed;
        dt = st->dt;
        const long long after = step + (p.count_step ? 1 : 0);
        const int every = st->rebuild_every;
        rebuild = p.count_step && every > 0 && after % every == 0;
        dyn = p.dyn_update > 0 && p.dyn_apply && after % p.dyn_update == 0;
        thermo = p.count_step && p.tau > 0.0 && step != 0;
        if (thermo) {
            const double count = (double)p.natoms + (p.ghosts ? (double)*p.ghosts : 0.0);
            a = dt * p.inv_tau;
            b = p.kin_set * count;
        }
    }
    // By one thread: ledger row, thermostat factor and step counter.
    __device__ __forceinline__ void finish(const FinParams& p, double* __restrict__ ledger, StepState* st) const {
        const double kinetic = 0.5 * f2_to_double(sums[0]), e = f2_to_double(sums[1]), w = f2_to_double(sums[2]);
        if (!(isfinite(kinetic) && isfinite(e))) atomicOr(p.status, ERR_NONFINITE);
        double* out = ledger + LEDGER_W * (size_t)slot;
        out[0] = kinetic;
        out[1] = e;
        out[2] = 0.5 * w;
        out[4] = (double)step;  // SysMonitor's Step, ElapsedTime and TimeStep of this step
        out[5] = elapsed;
        out[6] = dt;
        out[7] = 0.0;
        double lam = 1.0;
        // TempController::PostIntegration: lambda^2 = 1 + dt/tau (Tset/T - 1),
        // with Tset/T as the quotient of the kinetic energies
        if (thermo && kinetic > 0.0) lam = thermo_factor(a, b, kinetic);
        out[3] = lam;
        const double sqrmaxv = __longlong_as_double((long long)largest(p.need_vmax));
        if (p.need_vmax) st->sqrmaxv = sqrmaxv;
        if (p.count_step) {
            const double now = elapsed + dt;  // ElapsedTime += TimeStep; Step++ (system.cpp:979-980)
            st->lambda = lam;
            st->elapsed = now;
            st->step = step + 1;
            st->row = row + 1;
            if (rebuild) {
                st->rebuild = 1;
                st->rebuild_all = 1;
            }
            if (p.src_on) {  // EnergySource::PreIntegration of the next step
                int scale = 0;
                if (now >= p.src_start) {
                    if (st->src_first) st->src_first = 0;  // firstcall: return
                    else scale = now < p.src_stop ? 1 : 0;
                }
                st->src_scale = scale;
            }
        }
        if (dyn) {
            // DynamicTimeStep::PreIntegration of the next step
            const double v2 = p.need_vmax ? sqrmaxv : st->sqrmaxv;
            double ndt = p.dyn_maxdt;
            if (v2 > 0.0) {
                ndt = p.dyn_maxpath / (sqrt(v2) * 1.10);
                if (ndt > p.dyn_maxdt) ndt = p.dyn_maxdt;
            }
            st->dt = ndt;
            for (int t = 0; t < MAX_TYPES; t++) st->hdtm[t] = p.mass[t] > 0 ? (0.5 * ndt) / p.mass[t] : 0.0;
        }
        *p.ticket = 0u;
    }
};

constexpr int LEDGER_PREPARE = 96;  // the thread that prepares: the first one outside the summing warps

// Ledger row, thermostat factor and step counter from the block partials, by
// one block of T threads (FP32 pairs; FP64 only for the totals), which has
// prepared.  Partials are read through L2: other blocks wrote them.
template <int T>
__device__ __forceinline__ void finalize_block(LedgerSums<T>& s, const FinParams& p, int nblocks,
                                               const BlockPartial* partial, double* ledger, StepState* st) {
    F2 k = {0.f, 0.f}, e = {0.f, 0.f}, w = {0.f, 0.f};
    unsigned long long vm = 0ull;
#pragma unroll 4
    for (int b = threadIdx.x; b < nblocks; b += T) {
        const float4 ke = __ldcg(&partial[b].ke), wv = __ldcg(&partial[b].wv);
        k = f2_add(k, F2{ke.x, ke.y});
        e = f2_add(e, F2{ke.z, ke.w});
        w = f2_add(w, F2{wv.x, wv.y});
        if (p.need_vmax) vm = max(vm, vmax_bits(wv));
    }
    s.add(k, e, w, vm, p.need_vmax);
    if (threadIdx.x == 0) s.finish(p, ledger, st);
}

// What the neighbours' centre passes left for atom i (three-body kernels), in
// the slots of its own row's hits, added to its own part.  Four slots' loads
// are in flight at a time.  The row's other entries count as the zeros that
// they are: one of them after a hit folds a compensation of just half a unit
// in the last place into the sum (to even), and the rest change nothing.
struct SlotArgs {
    int hshift, maxnb;
    const int* nnb;
    const float4* slot;
    RowHits hits;
    int zero_virial;  // the reference SW does not accumulate a virial (sw.cpp:238)
};

__device__ __forceinline__ void slot_sum(const SlotArgs& a, int i, float& fx, float& fy, float& fz, float& pe) {
    Kahan gx, gy, gz, ge;
    gx.add(fx);
    gy.add(fy);
    gz.add(fz);
    ge.add(pe);
    const int m = a.nnb[i];
    int w0 = 0, s = -1;
    do {
        unsigned bits = a.hits.word(i, w0);
        while (bits) {
            float4 c[4];
            bool gap[4];
            int nk = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (bits) {
                    const int next = w0 + __ffs(bits) - 1;
                    gap[k] = next != s + 1;
                    s = next;
                    bits &= bits - 1u;
                    nk++;
                }
                c[k] = __ldg(a.slot + nbr_at(i, s, a.hshift, a.maxnb));
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < nk) {
                    if (gap[k]) gx.add(0.f), gy.add(0.f), gz.add(0.f), ge.add(0.f);
                    gx.add(c[k].x);
                    gy.add(c[k].y);
                    gz.add(c[k].z);
                    ge.add(c[k].w);
                }
        }
        w0 += 32;
    } while (w0 < m);
    if (s + 1 < m) gx.add(0.f), gy.add(0.f), gz.add(0.f), ge.add(0.f);
    fx = gx.value();
    fy = gy.value();
    fz = gz.value();
    pe = ge.value();
}

// One atom's second half-kick v += dt/2 f/m (of ux, uy, uz) and
// its ledger terms: m v^2 and the potential and virial as FP32 pairs, the
// squared speed's bits for DynamicTimeStep.  f is FP32 (the FP64 force path
// does not fuse).
__device__ __forceinline__ void kick_atom_terms(const IntParams& p, int i, int t, float fxi, float fyi, float fzi,
                                                float pei, float viri, double h, double& ux, double& uy, double& uz,
                                                F2& k, F2& e, F2& w, unsigned long long& vmax) {
    ux = fma(f2d_exact(fxi), h, ux);
    uy = fma(f2d_exact(fyi), h, uy);
    uz = fma(f2d_exact(fzi), h, uz);
    const F2 sx = f2_from(ux), sy = f2_from(uy), sz = f2_from(uz);
    const F2 v2 = f2_add(f2_add(f2_mul(sx, sx), f2_mul(sy, sy)), f2_mul(sz, sz));
    k = f2_add(k, f2_mul(v2, F2{p.mh[t], p.ml[t]}));
    e = f2_add(e, F2{pei, 0.f});
    w = f2_add(w, F2{viri, 0.f});
    if (p.need_vmax)  // sqrv = vx*vx + vy*vy + vz*vz (system.cpp:1086)
        vmax = max(vmax, (unsigned long long)__double_as_longlong(
                             __dadd_rn(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)), __dmul_rn(uz, uz))));
}

// The block's ledger partial from every thread's terms; the last block to
// finish sums the partials and writes the ledger row (finalize_block); a block
// alone has the sums.  Every thread of a block of T calls it, and its
// LEDGER_PREPARE-th has prepared.  What comes after the atoms is a chain of
// latencies in one block, the same for 512 atoms and a million: 12,000 cycles
// with a tree in every warp, fences around the ticket, the state's loads and
// three FP64 divisions in the thread that had the sums; some 6,500 now with the
// ticket and the partials, 3,800 without (one block).
// True in the thread that finished, when that asked for a periodic rebuild.
template <int T>
__device__ __forceinline__ bool ledger_block(LedgerSums<T>& s, const IntParams& p, const FinParams& f, F2 k, F2 e,
                                             F2 w, unsigned long long vmax, BlockPartial* __restrict__ partial,
                                             double* __restrict__ ledger, StepState* st) {
    __shared__ bool last;
    s.add(k, e, w, vmax, p.need_vmax);
    if (gridDim.x == 1) {
        if (threadIdx.x == 0) s.finish(f, ledger, st);
        return threadIdx.x == 0 && s.rebuild;
    }
    if (threadIdx.x == 0) {
        const unsigned long long bv = s.largest(p.need_vmax);
        partial[blockIdx.x].ke = make_float4(s.sums[0].hi, s.sums[0].lo, s.sums[1].hi, s.sums[1].lo);
        partial[blockIdx.x].wv = make_float4(s.sums[2].hi, s.sums[2].lo, __uint_as_float((unsigned)bv),
                                             __uint_as_float((unsigned)(bv >> 32)));
        // releases this partial, and acquires all others in the last block
        unsigned done;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(done) : "l"(f.ticket) : "memory");
        last = done == gridDim.x - 1;
    }
    __syncthreads();
    if (last) finalize_block<T>(s, f, gridDim.x, partial, ledger, st);
    return last && threadIdx.x == 0 && s.rebuild;
}

// One warp's ledger partial (the per-warp half of ledger_block): lane 0
// writes it.
__device__ __forceinline__ void warp_partial(const IntParams& p, F2 k, F2 e, F2 w, unsigned long long vmax,
                                             BlockPartial* __restrict__ out) {
    if (p.need_vmax)
        for (int o = 16; o > 0; o >>= 1) vmax = max(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    for (int o = 16; o > 0; o >>= 1) {
        k = f2_add(k, f2_shfl_xor(k, o));
        e = f2_add(e, f2_shfl_xor(e, o));
        w = f2_add(w, f2_shfl_xor(w, o));
    }
    if ((threadIdx.x & 31) == 0) {
        out->ke = make_float4(k.hi, k.lo, e.hi, e.lo);
        out->wv = make_float4(w.hi, w.lo, __uint_as_float((unsigned)vmax), __uint_as_float((unsigned)(vmax >> 32)));
    }
}

// Host: the kick's parameters for a context (integrate.cu).
struct KickArgs {
    IntParams p;
    FinParams f;
    BlockPartial* partial;  // one per block of the launch
    int partial_cap;
    StepState* st;
};

// The slot gather's arguments (threebody.cu).
SlotArgs slot_args(const Context* c, bool zero_virial);

bool kick_fusable(const Context* c);
void kick_args(Context* c, KickArgs& ka);
// One block sums nparts warp partials in order and writes the step's ledger row.
void launch_ledger_finalize(Context* c, const KickArgs& ka, int nparts);

}  // namespace omdg
