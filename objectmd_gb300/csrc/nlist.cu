// Linked-cell binning by counting sort and the Verlet-list build
// (replaces VerletList::Update, VerletList.cpp:126-199, and
// VerletListFull::Update, VerletListFull.cpp:138-230, together with the
// periodic ghost images of comhandler.cpp:288-377).
//
// Rebuild pipeline, all on the context stream:
//   1 cell_assign   wrap periodic owners into the box (systemgrid.cpp:129-151),
//                   cell of every atom, per-cell counts
//   2 scan          exclusive scan of the counts -> cell starts
//   3 scatter       atom -> slot in its cell
//   4 cell_sort     sort each cell's slots by previous index (deterministic order)
//   5 permute       reorder every per-atom array into cell order; position
//                   packs, displacement reference, screening positions
//                   (1 to 5 are k_sort_small in a small box or replica)
//   6 build         full list, slot-major nbr[s*n+i]; FP32 screen, FP64 tie-break
//   7 reverse       (three-body kernels) slot of i in each neighbour's row
#include <algorithm>
#include <cmath>

#include <climits>

#include <cooperative_groups.h>

#include "integrate_dev.cuh"

namespace omdg {

struct CellGeom {
    int nc[3];
    double org[3], h[3], inv_h[3];
    int periodic[3];
    double lo[3], L[3];
};

static CellGeom cell_geom(const Context* c) {
    CellGeom g;
    for (int d = 0; d < 3; d++) {
        g.nc[d] = c->box.nc[d];
        g.org[d] = c->box.cell_org[d];
        g.h[d] = c->box.cell_h[d];
        g.inv_h[d] = 1.0 / c->box.cell_h[d];
        g.periodic[d] = c->box.periodic[d];
        g.lo[d] = c->box.lo[d];
        g.L[d] = c->box.L[d];
    }
    return g;
}

// systemgrid.cpp:132-138: an atom is owned iff floor((x - x0) / lx) == 0,
// else it becomes the image x -/+ lx (comhandler.cpp:427-432).  Out of line:
// only atoms that crossed a face get here.
__device__ __noinline__ double wrap_crossed(double p, double lo, double L) {
    const int u = (int)floor(__ddiv_rn(__dsub_rn(p, lo), L));
    if (u < 0) return __dadd_rn(p, L);
    if (u >= 1) return __dadd_rn(p, -L);
    return p;
}

// Cell coordinate along one axis, wrapping p on a periodic axis first.  For
// a = p - x0 and lx positive, floor(a / lx) == 0 is 0 <= a < lx (a < lx gives
// fl(a / lx) < 1, a >= lx gives fl(a / lx) >= 1), tested on the bit patterns
// (non-negative doubles order as integers; NaN fails).  The cell is
// floor(a / h) by the reciprocal (the FP64 pipe divides slowly); cells are
// at least Rv (1 + 1e-12) wide, so a few ulps of misplacement at a face
// never separates a pair within Rv by more than one cell.  Periodic axes
// have their cell origin at x0.
__device__ __forceinline__ int axis_cell_of(double& p, int periodic, double lo, double L, double cell_org,
                                            double inv_h, int nc) {
    double a = __dsub_rn(p, periodic ? lo : cell_org);
    if (periodic) {
        const long long ba = __double_as_longlong(a);
        if (!(ba >= 0 && ba < __double_as_longlong(L))) {
            p = wrap_crossed(p, lo, L);
            a = __dsub_rn(p, lo);
        }
    }
    const int k = (int)floor(__dmul_rn(a, inv_h));
    return k < 0 ? 0 : (k >= nc ? nc - 1 : k);
}

// Wraps atom i's position into the box and returns its cell.
__device__ __forceinline__ int cell_of(int i, double* p, const CellGeom& g, unsigned* status) {
    const int cx = axis_cell_of(p[0], g.periodic[0], g.lo[0], g.L[0], g.org[0], g.inv_h[0], g.nc[0]);
    const int cy = axis_cell_of(p[1], g.periodic[1], g.lo[1], g.L[1], g.org[1], g.inv_h[1], g.nc[1]);
    const int cz = axis_cell_of(p[2], g.periodic[2], g.lo[2], g.L[2], g.org[2], g.inv_h[2], g.nc[2]);
    if (isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2])) return (cz * g.nc[1] + cy) * g.nc[0] + cx;
    // spread non-finite atoms over the cells so that the per-cell work stays
    // bounded; the run is already invalid and the status word says so
    atomicOr(status, ERR_NONFINITE);
    return i % (g.nc[0] * g.nc[1] * g.nc[2]);
}

__global__ void k_cell_assign(int n, double* __restrict__ x, double* __restrict__ y, double* __restrict__ z,
                              CellGeom g, int* __restrict__ cell, int* __restrict__ count, unsigned* status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double p[3] = {x[i], y[i], z[i]};
    const int c = cell_of(i, p, g, status);
    x[i] = p[0];
    y[i] = p[1];
    z[i] = p[2];
    cell[i] = c;
    atomicAdd(&count[c], 1);
}

// Exclusive scan of count[0..m) into start[0..m] in three launches: each
// block scans a tile of SCAN_TILE cells (k_scan_tiles), one block scans the
// tile totals (k_scan_totals), and k_scan_add adds the tile offsets.  The
// order of every sum is fixed.
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_PER = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_PER;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(int m, const int* __restrict__ count,
                                                             int* __restrict__ start, int* __restrict__ tile_sum) {
    __shared__ int warp_tot[SCAN_THREADS / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int base = blockIdx.x * SCAN_TILE + t * SCAN_PER;
    int v[SCAN_PER];
    int own = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) {
        v[k] = base + k < m ? count[base + k] : 0;
        own += v[k];
    }
    int incl = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = lane < SCAN_THREADS / 32 ? warp_tot[lane] : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        if (lane < SCAN_THREADS / 32) warp_tot[lane] = w;  // inclusive
    }
    __syncthreads();
    int run = incl - own + (warp > 0 ? warp_tot[warp - 1] : 0);
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) {
        if (base + k < m) start[base + k] = run;
        run += v[k];
    }
    if (t == SCAN_THREADS - 1) tile_sum[blockIdx.x] = warp_tot[SCAN_THREADS / 32 - 1];
}

// One block: tile totals -> exclusive tile offsets; start[m] = total.
// (and clears umax for the permutation, which packs)
__global__ void k_scan_totals(int ntiles, int m, int* __restrict__ tile_sum, int* __restrict__ start,
                              unsigned* umax) {
    __shared__ int warp_sum[32];
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31;
    if (t == 0) *umax = 0u;
    const int chunk = (ntiles + nt - 1) / nt;
    const int b = t * chunk, e = min(ntiles, b + chunk);
    int s = 0;
    for (int k = b; k < e; k++) s += tile_sum[k];
    int run = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += u;
    }
    if (lane == 31) warp_sum[t >> 5] = run;
    __syncthreads();
    if (t < 32) {
        int w = t < (nt >> 5) ? warp_sum[t] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        warp_sum[t] = w;
    }
    __syncthreads();
    if (t >= 32) run += warp_sum[(t >> 5) - 1];
    if (t == nt - 1) start[m] = run;
    run -= s;
    for (int k = b; k < e; k++) {
        const int c = tile_sum[k];
        tile_sum[k] = run;
        run += c;
    }
}

__global__ void k_scan_add(int m, int* __restrict__ start, const int* __restrict__ tile_off) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) start[k] += tile_off[k / SCAN_TILE];
}

// Replica filters of a partial rebuild: only atoms (by index) and cells of
// replicas whose flag is set take part; a null flag array takes everything.
__device__ __forceinline__ bool rep_on(const int* __restrict__ flag, const int* __restrict__ rep, int k) {
    return !flag || flag[rep[k]] != 0;
}

__global__ void k_scatter(int n, const int* __restrict__ cell, const int* __restrict__ start, int* __restrict__ fill,
                          int* __restrict__ perm, const int* __restrict__ rep_of, const int* __restrict__ rflag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !rep_on(rflag, rep_of, i)) return;
    int c = cell[i];
    int s = start[c] + atomicAdd(&fill[c], 1);
    perm[s] = i;
}

// Atomic slot order is arbitrary; sorting each cell by previous index makes
// the final order (and every later floating-point sum) deterministic.
constexpr int CELL_SORT_MAX = 1024;

// Cells of up to CELL_SORT_SMALL atoms, one thread each: the indices sort in
// registers by an odd-even transposition network (fully unrolled).
constexpr int CELL_SORT_SMALL = 8;

// Cells too large for it go to a queue (big[0] of them, cells from big[1])
// that k_cell_sort_warp then drains, so that the warps do not walk every
// cell of a sparse grid.
__global__ void k_cell_sort_small(int m, const int* __restrict__ start, int* __restrict__ perm,
                                  const int* __restrict__ cell_rep, const int* __restrict__ rflag,
                                  int* __restrict__ big) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m || !rep_on(rflag, cell_rep, c)) return;
    const int b = start[c], k = start[c + 1] - b;
    if (k > CELL_SORT_SMALL) big[1 + atomicAdd(big, 1)] = c;
    if (k <= 1 || k > CELL_SORT_SMALL) return;
    int v[CELL_SORT_SMALL];
#pragma unroll
    for (int q = 0; q < CELL_SORT_SMALL; q++) v[q] = q < k ? perm[b + q] : INT_MAX;
#pragma unroll
    for (int r = 0; r < CELL_SORT_SMALL; r++) {
#pragma unroll
        for (int q = r & 1; q + 1 < CELL_SORT_SMALL; q += 2) {
            const int lo = min(v[q], v[q + 1]), hi = max(v[q], v[q + 1]);
            v[q] = lo;
            v[q + 1] = hi;
        }
    }
#pragma unroll
    for (int q = 0; q < CELL_SORT_SMALL; q++)
        if (q < k) perm[b + q] = v[q];
}

// Larger cells, one warp each (k_cell_sort_small takes the cells of at most
// `skip` atoms when it runs): for cells of
// up to 32 atoms each lane holds one atom index and its rank (how many of the
// cell's indices are smaller) is counted with shuffles; the lanes then write
// in place.  Cells of more than 32 atoms take lane 0's insertion sort; a
// pathological cell beyond CELL_SORT_MAX is left unsorted (its order is then
// not reproducible) rather than sorted in O(k^2).
__global__ void k_cell_sort_warp(int m, const int* __restrict__ start, int* __restrict__ perm, int skip,
                                 const int* __restrict__ cell_rep, const int* __restrict__ rflag,
                                 const int* __restrict__ big) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int total = big ? big[0] : m;  // queued cells, or every cell
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total; w += warps) {
        const int c = big ? big[1 + w] : w;
        if (!rep_on(rflag, cell_rep, c)) continue;  // uniform over the warp
        const int b = start[c], k = start[c + 1] - b;
        if (k <= skip) continue;  // empty, single, or sorted by k_cell_sort_small
        if (k <= 32) {
            const int v = lane < k ? perm[b + lane] : INT_MAX;
            int r = 0;
            for (int q = 0; q < k; q++) r += __shfl_sync(0xffffffffu, v, q) < v;
            __syncwarp();
            if (lane < k) perm[b + r] = v;
        } else if (lane == 0 && k <= CELL_SORT_MAX) {
            for (int p = b + 1; p < b + k; p++) {
                const int v = perm[p];
                int q = p - 1;
                while (q >= b && perm[q] > v) {
                    perm[q + 1] = perm[q];
                    q--;
                }
                perm[q + 1] = v;
            }
        }
        __syncwarp();
    }
}


// Per-atom state that survives a rebuild, gathered into staging and copied
// back so every array keeps its address (a captured step graph replays the
// same pointers).
struct AtomArrays {
    double *x, *y, *z, *vx, *vy, *vz;
    int *type, *id;
    unsigned* flag;
    double* extra;   // optional per-atom FP64 state (extra_n values per atom, slot-major)
    int extra_n;
};

// Replica mode: every replica has its own periodic lengths and cell grid,
// and its cells occupy the global cell range [cell_base, cell_base + cells).
struct RepGeom {
    double lo[3], L[3], cell_org[3], cell_h[3], inv_h[3];
    int nc[3], periodic[3];
    int cell_base;
    ShiftF S;
};

// The pack coordinate is X = x + Q with Q = P - org, formed as FP32 hi + lo
// by pack_coord (the integrator refreshes the pack with the same function).
struct PackFrame {
    float Qh[3], Ql[3];
};

struct Corner {
    double lo[3];
};

// loc: the position from the box's (or the replica's) lower corner lo, rounded
// to FP32, which the list build screens (w: the type).  From the origin the
// band of pairs that take the FP64 test would grow with the box's distance from
// it: 256,000 EAM atoms, build and sort 254 us at the origin, 586 at an offset
// of 3e4 A, 3,550 at 1e6 A; now 254 at all three.
// One atom's packs; returns its share of umax.
__device__ __forceinline__ float pack_atom(int i, double X, double Y, double Z, int type, bool active,
                                           const PackFrame& f, const double* lo, PosPack* __restrict__ pack,
                                           float4* __restrict__ xref, float4* __restrict__ loc) {
    PosPack p;
    pack_coord(X, f.Qh[0], f.Ql[0], p.hi.x, p.lo.x);
    pack_coord(Y, f.Qh[1], f.Ql[1], p.hi.y, p.lo.y);
    pack_coord(Z, f.Qh[2], f.Ql[2], p.hi.z, p.lo.z);
    p.hi.w = __int_as_float(type);
    p.lo.w = 0.f;
    pack[i] = p;
    if (xref) xref[i] = make_float4(p.hi.x, p.hi.y, p.hi.z, 0.f);
    if (!loc) return 0.f;
    if (!active) {
        // inactive (SetActive false): far from every centre, so no list takes
        // it, and outside the band's max |x|
        loc[i] = make_float4(3.0e38f, 3.0e38f, 3.0e38f, 0.f);
        return 0.f;
    }
    const float ux = f2_from(X - lo[0]).hi, uy = f2_from(Y - lo[1]).hi, uz = f2_from(Z - lo[2]).hi;
    loc[i] = make_float4(ux, uy, uz, p.hi.w);
    const float m = fmaxf(fabsf(ux), fmaxf(fabsf(uy), fabsf(uz)));
    return m <= 3.0e38f ? m : 3.0e38f;  // non-finite: flagged by the cell assignment
}

// The largest |x - lo| sets the width of the screening band.  Whole warps.
__device__ __forceinline__ void pack_umax(float m, unsigned* umax) {
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    if ((threadIdx.x & 31) == 0 && m > 0.f && __float_as_uint(m) > *(volatile unsigned*)umax)
        atomicMax(umax, __float_as_uint(m));
}

// Also writes the sorted atoms' cells and the caller-to-sorted map (the new
// position k of caller atom id[o]).
// The permutation into the staging arrays, and the packs while the position is
// at hand (a pass of its own read it back: sort and pack of 512,000 atoms 112.7
// -> 99.5 us).
__global__ void k_permute_gather(int n, const int* __restrict__ perm, AtomArrays a, AtomArrays st,
                                 const int* __restrict__ cell_old, int* __restrict__ cell_new,
                                 int* __restrict__ inv, const int* __restrict__ rep_of,
                                 const int* __restrict__ rflag, PackFrame f, Corner corner,
                                 const RepGeom* __restrict__ rg, const unsigned* __restrict__ aflag,
                                 PosPack* __restrict__ pack, float4* __restrict__ xref, float4* __restrict__ loc,
                                 unsigned* umax) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    float u = 0.f;
    if (k < n && rep_on(rflag, rep_of, k)) {  // a replica's atoms stay in its index range
        int o = perm[k];
        cell_new[k] = cell_old[o];
        inv[a.id[o]] = k;
        const double X = a.x[o], Y = a.y[o], Z = a.z[o];
        const int type = a.type[o];
        const unsigned flag = a.flag[o];
        st.x[k] = X;
        st.y[k] = Y;
        st.z[k] = Z;
        st.vx[k] = a.vx[o];
        st.vy[k] = a.vy[o];
        st.vz[k] = a.vz[o];
        st.type[k] = type;
        st.id[k] = a.id[o];
        st.flag[k] = flag;
        for (int q = 0; q < a.extra_n; q++) st.extra[(size_t)q * n + k] = a.extra[(size_t)q * n + o];
        u = pack_atom(k, X, Y, Z, type, !aflag || (flag & 1u), f, rg ? rg[rep_of[k]].lo : corner.lo, pack, xref, loc);
    }
    pack_umax(u, umax);
}

// The state a rebuild reorders, copied before the rebuild of a step (unless
// an earlier rebuild of the queued steps overflowed: then the copy of that
// rebuild's input is kept), with the step state.
// Only the first rebuild of the queued steps takes it (taken is cleared when
// a new batch of steps starts and set after the copy): a recovery restores
// that earlier state and replays from there, which reaches the same state.
__global__ void k_snapshot(int n, const int* __restrict__ halted, const int* __restrict__ taken, AtomArrays a,
                           AtomArrays snap, const unsigned char* __restrict__ st, unsigned char* __restrict__ st_snap,
                           int st_bytes, const unsigned* __restrict__ status, int* __restrict__ errors) {
    if (*halted || *taken) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *errors = (int)*status;
    if (k < st_bytes) st_snap[k] = st[k];
    if (k >= n) return;
    snap.x[k] = a.x[k];
    snap.y[k] = a.y[k];
    snap.z[k] = a.z[k];
    snap.vx[k] = a.vx[k];
    snap.vy[k] = a.vy[k];
    snap.vz[k] = a.vz[k];
    snap.type[k] = a.type[k];
    snap.id[k] = a.id[k];
    snap.flag[k] = a.flag[k];
}

__global__ void k_set_one(int* p) { *p = 1; }

// An overflowed build halts the queued steps' later rebuilds.
__global__ void k_halt_on_overflow(const unsigned* __restrict__ status, int* halted) {
    if (*status & ERR_NBR_OVERFLOW) *halted = 1;
}

__global__ void k_permute_copyback(int n, AtomArrays st, AtomArrays a, const int* __restrict__ rep_of,
                                   const int* __restrict__ rflag) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || !rep_on(rflag, rep_of, k)) return;
    a.x[k] = st.x[k];
    a.y[k] = st.y[k];
    a.z[k] = st.z[k];
    a.vx[k] = st.vx[k];
    a.vy[k] = st.vy[k];
    a.vz[k] = st.vz[k];
    a.type[k] = st.type[k];
    a.id[k] = st.id[k];
    a.flag[k] = st.flag[k];
    for (int q = 0; q < a.extra_n; q++) a.extra[(size_t)q * n + k] = st.extra[(size_t)q * n + k];
}

__global__ void k_zero_ints(int m, int* __restrict__ a, int* __restrict__ b) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) {
        a[k] = 0;
        b[k] = 0;
    }
}

// The cell counters of the flagged replicas (and the sentinel past the last cell).
__global__ void k_zero_cells_rep(int m, int* __restrict__ count, int* __restrict__ fill,
                                 const int* __restrict__ cell_rep, const int* __restrict__ rflag) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > m || (k < m && !rep_on(rflag, cell_rep, k))) return;
    count[k] = 0;
    fill[k] = 0;
}

// After a build: count it for each replica rebuilt and clear the flags
// (all replicas after a full build).
__global__ void k_rep_build_done(int nrep, int full, int* __restrict__ rflag, int* __restrict__ builds) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrep; r += gridDim.x * blockDim.x) {
        if (full || rflag[r]) builds[r] += 1;
        rflag[r] = 0;
    }
}


__global__ void k_pack(int n, const double* __restrict__ x, const double* __restrict__ y,
                       const double* __restrict__ z, const int* __restrict__ type, PackFrame f,
                       PosPack* __restrict__ pack) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pack_atom(i, x[i], y[i], z[i], type[i], true, f, nullptr, pack, nullptr, nullptr);
}

// EAM cell tiles: besides the list entry, the build writes each entry's
// slot in the staged halo of its centre's tile (tile t, halo cell h:
// sb[t HC + h] + the candidate's offset in its cell).  Halo cells run z, y, x
// from the cell below the tile's first to the one above its last, the order
// the build visits a row's cells, so slots increase along a row.
struct TileOut {
    unsigned short* slot;  // null: no tile output
    const unsigned short* sb;
    const int* nst;
    int T[3], nt[3];
    int hx, hy;            // halo cells along x, y (T + 2)
    int HC, stride, cap;
};

struct BuildParams {
    const int *list, *list_n;  // partial replica build: the rebuilt atoms (else null)
    const int* on;  // build only if set (a small box's step; else null)
    TileOut to;
    int n, maxnb, hshift;
    int cap;              // LANES = 1: row entries a thread keeps in shared memory
    int nc[3];
    int periodic[3];
    ShiftF L;
    double L64[3];
    double rsq;           // Rv*Rv in FP64 (VerletList.cpp:161)
    float rv;             // Rv rounded to FP32
    float corner_err;     // FP64 rounding of two atoms' x - lo
    float lmax;           // largest periodic length (screening band)
};

// Per axis, how many (cell, image) candidates a cell has and the idx-th one,
// in traversal order: cells c-1, c, c+1 (a periodic axis wraps them with
// image -1 / +1, a free axis drops the ones off the grid); a periodic axis
// of fewer than 3 cells takes every cell with images -1, 0, +1.
__device__ __forceinline__ int axis_count(int nc, int periodic) { return (periodic && nc < 3) ? 3 * nc : 3; }

__device__ __forceinline__ bool axis_cell(int c, int nc, int periodic, int idx, int& cell, int& shift) {
    if (periodic) {
        if (nc >= 3) {
            int k = c + idx - 1;
            shift = 0;
            if (k < 0) {
                k += nc;
                shift = -1;
            } else if (k >= nc) {
                k -= nc;
                shift = 1;
            }
            cell = k;
        } else {
            cell = idx / 3;
            shift = idx % 3 - 1;
        }
        return true;
    }
    const int k = c + idx - 1;
    cell = k;
    shift = 0;
    return k >= 0 && k < nc;
}

// The candidates along x of the cells a..b as runs of consecutive cells under
// one image (the atoms of consecutive cells lie back to back): the cells
// a-1..b+1, cut where a periodic axis wraps; a periodic axis of fewer than 3
// cells gives one run per (cell, image).
__device__ __forceinline__ int axis_runs(int a, int b, int nc, int periodic) {
    if (!periodic) return 1;
    if (nc < 3) return 3 * nc;
    return 1 + (a == 0) + (b == nc - 1);
}

__device__ __forceinline__ void axis_run(int a, int b, int nc, int periodic, int idx, int& c0, int& c1, int& shift) {
    if (periodic && nc < 3) {
        c0 = c1 = idx / 3;
        shift = idx % 3 - 1;
        return;
    }
    if (periodic && a == 0) idx--;  // run -1: the last cell's image below
    shift = idx < 0 ? -1 : idx;
    c0 = idx < 0 ? nc - 1 : (idx == 0 ? max(a - 1, 0) : 0);
    c1 = idx < 0 ? nc - 1 : (idx == 0 ? min(b + 1, nc - 1) : 0);
}

// A pair inside the FP32 screening band, or closer than it can tell from an
// overlap: the reference's FP64 test (dx = x_i - (x_j + s), r2 = (dx*dx +
// dy*dy) + dz*dz <= Rv^2) and its overlap check (gadget.cpp:149).  Rare, out
// of line.
__device__ __noinline__ bool exact_within(double Lx, double Ly, double Lz, double rsq, const double* __restrict__ x,
                                          const double* __restrict__ y, const double* __restrict__ z, int i, int k,
                                          unsigned code, unsigned* status) {
    const int sx = nbr_sx(code), sy = nbr_sy(code), sz = nbr_sz(code);
    double gx = sx == 0 ? 0.0 : (sx > 0 ? Lx : -Lx);
    double gy = sy == 0 ? 0.0 : (sy > 0 ? Ly : -Ly);
    double gz = sz == 0 ? 0.0 : (sz > 0 ? Lz : -Lz);
    double dx = __dsub_rn(x[i], __dadd_rn(x[k], gx));
    double dy = __dsub_rn(y[i], __dadd_rn(y[k], gy));
    double dz = __dsub_rn(z[i], __dadd_rn(z[k], gz));
    double rr = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    if (!(rr <= rsq)) return false;
    if (rr < OMD_PROXIMITY) report_overlap(status, i, k);
    return true;
}

// The list build.  The candidates of the 27 cells are 9 runs of back-to-back
// atoms (axis_run); a candidate costs one 16-byte load of its FP32 position,
// six of them in flight, and the squared length of the difference.  Every
// FP32 step errs by at most an ulp of the box's extent, so pairs within a band of
// Rv (a few 1e-4 A for boxes of a few hundred A: one atom in thirty has such
// a pair), and pairs close enough to be an overlap, take the reference's FP64
// test, out of line: the list is the reference's exactly, in the traversal
// order of the cells.
//
// Accepted entries wait in a shared-memory column per thread: some lane of
// the warp accepts nearly every candidate, so the append has to be a
// predicated store and an add, not a branch around address arithmetic.
//
// LANES = 1: one thread per centre walks every run; its column holds the
// whole row (longer ones go out in pieces) and goes out as whole 32-byte
// sectors of the sliced layout.  Bound by instruction issue and the latency
// of the loads (370 warp instructions per EAM atom at 53 % issue; six loads
// in flight: with four 165 us, with eight 170).  256,000 EAM atoms, 13 a
// cell: 154 us, against 498 us for one CTA per cell on hi/lo packs and 200
// for one thread per centre with a loop per cell; 512,000 Tersoff atoms, 1.6
// a cell: 90 us against 113.  One warp per cell, its lanes over the
// candidates and eight centres in registers, took 239 us on EAM: appending
// by ballot or by bit mask costs more instructions than the loads it saves.
//
// LANES = 8, for boxes too small to fill the chip with a thread per centre:
// eight lanes take a run each, and after each round of eight runs the lanes'
// counts are scanned to place their entries.
constexpr int BUILD_THREADS = 128;
constexpr int BUILD_AHEAD = LOC_PAD;  // candidate loads in flight per thread
constexpr int BUILD_RUN = 32;      // LANES = 8: a lane's entries of one run in shared memory

// One run of candidates for the centre at (px, py, pz): the accepted entries
// go to the column at w (stride BUILD_THREADS), which out() empties when it
// is full.
template <bool ONE, class Out, class Slot>
__device__ __forceinline__ void build_run(const float4* __restrict__ u, int left, unsigned ent, unsigned self_ent,
                                          float px, float py, float pz, float rsq_lo, float rsq_hi, float rsq_ov,
                                          const double* __restrict__ x, const double* __restrict__ y,
                                          const double* __restrict__ z, int i, double rsq, double Lx, double Ly,
                                          double Lz, unsigned* status, unsigned*& w, const unsigned* w_full,
                                          unsigned& tmask, Out&& out, Slot&& slot) {
    const unsigned band = __float_as_uint(rsq_hi) - __float_as_uint(rsq_lo);
#pragma unroll 1
    for (; left > 0; left -= BUILD_AHEAD, u += BUILD_AHEAD, ent += BUILD_AHEAD) {
        if (w > w_full) out();
        float4 uk[BUILD_AHEAD];
#pragma unroll
        for (int t = 0; t < BUILD_AHEAD; t++) uk[t] = __ldg(u + t);  // the array is padded
        float r2[BUILD_AHEAD];
        bool in[BUILD_AHEAD];
        bool rare = false;
#pragma unroll
        for (int t = 0; t < BUILD_AHEAD; t++) {
            const float dx = px - uk[t].x, dy = py - uk[t].y, dz = pz - uk[t].z;
            r2[t] = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            in[t] = r2[t] <= rsq_hi && t < left;
            rare |= (__float_as_uint(r2[t]) - __float_as_uint(rsq_lo)) <= band || r2[t] < rsq_ov;
        }
        if (rare) {  // one in the band, the centre itself or an overlap
#pragma unroll
            for (int t = 0; t < BUILD_AHEAD; t++) {
                if (ent + t == self_ent) in[t] = false;
                if (in[t] && (r2[t] >= rsq_lo || r2[t] < rsq_ov))
                    in[t] = exact_within(Lx, Ly, Lz, rsq, x, y, z, i, (int)(ent & (unsigned)INDEX_MASK) + t, ent,
                                         status);
            }
        }
#pragma unroll
        for (int t = 0; t < BUILD_AHEAD; t++) {
            if (!ONE && in[t]) tmask |= 1u << (__float_as_int(uk[t].w) & 31);
            if (in[t]) {
                slot((int)(ent & (unsigned)INDEX_MASK) + t);
                *w = ent + t;
                w += BUILD_THREADS;
            }
        }
    }
}

// REP: the centre's replica supplies the grid and lengths.  TILES (LANES = 1):
// the rows also go out as EAM tile slots.  ONE: a single atom type (no type
// mask).
constexpr int BUILD_CTAS_PER_SM = 7;

template <int LANES, bool REP, bool TILES, bool ONE>
__device__ __forceinline__ void build_centre(
    const BuildParams& p, int i, int lane, const RepGeom* __restrict__ rg, const int* __restrict__ rep_of,
    const float4* __restrict__ loc, const double* __restrict__ x, const double* __restrict__ y,
    const double* __restrict__ z, const int* __restrict__ cell, const int* __restrict__ start,
    const unsigned* __restrict__ umax, unsigned* __restrict__ nbr, int* __restrict__ nnb, unsigned* status, int* need,
    unsigned* __restrict__ nbmask) {
    extern __shared__ unsigned s_row[];
    const RepGeom* g = REP ? rg + rep_of[i] : nullptr;
    const float4 ui = loc[i];
    if (ui.x == 3.0e38f) {  // inactive centre (pack_atom): an empty row
        if (lane == 0) {
            nnb[i] = 0;
            nbmask[i] = 0u;
        }
        return;
    }
    // band: per component the two positions, the image length and two
    // differences each round by half an ulp of at most U; 2x margin, sqrt(3)
    // for the length and 1e-6 relative for the squares
    const float U = __uint_as_float(*umax) + p.lmax;
    const float dlt = 1.7320509f * (6.f * U * 1.1920929e-7f + p.corner_err) + 1e-6f * p.rv;
    const float rl = fmaxf(p.rv - dlt, 0.f), rh = p.rv + dlt, ro = 1.0e-3f + dlt;
    const float rsq_lo = rl * rl * (1.f - 1e-6f), rsq_hi = rh * rh * (1.f + 1e-6f), rsq_ov = ro * ro;
    const int nx = REP ? g->nc[0] : p.nc[0], ny = REP ? g->nc[1] : p.nc[1], nz = REP ? g->nc[2] : p.nc[2];
    const int perx = REP ? g->periodic[0] : p.periodic[0], pery = REP ? g->periodic[1] : p.periodic[1],
              perz = REP ? g->periodic[2] : p.periodic[2];
    const int cbase = REP ? g->cell_base : 0;
    const ShiftF& L = REP ? g->S : p.L;
    const double* L64 = REP ? g->L : p.L64;
    const int ci = cell[i] - cbase;
    const int cx = ci % nx, cy = (ci / nx) % ny, cz = ci / (nx * ny);
    const int mx = axis_runs(cx, cx, nx, perx), my = axis_count(ny, pery), mz = axis_count(nz, perz);
    const unsigned self_ent = nbr_encode(i, 0, 0, 0);
    unsigned tmask = 0u;  // types the row holds
    unsigned* const out = nbr + nbr_at(i, 0, p.hshift, p.maxnb);
    unsigned* const col = s_row + threadIdx.x;
    unsigned* w = col;
    const unsigned* const w_full = col + ((LANES == 1 ? p.cap : BUILD_RUN) - BUILD_AHEAD) * BUILD_THREADS;
    int cnt = 0;  // entries of the row already out
    // tile slots (single box only): the centre's tile, where it is staged
    const unsigned short* tsb = nullptr;
    unsigned short* trow = nullptr;
    int tox = 0, toy = 0, toz = 0;
    if (TILES) {
        const int tx = cx / p.to.T[0], ty = cy / p.to.T[1], tz = cz / p.to.T[2];
        const int tt = (tz * p.to.nt[1] + ty) * p.to.nt[0] + tx;
        if (p.to.nst[tt] <= p.to.cap) {
            tsb = p.to.sb + (size_t)tt * p.to.HC;
            trow = p.to.slot + (size_t)i * p.to.stride;
            tox = cx - tx * p.to.T[0];
            toy = cy - ty * p.to.T[1];
            toz = cz - tz * p.to.T[2];
        }
    }
    const auto flush = [&]() {
        const int m = (int)(w - col) / BUILD_THREADS;
        const int put = min(m, p.maxnb - cnt);
        for (int s = 0; s < put; s++) out[(size_t)(cnt + s) << p.hshift] = col[s * BUILD_THREADS];
        cnt += m;
        w = col;
    };
    // run (a, b, q): its cells, image and candidates
    const auto run = [&](int a, int b, int q, auto&& emit) {
        int kz, sz, ky, sy, c0, c1, sx;
        if (!axis_cell(cz, nz, perz, a, kz, sz) || !axis_cell(cy, ny, pery, b, ky, sy)) return;
        axis_run(cx, cx, nx, perx, q, c0, c1, sx);
        const int row0 = cbase + (kz * ny + ky) * nx;
        const int k0 = start[row0 + c0], e = start[row0 + c1 + 1];
        // slot of candidate k in the tile's staged halo: tb + k (halo cells
        // along x are staged back to back, as the run is)
        int tb = 0;
        if (TILES && trow) {
            const int hx = sx < 0 ? 0 : (sx > 0 ? 2 : c0 - cx + 1);  // the run's first halo cell
            tb = (int)tsb[((toz + a) * p.to.hy + (toy + b)) * p.to.hx + (tox + hx)] - k0;
        }
        build_run<ONE>(loc + k0, e - k0, nbr_encode(k0, sx, sy, sz), self_ent, ui.x - sel_shift(sx, L.hx),
                       ui.y - sel_shift(sy, L.hy), ui.z - sel_shift(sz, L.hz), rsq_lo, rsq_hi, rsq_ov, x, y, z, i,
                       p.rsq, L64[0], L64[1], L64[2], status, w, w_full, tmask, emit, [&](int k) {
                           if (TILES && trow) {
                               const int at = cnt + (int)(w - col) / BUILD_THREADS;
                               if (at < p.maxnb) trow[at] = (unsigned short)(tb + k);
                           }
                       });
    };
    if (LANES == 1) {
#pragma unroll 1
        for (int a = 0; a < mz; a++)
#pragma unroll 1
            for (int b = 0; b < my; b++)
#pragma unroll 1
                for (int q = 0; q < mx; q++) run(a, b, q, flush);
        flush();
    } else {
        const unsigned group = 0xffu << (threadIdx.x & 24);
        const int runs = mx * my * mz;
#pragma unroll 1
        for (int r0 = 0; r0 < runs; r0 += LANES) {
            // a run of more than BUILD_RUN accepted entries is placed by
            // walking it twice: once to count, once from its place
            const int r = r0 + lane;
            const int q = r % mx, b = (r / mx) % my, a = r / (mx * my);
            int spilled = 0;
            w = col;
            if (r < runs)
                run(a, b, q, [&]() {
                    spilled += (int)(w - col) / BUILD_THREADS;
                    w = col;
                });
            const int m = (int)(w - col) / BUILD_THREADS;
            int incl = spilled + m;
            for (int o = 1; o < LANES; o <<= 1) {
                const int v = __shfl_up_sync(group, incl, o, LANES);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(group, incl, LANES - 1, LANES);
            const int row_cnt = cnt;
            cnt += incl - spilled - m;  // this lane's first place
            if (spilled) {
                w = col;
                run(a, b, q, flush);
                flush();
            } else {
                flush();
            }
            cnt = row_cnt + total;
            w = col;
        }
        if (!ONE)
            for (int o = 1; o < LANES; o <<= 1) tmask |= __shfl_xor_sync(group, tmask, o, LANES);
        if (lane != 0) return;
    }
    if (cnt > p.maxnb) {
        atomicOr(status, ERR_NBR_OVERFLOW);
        atomicMax(need, cnt);
        cnt = p.maxnb;
    }
    nnb[i] = cnt;
    nbmask[i] = ONE ? (cnt > 0 ? 1u : 0u) : tmask;
}

// A partial replica build goes over p.list (the atoms of the rebuilt replicas,
// p.list_n of them) with a resident grid.
template <int LANES, bool REP, bool TILES, bool ONE>
__global__ void __launch_bounds__(BUILD_THREADS, BUILD_CTAS_PER_SM) k_build(
    BuildParams p, const RepGeom* __restrict__ rg, const int* __restrict__ rep_of, const float4* __restrict__ loc,
    const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
    const int* __restrict__ cell, const int* __restrict__ start, const unsigned* __restrict__ umax,
    unsigned* __restrict__ nbr, int* __restrict__ nnb, unsigned* status, int* need, const int* __restrict__ rflag,
    unsigned* __restrict__ nbmask) {
    if (p.on && !*p.on) return;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (REP && p.list) {
        const int total = *p.list_n;
        for (; t / LANES < total; t += gridDim.x * blockDim.x)  // LANES = 8: whole groups go on together
            build_centre<LANES, REP, TILES, ONE>(p, p.list[t / LANES], t % LANES, rg, rep_of, loc, x, y, z, cell,
                                                 start, umax, nbr, nnb, status, need, nbmask);
        return;
    }
    const int i = t / LANES;
    if (i >= p.n) return;  // LANES = 8: whole groups leave together
    if (REP && rflag && !rflag[rep_of[i]]) return;  // the replica keeps its list
    build_centre<LANES, REP, TILES, ONE>(p, i, t % LANES, rg, rep_of, loc, x, y, z, cell, start, umax, nbr, nnb,
                                         status, need, nbmask);
}

// ------------------------------------------------------------------ EAM cell tiles

struct TilePrep {
    int T[3], nt[3], nc[3], periodic[3];
    int hx, hy, HC;
    double corg[3], h[3];   // cell grid origin and widths
    double borg[3], P[3];   // pack frame: X = x - borg + P
};

// One CTA per tile: the atom count of each halo cell (z, y, x from the cell
// below the tile's first to the one above its last; a periodic axis wraps,
// a free axis has no cells beyond the grid), their exclusive scan as each
// cell's first staged slot (saturating at 65535; such a tile exceeds every
// capacity), the total, and the tile's lower corner in the pack frame.
constexpr int TILE_PREP_THREADS = 256;  // >= the 216 halo cells of a 4x4x4 tile

__global__ void __launch_bounds__(TILE_PREP_THREADS) k_tile_prep(TilePrep tp, const int* __restrict__ start,
                                                                 unsigned short* __restrict__ sb,
                                                                 int* __restrict__ nst, float4* __restrict__ org) {
    __shared__ int s_warp[TILE_PREP_THREADS / 32];
    const int t = blockIdx.x;
    const int tx = t % tp.nt[0], ty = (t / tp.nt[0]) % tp.nt[1], tz = t / (tp.nt[0] * tp.nt[1]);
    const int h = threadIdx.x;
    int cnt = 0;
    if (h < tp.HC) {
        const int l[3] = {h % tp.hx, (h / tp.hx) % tp.hy, h / (tp.hx * tp.hy)};
        const int t3[3] = {tx, ty, tz};
        int k[3];
        bool ok = true;
        for (int d = 0; d < 3; d++) {
            int gk = t3[d] * tp.T[d] - 1 + l[d];
            if (tp.periodic[d]) {
                if (gk < 0) gk += tp.nc[d];
                else if (gk >= tp.nc[d]) gk -= tp.nc[d];
            } else if (gk < 0 || gk >= tp.nc[d]) {
                ok = false;
            }
            k[d] = gk;
        }
        if (ok) {
            const int c = (k[2] * tp.nc[1] + k[1]) * tp.nc[0] + k[0];
            cnt = start[c + 1] - start[c];
        }
    }
    // block exclusive scan
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        int v = lane < TILE_PREP_THREADS / 32 ? s_warp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane < TILE_PREP_THREADS / 32) s_warp[lane] = v;
    }
    __syncthreads();
    const int excl = incl - cnt + (w > 0 ? s_warp[w - 1] : 0);
    if (h < tp.HC) sb[(size_t)t * tp.HC + h] = (unsigned short)min(excl, 65535);
    if (h == tp.HC - 1) nst[t] = excl + cnt;
    if (h == 0) {
        const int t3[3] = {tx, ty, tz};
        float o[3];
        for (int d = 0; d < 3; d++)
            o[d] = (float)(__dadd_rn(__dsub_rn(fma((double)(t3[d] * tp.T[d]), tp.h[d], tp.corg[d]), tp.borg[d]),
                                     tp.P[d]));
        org[t] = make_float4(o[0], o[1], o[2], 0.f);
    }
}

// ------------------------------------------------------------------ replicas

__global__ void k_cell_assign_rep(int n, double* __restrict__ x, double* __restrict__ y, double* __restrict__ z,
                                  const int* __restrict__ rep_of, const RepGeom* __restrict__ rg,
                                  int* __restrict__ cell, int* __restrict__ count, unsigned* status,
                                  const int* __restrict__ rflag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !rep_on(rflag, rep_of, i)) return;
    const RepGeom& g = rg[rep_of[i]];
    double p[3] = {x[i], y[i], z[i]};
    const int cx = axis_cell_of(p[0], g.periodic[0], g.lo[0], g.L[0], g.cell_org[0], g.inv_h[0], g.nc[0]);
    const int cy = axis_cell_of(p[1], g.periodic[1], g.lo[1], g.L[1], g.cell_org[1], g.inv_h[1], g.nc[1]);
    const int cz = axis_cell_of(p[2], g.periodic[2], g.lo[2], g.L[2], g.cell_org[2], g.inv_h[2], g.nc[2]);
    x[i] = p[0];
    y[i] = p[1];
    z[i] = p[2];
    int c = g.cell_base + (cz * g.nc[1] + cy) * g.nc[0] + cx;
    if (!(isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]))) {
        atomicOr(status, ERR_NONFINITE);
        c = g.cell_base + i % (g.nc[0] * g.nc[1] * g.nc[2]);
    }
    cell[i] = c;
    atomicAdd(&count[c], 1);
}

// rev at (i, s): the slot of (i, -image) in the row of j = nbr at (i, s).
// For every list entry (i, s) -> j, the slot of i in row j: REV_LANES
// threads per centre, each searching for every REV_LANES-th entry (the
// searches are independent chains of loads; lanes keep more of them in
// flight).  A search finds both entries of a pair, so only the lower atom
// searches: 194,184 Stillinger-Weber atoms 45.0 -> 36.4 us, 512,000 Tersoff
// atoms 22.5 -> 20.8.
constexpr int REV_LANES = 4;

__device__ __forceinline__ void reverse_centre(int i, int lane, int hshift, int maxnb,
                                               const unsigned* __restrict__ nbr, const int* __restrict__ nnb,
                                               int* __restrict__ rev, unsigned* status) {
    int m = nnb[i];
    for (int s = lane; s < m; s += REV_LANES) {
        unsigned e = nbr[nbr_at(i, s, hshift, maxnb)];
        int j = nbr_index(e);
        if (j < i) continue;  // j's search finds both
        unsigned want = nbr_encode(i, -nbr_sx(e), -nbr_sy(e), -nbr_sz(e));
        int mj = nnb[j], found = -1;
        for (int u = 0; u < mj; u++)
            if (nbr[nbr_at(j, u, hshift, maxnb)] == want) {
                found = u;
                break;
            }
        if (found < 0) atomicOr(status, ERR_NBR_OVERFLOW);
        else rev[nbr_at(j, found, hshift, maxnb)] = s;
        rev[nbr_at(i, s, hshift, maxnb)] = found < 0 ? 0 : found;
    }
}

__global__ void k_reverse(int n, int hshift, int maxnb, const unsigned* __restrict__ nbr,
                          const int* __restrict__ nnb, int* __restrict__ rev, unsigned* status,
                          const int* __restrict__ rep_of, const int* __restrict__ rflag,
                          const int* __restrict__ on, const int* __restrict__ list,
                          const int* __restrict__ list_n) {
    if (on && !*on) return;
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (list) {  // a partial replica build (k_build)
        const int total = *list_n;
        for (long q = t; q / REV_LANES < total; q += gridDim.x * (long)blockDim.x)
            reverse_centre(list[q / REV_LANES], (int)(q % REV_LANES), hshift, maxnb, nbr, nnb, rev, status);
        return;
    }
    const int i = (int)(t / REV_LANES), lane = (int)(t % REV_LANES);
    if (i >= n) return;
    if (rflag && !rflag[rep_of[i]]) return;  // the replica kept its rows, and so their reverse slots
    reverse_centre(i, lane, hshift, maxnb, nbr, nnb, rev, status);
}

// ---------------------------------------------------------------- host side

// Centres per SM up to which the list build takes eight lanes each: the chip
// holds 896 threads of it a SM, so a thread per centre fills a quarter of
// that or less.  14,212 EAM atoms: 25 us against 54; 4,000 LJ atoms (79 a row): 36
// against 90; 512 Tersoff atoms: 14 against 23.
constexpr int BUILD_SMALL_PER_SM = 256;

// Cells along an axis of extent ext: as many as fit with each at least
// Rv (1 + 1e-12) wide (the margin absorbs cell_coord's rounding).
static int cells_along(double ext, double rv) {
    const int nc = (int)(ext / (rv * (1.0 + 1e-12)));
    return nc < 1 ? 1 : nc;
}

void nlist_prepare_geometry(Context* c) {
    double rv = c->rc_max + c->skin;
    BoxGeom& b = c->box;
    for (int d = 0; d < 3; d++) {
        if (b.periodic[d]) {
            b.cell_org[d] = b.lo[d];
            b.nc[d] = cells_along(b.L[d], rv);
            b.cell_h[d] = b.L[d] / b.nc[d];
        } else {
            // free axis: a fixed grid over the box with a margin; atoms
            // beyond it are clamped into the edge cells, which keeps the
            // 27-cell search complete.
            double margin = 2.0 * rv;
            b.cell_org[d] = b.lo[d] - margin;
            double ext = b.L[d] + 2.0 * margin;
            b.nc[d] = cells_along(ext, rv);
            b.cell_h[d] = ext / b.nc[d];
        }
    }
}

// Cell grids of the replicas (same rules as nlist_prepare_geometry, per
// replica) and the replica of every atom; uploads both.
int replica_prepare(Context* c) {
    const double rv = c->rc_max + c->skin;
    std::vector<RepGeom> rg(c->nrep);
    std::vector<ShiftF> sh(c->nrep);
    int base = 0;
    double lmax = 0.0;
    for (int r = 0; r < c->nrep; r++) {
        RepGeom& g = rg[r];
        for (int d = 0; d < 3; d++) {
            g.lo[d] = c->rep_lo[3 * r + d];
            g.L[d] = c->rep_hi[3 * r + d] - c->rep_lo[3 * r + d];
            g.periodic[d] = c->rep_periodic[d];
            if (g.periodic[d]) {
                g.cell_org[d] = g.lo[d];
                g.nc[d] = cells_along(g.L[d], rv);
                g.cell_h[d] = g.L[d] / g.nc[d];
            } else {
                const double margin = 2.0 * rv;
                g.cell_org[d] = g.lo[d] - margin;
                const double ext = g.L[d] + 2.0 * margin;
                g.nc[d] = cells_along(ext, rv);
                g.cell_h[d] = ext / g.nc[d];
            }
            g.inv_h[d] = 1.0 / g.cell_h[d];
            if (g.periodic[d]) lmax = std::max(lmax, g.L[d]);
        }
        const float lh[3] = {(float)g.L[0], (float)g.L[1], (float)g.L[2]};
        g.S.hx = lh[0];
        g.S.hy = lh[1];
        g.S.hz = lh[2];
        g.S.lx = (float)(g.L[0] - (double)lh[0]);
        g.S.ly = (float)(g.L[1] - (double)lh[1]);
        g.S.lz = (float)(g.L[2] - (double)lh[2]);
        sh[r] = g.S;
        g.cell_base = base;
        base += g.nc[0] * g.nc[1] * g.nc[2];
    }
    c->rep_cells = base;
    c->rep_lmax = lmax;
    c->rep_max_atoms = c->rep_max_cells = 0;
    for (int r = 0; r < c->nrep; r++) {
        c->rep_max_atoms = std::max(c->rep_max_atoms, c->rep_start[r + 1] - c->rep_start[r]);
        c->rep_max_cells = std::max(c->rep_max_cells, (r + 1 < c->nrep ? rg[r + 1].cell_base : base) - rg[r].cell_base);
    }
    // The step graph holds these pointers: allocate once (omdg_set_replicas
    // frees them) and reallocate only for a larger atom capacity, dropping
    // the graph then.  Contents are rewritten in place.
    cudaError_t e = cudaSuccess;
    if (!c->d_rep_geom) e = cudaMalloc(&c->d_rep_geom, sizeof(RepGeom) * c->nrep);
    if (e == cudaSuccess && !c->d_rep_shift) e = cudaMalloc(&c->d_rep_shift, sizeof(ShiftF) * c->nrep);
    if (e == cudaSuccess && !c->d_rep_start) e = cudaMalloc(&c->d_rep_start, sizeof(int) * (c->nrep + 1));
    if (e == cudaSuccess && !c->d_rep_sums) e = cudaMalloc(&c->d_rep_sums, sizeof(double) * 2 * c->nrep);
    if (e == cudaSuccess && !c->d_rep_flag) {
        e = cudaMalloc(&c->d_rep_flag, sizeof(int) * c->nrep);
        if (e == cudaSuccess) e = cudaMemsetAsync(c->d_rep_flag, 0, sizeof(int) * c->nrep, c->stream);
    }
    if (e == cudaSuccess && !c->d_rep_builds) {
        e = cudaMalloc(&c->d_rep_builds, sizeof(int) * c->nrep);
        if (e == cudaSuccess) e = cudaMemsetAsync(c->d_rep_builds, 0, sizeof(int) * c->nrep, c->stream);
    }
    if (e == cudaSuccess && (!c->d_cell_rep || c->rep_cells_cap < base)) {
        cudaFree(c->d_cell_rep);
        c->d_cell_rep = nullptr;
        e = cudaMalloc(&c->d_cell_rep, sizeof(int) * std::max(1, base));
        c->rep_cells_cap = base;
        invalidate_graph(c);
    }
    if (e == cudaSuccess && (!c->d_rep_of || c->rep_of_cap < c->cap)) {
        cudaFree(c->d_rep_of);
        c->d_rep_of = nullptr;
        e = cudaMalloc(&c->d_rep_of, sizeof(int) * std::max(1, c->cap));
        c->rep_of_cap = c->cap;
        invalidate_graph(c);
    }
    if (e != cudaSuccess) return set_error(c, OMDG_ENOMEM, "replica tables");
    std::vector<int> of(c->n), cell_rep(std::max(1, base));
    for (int r = 0; r < c->nrep; r++)
        for (int i = c->rep_start[r]; i < c->rep_start[r + 1]; i++) of[i] = r;
    for (int r = 0; r < c->nrep; r++)
        for (int k = rg[r].cell_base; k < (r + 1 < c->nrep ? rg[r + 1].cell_base : base); k++) cell_rep[k] = r;
    cudaMemcpyAsync(c->d_cell_rep, cell_rep.data(), sizeof(int) * cell_rep.size(), cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(c->d_rep_geom, rg.data(), sizeof(RepGeom) * c->nrep, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(c->d_rep_shift, sh.data(), sizeof(ShiftF) * c->nrep, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(c->d_rep_of, of.data(), sizeof(int) * c->n, cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(c->d_rep_start, c->rep_start.data(), sizeof(int) * (c->nrep + 1), cudaMemcpyHostToDevice,
                    c->stream);
    return check_cuda(c, cudaStreamSynchronize(c->stream), "replica tables");
}

// The tiled EAM passes apply to one box (no replicas) whose periodic axes
// have at least three cells (the build's 27-cell stencil), with tiles of at
// most 4 cells a side.
int tile_prepare(Context* c) {
    c->tile_want = false;
    c->tile_valid = false;
    if (!tiles_apply(c)) return OMDG_OK;
    const BoxGeom& b = c->box;
    for (int d = 0; d < 3; d++) {
        if (b.periodic[d] && b.nc[d] < 3) return OMDG_OK;
        if (c->tile_dim[d] < 1 || c->tile_dim[d] > 4) return OMDG_OK;
    }
    int nt[3], hc = 1;
    for (int d = 0; d < 3; d++) {
        nt[d] = (b.nc[d] + c->tile_dim[d] - 1) / c->tile_dim[d];
        hc *= c->tile_dim[d] + 2;
    }
    const int ntiles = nt[0] * nt[1] * nt[2];
    if ((long long)ntiles * hc > c->tile_alloc || !c->tile_sb) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(c->stream, &cs);
        if (cs != cudaStreamCaptureStatusNone) return set_error(c, OMDG_ESTATE, "tile grid grew inside a capture");
        invalidate_graph(c);
        cudaFree(c->tile_sb);
        cudaFree(c->tile_nst);
        cudaFree(c->tile_org);
        c->tile_sb = nullptr;
        c->tile_nst = nullptr;
        c->tile_org = nullptr;
        c->tile_alloc = 0;
        if (cudaMalloc(&c->tile_sb, sizeof(unsigned short) * (size_t)ntiles * hc) != cudaSuccess ||
            cudaMalloc(&c->tile_nst, sizeof(int) * ntiles) != cudaSuccess ||
            cudaMalloc(&c->tile_org, sizeof(float4) * ntiles) != cudaSuccess)
            return set_error(c, OMDG_ENOMEM, "tile tables");
        c->tile_alloc = ntiles * hc;
    }
    for (int d = 0; d < 3; d++) c->tile_nt[d] = nt[d];
    c->tile_count = ntiles;
    c->tile_hc = hc;
    c->tile_want = true;
    return tile_reserve_slots(c);
}

// The slot rows: one per atom of the capacity, maxnb rounded up to 8 slots.
int tile_reserve_slots(Context* c) {
    if (!c->tile_want || c->maxnb <= 0) return OMDG_OK;
    const int stride = (c->maxnb + 7) & ~7;
    const size_t need = (size_t)c->cap * stride;
    if (need > c->tslot_alloc || !c->tslot) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(c->stream, &cs);
        if (cs != cudaStreamCaptureStatusNone) return set_error(c, OMDG_ESTATE, "tile slots grew inside a capture");
        invalidate_graph(c);
        cudaFree(c->tslot);
        c->tslot = nullptr;
        c->tslot_alloc = 0;
        if (cudaMalloc(&c->tslot, need * sizeof(unsigned short)) != cudaSuccess)
            return set_error(c, OMDG_ENOMEM, "tile slot rows");
        c->tslot_alloc = need;
    }
    if (stride != c->tile_stride) invalidate_graph(c);
    c->tile_stride = stride;
    return OMDG_OK;
}

void tile_release(Context* c) {
    cudaFree(c->tile_sb);
    cudaFree(c->tile_nst);
    cudaFree(c->tile_org);
    cudaFree(c->tslot);
    c->tile_sb = nullptr;
    c->tile_nst = nullptr;
    c->tile_org = nullptr;
    c->tslot = nullptr;
    c->tile_alloc = 0;
    c->tslot_alloc = 0;
    c->tile_want = false;
    c->tile_valid = false;
}

PackFrame pack_frame(const Context* c) {
    PackFrame f;
    for (int d = 0; d < 3; d++) {
        const double Q = c->box.P[d] - c->box.org[d];
        f.Qh[d] = (float)Q;
        f.Ql[d] = (float)(Q - (double)f.Qh[d]);
    }
    return f;
}

// The whole re-sort of a small box in one kernel, PER atoms a thread, one
// cluster: snapshot, wrap, count, scan, order, permute and pack.  An atom stays
// in its thread's registers from the first phase to the last, so the permutation needs no staging; a barrier of the
// cluster stands where the general path ends a kernel (14 of them).  Both with
// the pack, us with some 5 and 10 of launch: 512 atoms 15.2 and 58.6, 4,096 19.1
// and 64.2, 13,824 25.3 and 65.5, 32,768 42.1 and 65.9.  Same order as there: by cell, then by the old
// index; a cell of more than CELL_SORT_MAX atoms stays as it came.
// With `on_request` the kernel is part of every step and returns unless the
// step's kick_drift asked for a rebuild; the list kernels after it go by
// st->building: three launches that return cost less than a conditional node
// that is not taken.  A step of 512 Tersoff atoms, us: 23.5 and 28.4, of 8,000
// 26.5 and 31.1, of 32,768 31.1 and 36.0.
// Replicas: a cluster each, and those that keep their rows return at once,
// where the general path's eleven kernels went over every atom and cell; the
// list kernels go over the rebuilt atoms only.  A step of the impact ensemble
// (1.47 M atoms in 256 replicas, some of them rebuilt in every step), us: sort
// and pack 116 -> 66, build 74 -> 63, reverse 33 -> 18.
constexpr int SORT_THREADS = 1024, SORT_CTAS = 8;
constexpr int SORT_PER = 4, SORT_CELLS = 8;  // atoms a thread moves, and cells it scans, at most

struct SortArgs {
    int n, m, on_request, st_bytes;
    CellGeom g;
    PackFrame f;
    StepState* st;
    unsigned* status;
    int* taken;  // [1]: the error bits at the time
    AtomArrays a, snap;  // snap.x null: no snapshot
    unsigned char* st_snap;
    int *count, *start, *perm, *cell, *inv;
    const unsigned* aflag;  // null: every atom is active
    // replica mode: a cluster a replica, of those flagged (rflag null: of all)
    const RepGeom* rg;
    const int *rep_start, *rflag;
    int *list, *list_n;
    PosPack* pack;
    float4 *xref, *loc;
    unsigned* umax;
};

template <int PER, bool REP>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_small(SortArgs a) {
    static_assert(sizeof(StepState) <= SORT_THREADS, "a block copies the step state");
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    __shared__ int warp_sum[SORT_THREADS / 32], total, list_at;
    __shared__ CellGeom sg;
    const int rank = (int)cl.block_rank(), t = threadIdx.x, lane = t & 31;
    const int threads = (int)cl.num_blocks() * SORT_THREADS;
    const int i = rank * SORT_THREADS + t;
    // this cluster's atoms [a0, a0 + n) and cells [c0, c0 + m)
    int a0 = 0, n = a.n, c0 = 0, m = a.m;
    if (REP) {
        const int r = blockIdx.x / cl.num_blocks();
        if (a.rflag && !a.rflag[r]) return;  // the replica keeps its order and rows
        const RepGeom& g = a.rg[r];
        a0 = a.rep_start[r];
        n = a.rep_start[r + 1] - a0;
        c0 = g.cell_base;
        m = g.nc[0] * g.nc[1] * g.nc[2];
        if (t < 3) {
            sg.nc[t] = g.nc[t];
            sg.org[t] = g.cell_org[t];
            sg.h[t] = g.cell_h[t];
            sg.inv_h[t] = g.inv_h[t];
            sg.periodic[t] = g.periodic[t];
            sg.lo[t] = g.lo[t];
            sg.L[t] = g.L[t];
        }
        if (rank == 0 && t == 0 && a.rflag) list_at = atomicAdd(a.list_n, n);
    }
    const CellGeom& geom = REP ? sg : a.g;
    if (a.on_request) {
        // a build that overflowed its rows halts the queued steps' later ones
        const bool halted = a.st->halted || (a.st->building && (*a.status & ERR_NBR_OVERFLOW));
        const bool go = !halted && a.st->rebuild;
        cl.sync();  // every thread has read the same words before one changes them
        if (!go) {
            if (i == 0) {
                a.st->building = 0;
                if (halted) a.st->halted = 1;
            }
            return;
        }
    }
    const bool snap = !REP && a.snap.x && !a.st->halted && !*a.taken;
    const unsigned errors = *a.status;  // before this sort
    double p[PER][3], v[PER][3];
    int type[PER], id[PER], c[PER], slot[PER];
    unsigned flag[PER];
#pragma unroll
    for (int w = 0; w < PER; w++) {
        const int j = a0 + w * threads + i;
        if (j >= a0 + n) continue;
        p[w][0] = a.a.x[j];
        p[w][1] = a.a.y[j];
        p[w][2] = a.a.z[j];
        v[w][0] = a.a.vx[j];
        v[w][1] = a.a.vy[j];
        v[w][2] = a.a.vz[j];
        type[w] = a.a.type[j];
        id[w] = a.a.id[j];
        flag[w] = a.a.flag[j];
        if (snap) {
            a.snap.x[j] = p[w][0];
            a.snap.y[j] = p[w][1];
            a.snap.z[j] = p[w][2];
            a.snap.vx[j] = v[w][0];
            a.snap.vy[j] = v[w][1];
            a.snap.vz[j] = v[w][2];
            a.snap.type[j] = type[w];
            a.snap.id[j] = id[w];
            a.snap.flag[j] = flag[w];
        }
    }
    for (int q = i; q < m; q += threads) a.count[c0 + q] = 0;
    if (!REP && i == 0) *a.umax = 0u;
    cl.sync();  // the counts are zero, and `taken` read
    if (!REP && rank == 0) {
        if (t == 0 && a.on_request) {
            a.st->nrebuild += 1;
            a.st->rebuild = 0;
            a.st->rebuild_all = 0;
            a.st->building = 1;
        }
        if (snap) {  // the state as it is after the request was taken
            __syncthreads();
            if (t < a.st_bytes) a.st_snap[t] = reinterpret_cast<const unsigned char*>(a.st)[t];
            if (t == 0) {
                a.taken[0] = 1;
                a.taken[1] = (int)errors;
            }
        }
    }
#pragma unroll
    for (int w = 0; w < PER; w++) {
        const int j = a0 + w * threads + i;
        if (j >= a0 + n) continue;
        c[w] = c0 + cell_of(j, p[w], geom, a.status);
        slot[w] = atomicAdd(&a.count[c[w]], 1);
    }
    cl.sync();
    // exclusive scan: a thread's run of cells, the block's threads, the blocks
    const int per = (m + threads - 1) / threads;
    const int q0 = min(m, i * per), q1 = min(m, q0 + per);
    int cells[SORT_CELLS], sum = 0;
#pragma unroll
    for (int k = 0; k < SORT_CELLS; k++) {
        cells[k] = q0 + k < q1 ? a.count[c0 + q0 + k] : 0;
        sum += cells[k];
    }
    int run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += u;
    }
    if (lane == 31) warp_sum[t >> 5] = run;
    __syncthreads();
    if (t < 32) {
        int w = warp_sum[t];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        warp_sum[t] = w;
        if (t == 31) total = w;
    }
    cl.sync();
    run += a0 + (t >= 32 ? warp_sum[(t >> 5) - 1] : 0) - sum;
    for (int r = 0; r < rank; r++) run += *cl.map_shared_rank(&total, r);
#pragma unroll
    for (int k = 0; k < SORT_CELLS; k++)
        if (q0 + k < q1) {
            a.start[c0 + q0 + k] = run;
            run += cells[k];
        }
    if (i == 0 && a0 + n == a.n) a.start[c0 + m] = a.n;
    if (REP && a.rflag) {  // the rebuilt atoms, for the list kernels
        const int at = *cl.map_shared_rank(&list_at, 0);
        for (int q = i; q < n; q += threads) a.list[at + q] = a0 + q;
    }
    cl.sync();
#pragma unroll
    for (int w = 0; w < PER; w++)
        if (w * threads + i < n) a.perm[a.start[c[w]] + slot[w]] = a0 + w * threads + i;
    cl.sync();
    float u = 0.f;
#pragma unroll
    for (int w = 0; w < PER; w++) {
        const int j = a0 + w * threads + i;
        if (j >= a0 + n) continue;
        const int base = a.start[c[w]];
        const int in_cell = (c[w] + 1 < c0 + m ? a.start[c[w] + 1] : a0 + n) - base;
        if (in_cell <= CELL_SORT_MAX) {
            slot[w] = 0;
            for (int q = 0; q < in_cell; q++) slot[w] += a.perm[base + q] < j;
        }
        const int k = slot[w] = base + slot[w];
        a.a.x[k] = p[w][0];
        a.a.y[k] = p[w][1];
        a.a.z[k] = p[w][2];
        a.a.vx[k] = v[w][0];
        a.a.vy[k] = v[w][1];
        a.a.vz[k] = v[w][2];
        a.a.type[k] = type[w];
        a.a.id[k] = id[w];
        a.a.flag[k] = flag[w];
        a.cell[k] = c[w];
        a.inv[id[w]] = k;
        u = fmaxf(u, pack_atom(k, p[w][0], p[w][1], p[w][2], type[w], !a.aflag || (flag[w] & 1u), a.f, geom.lo, a.pack,
                               a.xref, a.loc));
    }
    pack_umax(u, a.umax);
    for (int q = 0; q < a.a.extra_n; q++) {
        double* x = a.a.extra + (size_t)q * a.n;
        double keep[PER];
#pragma unroll
        for (int w = 0; w < PER; w++) keep[w] = w * threads + i < n ? x[a0 + w * threads + i] : 0.0;
        cl.sync();
#pragma unroll
        for (int w = 0; w < PER; w++)
            if (w * threads + i < n) x[slot[w]] = keep[w];
    }
}

static int cells_of(const Context* c) { return c->box.nc[0] * c->box.nc[1] * c->box.nc[2]; }

// One cluster's share: its atoms and cells.
static bool sort_fits(long atoms, long cells) {
    return atoms <= SORT_CTAS * SORT_THREADS * SORT_PER && cells <= SORT_CTAS * SORT_THREADS * SORT_CELLS;
}

bool small_sort(const Context* c) {
    return c->nrep == 0 && !c->tile_want &&
           sort_fits(c->n, (long)c->box.nc[0] * c->box.nc[1] * c->box.nc[2]);
}

static int launch_sort_small(Context* c, const CellGeom& g, int m, bool on_request, unsigned* umax, const int* rflag,
                             int* list_n) {
    SortArgs a;
    a.n = c->n;
    a.m = m;
    a.on_request = on_request ? 1 : 0;
    a.st_bytes = (int)step_state_bytes();
    a.g = g;
    a.f = pack_frame(c);
    a.st = reinterpret_cast<StepState*>(c->d_state);
    a.status = c->d_status;
    a.taken = c->d_flags + 6;
    a.a = AtomArrays{c->x, c->y, c->z, c->vx, c->vy, c->vz, c->type, c->id, c->aflag, c->extra, c->extra_n};
    a.snap = AtomArrays{};
    if (c->build_in_step && c->snap_d)
        a.snap = AtomArrays{c->snap_d, c->snap_d + c->cap, c->snap_d + 2 * (size_t)c->cap, c->snap_d + 3 * (size_t)c->cap,
                            c->snap_d + 4 * (size_t)c->cap, c->snap_d + 5 * (size_t)c->cap, c->snap_i,
                            c->snap_i + c->cap, reinterpret_cast<unsigned*>(c->snap_i + 2 * (size_t)c->cap), nullptr, 0};
    a.st_snap = static_cast<unsigned char*>(c->snap_state);
    a.count = c->cell_count;
    a.start = c->cell_start;
    a.perm = c->perm;
    a.cell = c->cell_sorted;
    a.inv = c->inv;
    a.aflag = c->flags_used ? c->aflag : nullptr;
    a.pack = c->pack;
    a.xref = c->xref;
    a.loc = c->loc;
    a.umax = umax;
    a.rg = static_cast<const RepGeom*>(c->d_rep_geom);
    a.rep_start = c->d_rep_start;
    a.rflag = rflag;
    a.list = c->cell;  // (the general path's cell numbers)
    a.list_n = list_n;
    // a replica's cluster is as small as four atoms a thread allow: many run
    // beside each other
    const bool reps = c->nrep > 0;
    const int atoms = reps ? c->rep_max_atoms : c->n, cells = reps ? c->rep_max_cells : m;
    const int most = reps ? SORT_PER : 1;
    int blocks = 1;
    while (blocks < SORT_CTAS && (blocks * SORT_THREADS * most < atoms || blocks * SORT_THREADS * SORT_CELLS < cells))
        blocks *= 2;
    const int per = grid_for(atoms, blocks * SORT_THREADS);
    auto kernel = reps ? (per <= 1 ? k_sort_small<1, true> : per <= 2 ? k_sort_small<2, true> : k_sort_small<4, true>)
                       : (per <= 1 ? k_sort_small<1, false> : per <= 2 ? k_sort_small<2, false> : k_sort_small<4, false>);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks * (reps ? c->nrep : 1));
    cfg.blockDim = dim3(SORT_THREADS);
    cfg.stream = c->stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    c->launches++;
    return check_cuda(c, cudaLaunchKernelEx(&cfg, kernel, a), "small sort");
}

size_t nlist_slots(const Context* c, int maxnb) {
    size_t H = (size_t)1 << c->nbr_hshift;
    size_t slices = ((size_t)c->cap + H - 1) / H;
    return slices * H * (size_t)maxnb;
}

int nlist_reserve(Context* c, int maxnb) {
    size_t need = nlist_slots(c, maxnb) * sizeof(unsigned);
    if (maxnb <= c->maxnb && c->nbr) return OMDG_OK;
    cudaFree(c->nbr);
    cudaFree(c->rev);
    cudaFree(c->slot_buf);
    cudaFree(c->row_hits);
    c->nbr = nullptr;
    c->rev = nullptr;
    c->slot_buf = nullptr;
    c->row_hits = nullptr;
    if (cudaMalloc(&c->nbr, need) != cudaSuccess) return set_error(c, OMDG_ENOMEM, "neighbour list allocation");
    if (c->need_rev) {
        if (cudaMalloc(&c->rev, need) != cudaSuccess) return set_error(c, OMDG_ENOMEM, "reverse slot allocation");
        // a row that overflows can leave an entry without its reverse: it stays a valid slot
        cudaMemsetAsync(c->rev, 0, need, c->stream);
        if (cudaMalloc(&c->slot_buf, nlist_slots(c, maxnb) * sizeof(float4)) != cudaSuccess)
            return set_error(c, OMDG_ENOMEM, "slot buffer allocation");
        if (cudaMalloc(&c->row_hits, sizeof(unsigned) * (size_t)((maxnb + 31) / 32) * c->cap) != cudaSuccess)
            return set_error(c, OMDG_ENOMEM, "row hits allocation");
    }
    c->maxnb = maxnb;
    c->nbr_bytes = (long)need;
    return tile_reserve_slots(c);
}

static int ensure_cells(Context* c, int m) {
    if (m + 1 <= c->ncell_cap) return OMDG_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(c->stream, &cs);
    if (cs != cudaStreamCaptureStatusNone) return set_error(c, OMDG_ESTATE, "cell grid grew inside a captured step");
    invalidate_graph(c);  // a captured step holds the old cell arrays
    cudaFree(c->cell_count);
    cudaFree(c->cell_start);
    cudaFree(c->cell_fill);
    cudaFree(c->cell_tile_sum);
    int cap = m + 1;
    if (cudaMalloc(&c->cell_count, cap * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&c->cell_start, (cap + 1) * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&c->cell_fill, cap * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&c->cell_tile_sum, (cap / SCAN_TILE + 2) * sizeof(int)) != cudaSuccess)
        return set_error(c, OMDG_ENOMEM, "cell arrays");
    c->ncell_cap = cap;
    return OMDG_OK;
}

int integrate_pack(Context* c) {
    if (c->n == 0) return OMDG_OK;
    // xref keeps the positions of the last build (the displacement reference)
    k_pack<<<grid_for(c->n, 256), 256, 0, c->stream>>>(c->n, c->x, c->y, c->z, c->type, pack_frame(c), c->pack);
    c->launches++;
    return check_cuda(c, cudaGetLastError(), "pack");
}

// on_request: the kernels look for the step's request themselves (small_sort
// boxes, inside a captured step).
int nlist_build(Context* c, bool on_request) {
    int n = c->n;
    if (n == 0) return OMDG_OK;
    CellGeom g = cell_geom(c);
    const bool reps = c->nrep > 0;
    int m = reps ? c->rep_cells : cells_of(c);
    int rc = ensure_cells(c, m);
    if (rc) return rc;
    cudaStream_t s = c->stream;
    unsigned* umax = reinterpret_cast<unsigned*>(c->d_flags + 3);
    const RepGeom* rg = reps ? static_cast<const RepGeom*>(c->d_rep_geom) : nullptr;
    int* cell_sorted = c->cell_sorted;
    // a partial build (replica mode, inside a step): only the replicas whose
    // atoms moved past skin/2 are re-sorted and re-listed; every replica keeps
    // its index range and cell range, so the others' arrays stay valid
    const int* rflag = (reps && c->build_partial) ? c->d_rep_flag : nullptr;
    prof_begin(c, "cell_sort");
    // a replica's cluster cannot see the others': the snapshot of all atoms is
    // taken before
    const bool small_reps = reps && sort_fits(c->rep_max_atoms, c->rep_max_cells);
    const bool small_one = small_sort(c);
    int* list_n = c->d_flags + 5;
    if (!small_one && c->build_in_step && c->snap_d) {
        AtomArrays cur0{c->x, c->y, c->z, c->vx, c->vy, c->vz, c->type, c->id, c->aflag, nullptr, 0};
        AtomArrays snap{c->snap_d, c->snap_d + c->cap, c->snap_d + 2 * (size_t)c->cap, c->snap_d + 3 * (size_t)c->cap,
                        c->snap_d + 4 * (size_t)c->cap, c->snap_d + 5 * (size_t)c->cap, c->snap_i,
                        c->snap_i + c->cap, reinterpret_cast<unsigned*>(c->snap_i + 2 * (size_t)c->cap), nullptr, 0};
        const int sb = (int)step_state_bytes();
        int* taken = c->d_flags + 6;
        k_snapshot<<<grid_for(std::max(n, sb), 256), 256, 0, s>>>(
            n, step_state_halted(c), taken, cur0, snap, static_cast<const unsigned char*>(c->d_state),
            static_cast<unsigned char*>(c->snap_state), sb, c->d_status, taken + 1);
        k_set_one<<<1, 1, 0, s>>>(taken);
        c->launches += 2;
    }
    if (small_one || small_reps) {
        if (small_reps) {
            k_zero_ints<<<1, 32, 0, s>>>(1, c->d_flags + 3, list_n);
            c->launches++;
        }
        if ((rc = launch_sort_small(c, g, m, on_request, umax, rflag, list_n))) return rc;
        prof_end(c);
    } else {
        if (rflag)
            k_zero_cells_rep<<<grid_for(m + 1, 256), 256, 0, s>>>(m, c->cell_count, c->cell_fill, c->d_cell_rep, rflag);
        else
            k_zero_ints<<<grid_for(m + 1, 256), 256, 0, s>>>(m + 1, c->cell_count, c->cell_fill);
        if (reps)
            k_cell_assign_rep<<<grid_for(n, 256), 256, 0, s>>>(n, c->x, c->y, c->z, c->d_rep_of,
                                                                 static_cast<const RepGeom*>(c->d_rep_geom), c->cell,
                                                                 c->cell_count, c->d_status, rflag);
        else
            k_cell_assign<<<grid_for(n, 256), 256, 0, s>>>(n, c->x, c->y, c->z, g, c->cell, c->cell_count,
                                                             c->d_status);
        const int ntiles = (m + SCAN_TILE - 1) / SCAN_TILE;
        k_scan_tiles<<<ntiles, SCAN_THREADS, 0, s>>>(m, c->cell_count, c->cell_start, c->cell_tile_sum);
        k_scan_totals<<<1, 1024, 0, s>>>(ntiles, m, c->cell_tile_sum, c->cell_start, umax);
        k_scan_add<<<grid_for(m, 256), 256, 0, s>>>(m, c->cell_start, c->cell_tile_sum);
        k_scatter<<<grid_for(n, 256), 256, 0, s>>>(n, c->cell, c->cell_start, c->cell_fill, c->perm, c->d_rep_of, rflag);
        // most cells of a sparse grid (replica margins, vacuum) hold 0 or 1 atoms:
        // a bounded grid of warps strides over the cells instead of one warp each
        // sparse grids (a few atoms per cell) sort most cells a thread each;
        // dense ones (EAM: ~20 atoms per cell) leave every cell to the warps
        const bool sparse = n < 8 * m;
        int* big = nullptr;  // the queue of cells for the warps: the cell_fill array, free again after the scatter
        if (sparse) {
            big = c->cell_fill;
            k_zero_ints<<<1, 32, 0, s>>>(1, big, big);
            k_cell_sort_small<<<grid_for(m, 256), 256, 0, s>>>(m, c->cell_start, c->perm, c->d_cell_rep, rflag, big);
            c->launches += 2;
        }
        k_cell_sort_warp<<<std::min(grid_for(m, 8), 16 * c->num_sms), 256, 0, s>>>(
            m, c->cell_start, c->perm, sparse ? CELL_SORT_SMALL : 1, c->d_cell_rep, rflag, big);
        c->launches += 7;
        AtomArrays cur{c->x, c->y, c->z, c->vx, c->vy, c->vz, c->type, c->id, c->aflag, c->extra, c->extra_n};
        AtomArrays stg{c->stage_d, c->stage_d + c->cap, c->stage_d + 2 * (size_t)c->cap, c->stage_d + 3 * (size_t)c->cap,
                       c->stage_d + 4 * (size_t)c->cap, c->stage_d + 5 * (size_t)c->cap, c->stage_i,
                       c->stage_i + c->cap, reinterpret_cast<unsigned*>(c->stage_i + 2 * (size_t)c->cap),
                       c->stage_extra, c->extra_n};
        k_permute_gather<<<grid_for(n, 256), 256, 0, s>>>(n, c->perm, cur, stg, c->cell, cell_sorted, c->inv,
                                                          c->d_rep_of, rflag, pack_frame(c),
                                                          Corner{g.lo[0], g.lo[1], g.lo[2]}, rg, c->flags_used ? c->aflag : nullptr, c->pack, c->xref, c->loc,
                                                          umax);
        k_permute_copyback<<<grid_for(n, 256), 256, 0, s>>>(n, stg, cur, c->d_rep_of, rflag);
        c->launches += 2;
        prof_end(c);
    }

    BuildParams bp;
    bp.to = TileOut{};
    // tile slots: prepared per tile after the scan, written by the list build
    const bool tiles = c->tile_want && !reps && c->tslot && c->tile_stride >= c->maxnb;
    if (tiles) {
        TilePrep tp;
        for (int d = 0; d < 3; d++) {
            tp.T[d] = c->tile_dim[d];
            tp.nt[d] = c->tile_nt[d];
            tp.nc[d] = g.nc[d];
            tp.periodic[d] = g.periodic[d];
            tp.corg[d] = g.org[d];
            tp.h[d] = g.h[d];
            tp.borg[d] = c->box.org[d];
            tp.P[d] = c->box.P[d];
        }
        tp.hx = tp.T[0] + 2;
        tp.hy = tp.T[1] + 2;
        tp.HC = c->tile_hc;
        k_tile_prep<<<c->tile_count, TILE_PREP_THREADS, 0, s>>>(tp, c->cell_start, c->tile_sb, c->tile_nst,
                                                                c->tile_org);
        c->launches++;
        bp.to.slot = c->tslot;
        bp.to.sb = c->tile_sb;
        bp.to.nst = c->tile_nst;
        for (int d = 0; d < 3; d++) {
            bp.to.T[d] = tp.T[d];
            bp.to.nt[d] = tp.nt[d];
        }
        bp.to.hx = tp.hx;
        bp.to.hy = tp.hy;
        bp.to.HC = tp.HC;
        bp.to.stride = c->tile_stride;
        bp.to.cap = c->tile_cap;
    }
    c->tile_valid = tiles;
    bp.on = on_request ? step_state_building(c) : nullptr;
    bp.list = small_reps && rflag ? c->cell : nullptr;
    bp.list_n = list_n;
    bp.n = n;
    bp.maxnb = c->maxnb;
    bp.hshift = c->nbr_hshift;
    for (int d = 0; d < 3; d++) {
        bp.nc[d] = g.nc[d];
        bp.periodic[d] = g.periodic[d];
        bp.L64[d] = g.L[d];
    }
    bp.L = make_shift(c->box);
    double rv = c->rc_max + c->skin;
    bp.rsq = rv * rv;
    bp.rv = (float)rv;
    prof_begin(c, "nlist_build");
    bp.lmax = 0.f;
    for (int d = 0; d < 3; d++)
        if (g.periodic[d]) bp.lmax = fmaxf(bp.lmax, (float)g.L[d]);
    if (reps) bp.lmax = (float)c->rep_lmax;
    double far = 0.0;  // the corner farthest from the origin
    for (int d = 0; d < 3; d++) far = std::max(far, std::fabs(g.lo[d]));
    if (reps)
        for (double q : c->rep_lo) far = std::max(far, std::fabs(q));
    bp.corner_err = (float)(far * 0x1p-51);
    // shared-memory columns: maxnb is twice the mean row and 32 at first, so
    // half of it and 8 holds nearly every row; 64 entries (32 KB a block)
    // keep seven blocks on a SM.  Longer rows go out in pieces.
    bp.cap = std::max(2 * BUILD_AHEAD, std::min(64, c->maxnb / 2 + 8));
    const bool one = c->ntypes == 1;
    // eight lanes a centre while a thread per centre would leave most of the
    // chip's warp slots empty (BUILD_SMALL_PER_SM)
    const bool small = c->build_lanes == 8 || (c->build_lanes != 1 && n <= BUILD_SMALL_PER_SM * c->num_sms);
    const int lanes = small && !tiles ? 8 : 1;  // only the one-thread form writes tile slots
    const size_t smem = sizeof(unsigned) * BUILD_THREADS * (lanes == 1 ? bp.cap : BUILD_RUN);
    const auto launch = [&](auto kernel) {
        const int all = grid_for(n, BUILD_THREADS / lanes);
        kernel<<<bp.list ? std::min(all, BUILD_CTAS_PER_SM * c->num_sms) : all, BUILD_THREADS, smem, s>>>(
            bp, rg, c->d_rep_of, c->loc, c->x, c->y, c->z, cell_sorted, c->cell_start, umax,
            reinterpret_cast<unsigned*>(c->nbr), c->nnb, c->d_status, c->d_flags + 1, rflag, c->nbmask);
    };
    if (lanes == 8) {
        if (reps) one ? launch(k_build<8, true, false, true>) : launch(k_build<8, true, false, false>);
        else one ? launch(k_build<8, false, false, true>) : launch(k_build<8, false, false, false>);
    } else {
        if (reps) one ? launch(k_build<1, true, false, true>) : launch(k_build<1, true, false, false>);
        else if (tiles) launch(k_build<1, false, true, true>);  // the tiled passes take one type
        else one ? launch(k_build<1, false, false, true>) : launch(k_build<1, false, false, false>);
    }
    c->launches++;
    if (c->build_in_step && !on_request) {  // (k_sort_small looks for itself)
        k_halt_on_overflow<<<1, 1, 0, s>>>(c->d_status, step_state_halted(c));
        c->launches++;
    }

    prof_end(c);
    if (c->need_rev) {
        prof_begin(c, "nlist_reverse");
        const int all = grid_for(n, 128 / REV_LANES);
        k_reverse<<<bp.list ? std::min(all, 16 * c->num_sms) : all, 128, 0, s>>>(n, c->nbr_hshift, c->maxnb,
                                                   reinterpret_cast<const unsigned*>(c->nbr), c->nnb, c->rev,
                                                   c->d_status, c->d_rep_of, rflag, bp.on, bp.list, bp.list_n);
        c->launches++;
        prof_end(c);
    }
    if (reps) {
        k_rep_build_done<<<grid_for(c->nrep, 256), 256, 0, s>>>(c->nrep, rflag ? 0 : 1, c->d_rep_flag,
                                                                 c->d_rep_builds);
        c->launches++;
    }
    c->rebuilds++;
    c->list_valid = true;
    c->steps_since_build = 0;
    return check_cuda(c, cudaGetLastError(), "neighbour build");
}

}  // namespace omdg
