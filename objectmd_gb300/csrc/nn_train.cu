// Training of the neural surrogate on the GPU (no reference counterpart).
//
// A dataset is a set of periodic configurations (positions, box lengths,
// reference total energies and forces).  Its descriptors G and their
// Jacobian J (dG_i/dx_j for every neighbour j inside the cutoff; dG_i/dx_i is
// minus their sum) are computed once.  One training step over a batch of
// configurations:
//   1. k_nn_fwd        E_i and u_i = dE_i/dG_i (FP32, per atom)
//   2. k_nn_conf_energy  per configuration: dE = (sum E_i - E_ref) / N
//   3. k_nn_force      F_k = sum_s (J_ks^T u_k - J_(j,rev)^T u_j), force residual
//   4. k_nn_vvec       v_i = dL/du_i = sum_s J_is (rho_i - rho_j)
//   5. k_nn_grad       per chunk of atoms the energy and force gradients (the
//                      force term differentiates u_i . v_i through the network:
//                      forward-mode tangent, then reverse mode) and their
//                      outer-product sums, fixed order (deterministic)
//   6. k_nn_step       sums of the chunks and the loss, Adam update of the
//                      FP32 parameters
// Loss: L = wE mean_c (dE_c)^2 + wF mean_(k,a) (F_ka - F_ka^ref)^2.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "device_common.cuh"
#include "nn_desc.cuh"
#include "tc_common.cuh"

struct omdg_nn {
    int device = 0;
    int num_sms = 152;
    cudaStream_t stream = nullptr;
    std::string err;
    omdg::NNModel model;
    bool have_weights = false;
    // dataset (host bookkeeping)
    int nconf = 0;
    long natoms = 0, nslots = 0;
    std::vector<int> conf_start;  // nconf + 1
    // dataset (device)
    int* d_conf_start = nullptr;
    int* d_atom_conf = nullptr;
    double* d_x = nullptr;
    double* d_L = nullptr;
    float* d_eref = nullptr;
    float* d_fref = nullptr;
    float* d_fw = nullptr;      // per-configuration force-loss weight
    float* d_eatom = nullptr;   // per-atom reference energies (per-atom energy loss) or null
    float* d_ewa = nullptr;     // per atom dL/dE_i in the per-atom mode
    std::vector<float> fms;     // per-configuration mean square reference force
    int* d_slot_start = nullptr;
    int* d_slot_j = nullptr;
    int* d_slot_rev = nullptr;
    float4* d_slot_d = nullptr;
    float* d_G = nullptr;   // raw descriptors
    float* d_Gt = nullptr;  // normalised
    float* d_J = nullptr;   // nslots x 3 x 32
    // training state
    float* d_params = nullptr;
    float* d_adam_m = nullptr;
    float* d_adam_v = nullptr;
    float* d_grad = nullptr;
    float* d_E = nullptr;
    float* d_u = nullptr;
    float* d_F = nullptr;
    float* d_rho = nullptr;
    float* d_vvec = nullptr;
    float* d_ew = nullptr;       // per configuration dL/dE_i
    float* d_lossE = nullptr;    // per batch configuration
    float* d_lossF = nullptr;    // per batch atom
    float* d_acts = nullptr;     // per batch chunk: the forward pass's activations (NT_ACTS x 32 atoms)
    float* d_partial = nullptr;  // per chunk x NN_PARAMS
    double* d_loss = nullptr;    // per batch of the queued epochs
    long cap_loss = 0;
    int* d_list = nullptr;       // atom order of the epoch
    int* d_clist = nullptr;      // configuration order of the queued epochs, then where each one's atoms begin
    long cap_clist = 0;
    unsigned* d_status = nullptr;
    long cap_batch_atoms = 0;
    long adam_t = 0;
    omdg::NNDevNet net;
};

namespace omdg {

constexpr int NN_CHUNK = 32;  // atoms per block and gradient partial

// ------------------------------------------------------------------ dataset kernels
__device__ __forceinline__ double nn_min_image(double d, double L) { return d - L * rint(d / L); }

__global__ void k_nn_count(long n, const int* __restrict__ atom_conf, const int* __restrict__ conf_start,
                           const double* __restrict__ x, const double* __restrict__ L, double rc2,
                           int* __restrict__ count) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = atom_conf[i];
    const double lx = L[3 * c], ly = L[3 * c + 1], lz = L[3 * c + 2];
    int k = 0;
    for (int j = conf_start[c]; j < conf_start[c + 1]; j++) {
        if (j == i) continue;
        const double dx = nn_min_image(x[3 * j] - x[3 * i], lx);
        const double dy = nn_min_image(x[3 * j + 1] - x[3 * i + 1], ly);
        const double dz = nn_min_image(x[3 * j + 2] - x[3 * i + 2], lz);
        if (dx * dx + dy * dy + dz * dz < rc2) k++;
    }
    count[i] = k;
}

__global__ void k_nn_fill(long n, const int* __restrict__ atom_conf, const int* __restrict__ conf_start,
                          const double* __restrict__ x, const double* __restrict__ L, double rc2,
                          const int* __restrict__ slot_start, int* __restrict__ slot_j, float4* __restrict__ slot_d) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = atom_conf[i];
    const double lx = L[3 * c], ly = L[3 * c + 1], lz = L[3 * c + 2];
    int s = slot_start[i];
    for (int j = conf_start[c]; j < conf_start[c + 1]; j++) {
        if (j == i) continue;
        const double dx = nn_min_image(x[3 * j] - x[3 * i], lx);
        const double dy = nn_min_image(x[3 * j + 1] - x[3 * i + 1], ly);
        const double dz = nn_min_image(x[3 * j + 2] - x[3 * i + 2], lz);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < rc2) {
            slot_j[s] = j;
            slot_d[s] = make_float4((float)dx, (float)dy, (float)dz, (float)sqrt(r2));
            s++;
        }
    }
}

__global__ void k_nn_rev(long n, const int* __restrict__ slot_start, const int* __restrict__ slot_j,
                         int* __restrict__ rev, unsigned* status) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int s = slot_start[i]; s < slot_start[i + 1]; s++) {
        const int j = slot_j[s];
        int found = -1;
        for (int q = slot_start[j]; q < slot_start[j + 1]; q++)
            if (slot_j[q] == (int)i) found = q;
        if (found < 0) atomicOr(status, ERR_NBR_OVERFLOW);
        rev[s] = found < 0 ? s : found;
    }
}

// G and J of one atom from its neighbour slots (d = x_j - x_i, w = r).
__global__ void k_nn_train_desc(NNDescParams p, long n, const int* __restrict__ slot_start,
                                const float4* __restrict__ slot_d, float* __restrict__ G, float* __restrict__ J) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float g[NN_DESC];
#pragma unroll
    for (int k = 0; k < NN_DESC; k++) g[k] = 0.f;
    const int s0 = slot_start[i], s1 = slot_start[i + 1];
    for (int s = s0; s < s1; s++) {
        const float4 d = slot_d[s];
        const float r = d.w, ir = 1.f / r;
        const float e[3] = {d.x * ir, d.y * ir, d.z * ir};
        float dfc;
        const float fc = nn_fc(p, r, dfc);
        float* Js = J + (size_t)s * 3 * NN_DESC;
        for (int k = 0; k < NN_RAD; k++) {
            float v, ddr;
            nn_radial(p, r, fc, dfc, k, v, ddr);
            g[k] += v;
            for (int c = 0; c < 3; c++) Js[c * NN_DESC + k] = ddr * e[c];
        }
        for (int c = 0; c < 3; c++)
            for (int m = 0; m < NN_ANG; m++) Js[c * NN_DESC + NN_RAD + m] = 0.f;
    }
    for (int a = s0; a < s1; a++) {
        const float4 da = slot_d[a];
        const float ra = da.w, ia = 1.f / ra;
        const float ea[3] = {da.x * ia, da.y * ia, da.z * ia};
        float dfa;
        const float fa = nn_fc(p, ra, dfa);
        float* Ja = J + (size_t)a * 3 * NN_DESC + NN_RAD;
        for (int b = a + 1; b < s1; b++) {
            const float4 db = slot_d[b];
            const float rb = db.w, ib = 1.f / rb;
            const float eb[3] = {db.x * ib, db.y * ib, db.z * ib};
            float dfb;
            const float fb = nn_fc(p, rb, dfb);
            const float cs = ea[0] * eb[0] + ea[1] * eb[1] + ea[2] * eb[2];
            float dca[3], dcb[3];
            for (int c = 0; c < 3; c++) {
                dca[c] = (eb[c] - cs * ea[c]) * ia;
                dcb[c] = (ea[c] - cs * eb[c]) * ib;
            }
            float* Jb = J + (size_t)b * 3 * NN_DESC + NN_RAD;
            const float s2 = ra * ra + rb * rb;
            NNAngExp ex;
            for (int m = 0; m < NN_ANG; m++) {
                float v, d_ra, d_rb, d_cs;
                nn_angular(p, m, ra, rb, cs, fa, dfa, fb, dfb, ex.get(p.eta_a[m], s2), v, d_ra, d_rb, d_cs);
                g[NN_RAD + m] += v;
                for (int c = 0; c < 3; c++) {
                    Ja[c * NN_DESC + m] += d_ra * ea[c] + d_cs * dca[c];
                    Jb[c * NN_DESC + m] += d_rb * eb[c] + d_cs * dcb[c];
                }
            }
        }
    }
    for (int k = 0; k < NN_DESC; k++) G[i * NN_DESC + k] = g[k];
}

__global__ void k_nn_normalize(NNDescParams p, long n, const float* __restrict__ G, float* __restrict__ Gt) {
    const long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= n * NN_DESC) return;
    const int d = (int)(q % NN_DESC);
    Gt[q] = (G[q] - p.mu[d]) * p.isig[d];
}

// ------------------------------------------------------------------ training kernels
// A block takes NN_CHUNK = 32 atoms.  Weights and the atoms' vectors sit in
// shared memory, a vector as one row of 32 atoms per feature (stride 36), and
// the layers are register-tiled products: a thread holds four atoms by two
// of 64 features.  Every output
// sums its terms in the order of the feature index, in FP32.  Bound by the
// shared loads' latency and wavefronts at two blocks a SM (LSU 50 %).  For a
// batch of 16 x 512 atoms a step's kernels take 17 (forward), 7 (forces), 6
// (dL/du), 25 (gradient) and 12 us (sums and Adam) under ncu (warm caches), a step 82 us in
// the loop; one thread per atom, as it was, ran 64 blocks of 128 threads with
// 64-wide vectors in local memory and took 348 us a step.
constexpr int NT_THREADS = 256;
constexpr int NT_TO = NT_THREADS / 8;   // threads along the features; eight along the atoms (four each)
constexpr int NT_R = NN_H / NT_TO;      // features of 64 a thread
constexpr int NT_AS = NN_CHUNK + 4;     // stride of a feature row
constexpr int NT_W1S = NN_DESC + 4;     // stride of a row of W1 (64 x 32)
constexpr int NT_W2S = NN_H + 4;        // stride of a row of W2 (64 x 64)
constexpr int NT_ACTS = 3 * NN_H;       // features kept from the forward pass: a1, a2, W2^T d2
constexpr int NT_VEC = 4 * NN_H;        // b1, b2, w3, b3
constexpr int NT_W_FLOATS = NN_H * NT_W1S + NN_H * NT_W2S + NT_VEC;
constexpr int NT_FWD_FLOATS = NT_W_FLOATS + (NN_DESC + 3 * NN_H) * NT_AS;
constexpr int NT_GRAD_FLOATS = NT_W_FLOATS + (2 * NN_DESC + 7 * NN_H) * NT_AS + NN_CHUNK;

struct NTWeights {
    float *W1, *W2, *b1, *b2, *w3, *b3;
};

__device__ __forceinline__ NTWeights nt_load_weights(const float* __restrict__ w, float* s) {
    NTWeights q;
    q.W1 = s;
    q.W2 = q.W1 + NN_H * NT_W1S;
    q.b1 = q.W2 + NN_H * NT_W2S;
    q.b2 = q.b1 + NN_H;
    q.w3 = q.b2 + NN_H;
    q.b3 = q.w3 + NN_H;
    const float4* w1 = reinterpret_cast<const float4*>(w + NN_OFF_W1);
    const float4* w2 = reinterpret_cast<const float4*>(w + NN_OFF_W2);
#pragma unroll
    for (int c = 0; c < NN_H * NN_DESC / 4 / NT_THREADS; c++) {
        const int k = c * NT_THREADS + threadIdx.x;
        *reinterpret_cast<float4*>(q.W1 + (k / (NN_DESC / 4)) * NT_W1S + 4 * (k % (NN_DESC / 4))) = __ldg(w1 + k);
    }
#pragma unroll
    for (int c = 0; c < NN_H * NN_H / 4 / NT_THREADS; c++) {
        const int k = c * NT_THREADS + threadIdx.x;
        *reinterpret_cast<float4*>(q.W2 + (k / (NN_H / 4)) * NT_W2S + 4 * (k % (NN_H / 4))) = __ldg(w2 + k);
    }
    for (int k = threadIdx.x; k < NN_H; k += NT_THREADS) {
        q.b1[k] = __ldg(w + NN_OFF_B1 + k);
        q.b2[k] = __ldg(w + NN_OFF_B2 + k);
        q.w3[k] = __ldg(w + NN_OFF_W3 + k);
    }
    if (threadIdx.x == 0) q.b3[0] = __ldg(w + NN_OFF_B3);
    return q;
}

// acc[o][a] += sum_k W[row o][k] X[k][a], rows to + NT_TO o, atoms 4 ta + a
template <int K, int WS>
__device__ __forceinline__ void nt_rows(const float* W, const float* X, int to, int ta, float (&acc)[NT_R][4]) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 w[NT_R];
#pragma unroll
        for (int o = 0; o < NT_R; o++) w[o] = *reinterpret_cast<const float4*>(W + (to + NT_TO * o) * WS + k);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 x = *reinterpret_cast<const float4*>(X + (k + q) * NT_AS + 4 * ta);
#pragma unroll
            for (int o = 0; o < NT_R; o++) {
                const float v = q == 0 ? w[o].x : (q == 1 ? w[o].y : (q == 2 ? w[o].z : w[o].w));
                acc[o][0] = fmaf(v, x.x, acc[o][0]);
                acc[o][1] = fmaf(v, x.y, acc[o][1]);
                acc[o][2] = fmaf(v, x.z, acc[o][2]);
                acc[o][3] = fmaf(v, x.w, acc[o][3]);
            }
        }
    }
}

// acc[c][a] += sum_k X[k][a] W[k][NC to + c]
template <int NC, int WS>
__device__ __forceinline__ void nt_cols(const float* W, const float* X, int to, int ta, float (&acc)[NC][4]) {
#pragma unroll 4
    for (int k = 0; k < NN_H; k++) {
        const float4 x = *reinterpret_cast<const float4*>(X + k * NT_AS + 4 * ta);
        float v[NC];
        if (NC == 2) {
            const float2 w = *reinterpret_cast<const float2*>(W + k * WS + 2 * to);
            v[0] = w.x, v[NC - 1] = w.y;
        } else {
            v[0] = W[k * WS + to];
        }
#pragma unroll
        for (int c = 0; c < NC; c++) {
            acc[c][0] = fmaf(v[c], x.x, acc[c][0]);
            acc[c][1] = fmaf(v[c], x.y, acc[c][1]);
            acc[c][2] = fmaf(v[c], x.z, acc[c][2]);
            acc[c][3] = fmaf(v[c], x.w, acc[c][3]);
        }
    }
}

template <int N>
__device__ __forceinline__ void nt_zero(float (&acc)[N][4]) {
#pragma unroll
    for (int o = 0; o < N; o++) acc[o][0] = acc[o][1] = acc[o][2] = acc[o][3] = 0.f;
}

__device__ __forceinline__ float4& nt_at(float* X, int row, int ta) {
    return *reinterpret_cast<float4*>(X + row * NT_AS + 4 * ta);
}

// 32-wide rows of the chunk's atoms into feature rows; absent atoms give zeros
template <bool SCALE>
__device__ __forceinline__ void nt_load_rows(const float* __restrict__ src, const float* scale,
                                             const int* __restrict__ list, int cnt, float* X) {
    const int d = threadIdx.x & 31;
    for (int a = threadIdx.x >> 5; a < NN_CHUNK; a += NT_THREADS / 32) {
        float v = a < cnt ? src[(size_t)__ldg(list + a) * NN_DESC + d] : 0.f;
        if (SCALE) v *= scale[d];
        X[d * NT_AS + a] = v;
    }
}

// E_i and u_i (raw descriptor units) for the atoms list[a0 .. a0 + na); with
// acts, the activations the gradient needs; with eatom, the per-atom energy
// residuals (dL/dE_i) and their loss terms.
__global__ void __launch_bounds__(NT_THREADS) k_nn_fwd(const float* __restrict__ w, const float* __restrict__ Gt,
                                                       NNDescParams p, const int* __restrict__ list, int a0, int na,
                                                       float* __restrict__ E, float* __restrict__ U,
                                                       float* __restrict__ acts, const float* __restrict__ eatom,
                                                       float wE, float* __restrict__ ewa,
                                                       float* __restrict__ lossE) {
    extern __shared__ __align__(16) float sm[];
    const NTWeights q = nt_load_weights(w, sm);
    float* G = sm + NT_W_FLOATS;
    float* A1 = G + NN_DESC * NT_AS;
    float* D2 = A1 + NN_H * NT_AS;
    float* A2 = D2 + NN_H * NT_AS;
    const int t0 = blockIdx.x * NN_CHUNK, cnt = min(NN_CHUNK, na - t0);
    list += a0 + t0;
    nt_load_rows<false>(Gt, nullptr, list, cnt, G);
    __syncthreads();
    const int ta = threadIdx.x & 7, to = threadIdx.x >> 3;
    float* act = acts ? acts + (size_t)blockIdx.x * NT_ACTS * NN_CHUNK + 4 * ta : nullptr;
    float z[NT_R][4];
#pragma unroll
    for (int o = 0; o < NT_R; o++) z[o][0] = z[o][1] = z[o][2] = z[o][3] = q.b1[to + NT_TO * o];
    nt_rows<NN_DESC, NT_W1S>(q.W1, G, to, ta, z);
#pragma unroll
    for (int o = 0; o < NT_R; o++) {
        const float4 v = make_float4(tanhf(z[o][0]), tanhf(z[o][1]), tanhf(z[o][2]), tanhf(z[o][3]));
        nt_at(A1, to + NT_TO * o, ta) = v;
        if (act) *reinterpret_cast<float4*>(act + (to + NT_TO * o) * NN_CHUNK) = v;
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < NT_R; o++) z[o][0] = z[o][1] = z[o][2] = z[o][3] = q.b2[to + NT_TO * o];
    nt_rows<NN_H, NT_W2S>(q.W2, A1, to, ta, z);
#pragma unroll
    for (int o = 0; o < NT_R; o++) {
        const float4 v = make_float4(tanhf(z[o][0]), tanhf(z[o][1]), tanhf(z[o][2]), tanhf(z[o][3]));
        const float w3 = q.w3[to + NT_TO * o];
        nt_at(A2, to + NT_TO * o, ta) = v;
        nt_at(D2, to + NT_TO * o, ta) = make_float4(w3 * (1.f - v.x * v.x), w3 * (1.f - v.y * v.y),
                                                 w3 * (1.f - v.z * v.z), w3 * (1.f - v.w * v.w));
        if (act) *reinterpret_cast<float4*>(act + (NN_H + to + NT_TO * o) * NN_CHUNK) = v;
    }
    __syncthreads();
    if (threadIdx.x < cnt) {
        float e = q.b3[0];
#pragma unroll 8
        for (int o = 0; o < NN_H; o++) e = fmaf(q.w3[o], A2[o * NT_AS + threadIdx.x], e);
        const int atom = list[threadIdx.x];
        E[atom] = e;
        if (eatom) {
            const float r = e - eatom[atom];
            ewa[atom] = 2.f * wE * r / na;
            lossE[t0 + threadIdx.x] = wE * r * r / na;
        }
    }
    nt_zero(z);
    nt_cols<NT_R, NT_W2S>(q.W2, D2, to, ta, z);
    __syncthreads();  // D2 is done: it takes d1
#pragma unroll
    for (int c = 0; c < NT_R; c++) {
        const int j = NT_R * to + c;
        const float4 a1 = nt_at(A1, j, ta);
        if (act)
            *reinterpret_cast<float4*>(act + (2 * NN_H + j) * NN_CHUNK) = make_float4(z[c][0], z[c][1], z[c][2], z[c][3]);
        nt_at(D2, j, ta) = make_float4(z[c][0] * (1.f - a1.x * a1.x), z[c][1] * (1.f - a1.y * a1.y),
                                       z[c][2] * (1.f - a1.z * a1.z), z[c][3] * (1.f - a1.w * a1.w));
    }
    __syncthreads();
    float u[NT_R / 2][4];
    nt_zero(u);
    nt_cols<NT_R / 2, NT_W1S>(q.W1, D2, to, ta, u);
#pragma unroll
    for (int a = 0; a < 4; a++)
        if (4 * ta + a < cnt)
#pragma unroll
            for (int c = 0; c < NT_R / 2; c++) {
                const int d = NT_R / 2 * to + c;
                U[(size_t)list[4 * ta + a] * NN_DESC + d] = u[c][a] * p.isig[d];
            }
}

// One block per batch configuration: energy residual and its loss term.
__global__ void k_nn_conf_energy(const int* __restrict__ clist, int c0, int nb, const int* __restrict__ conf_start,
                                 const float* __restrict__ E, const float* __restrict__ eref, float wE,
                                 float* __restrict__ ew, float* __restrict__ lossE) {
    __shared__ double red[256];
    const int conf = clist[c0 + blockIdx.x];
    const int a = conf_start[conf], b = conf_start[conf + 1];
    double s = 0.0;
    for (int i = a + threadIdx.x; i < b; i += blockDim.x) s += (double)E[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const int n = b - a;
        const double de = (red[0] - (double)eref[conf]) / n;
        ew[conf] = (float)(2.0 * wE * de / ((double)n * nb));
        lossE[blockIdx.x] = (float)(wE * de * de / nb);
    }
}

// Forces from J and u; the force residual, rho = dL/dF and its loss term.
// One warp per atom, a lane per descriptor: the Jacobian's rows (32 floats)
// and u are read as whole lines, and the descriptors sum in an xor tree.
__global__ void __launch_bounds__(256) k_nn_force(const int* __restrict__ list, int a0, int na,
                                                  const int* __restrict__ slot_start, const int* __restrict__ slot_j,
                                                  const int* __restrict__ rev, const float* __restrict__ J,
                                                  const float* __restrict__ U, const float* __restrict__ fref,
                                                  float wF_over_ncomp, const float* __restrict__ fw,
                                                  const int* __restrict__ atom_conf, float* __restrict__ F,
                                                  float* __restrict__ rho, float* __restrict__ lossF) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= na) return;
    const int k = list[a0 + t];
    const int s0 = slot_start[k], s1 = slot_start[k + 1];
    const float uk = U[(size_t)k * NN_DESC + lane];
    float f[3] = {0.f, 0.f, 0.f};
#pragma unroll 2
    for (int s = s0; s < s1; s++) {
        const float* Js = J + (size_t)s * 3 * NN_DESC + lane;
        const float* Jr = J + (size_t)rev[s] * 3 * NN_DESC + lane;
        const float uj = U[(size_t)slot_j[s] * NN_DESC + lane];
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] = fmaf(-Jr[c * NN_DESC], uj, fmaf(Js[c * NN_DESC], uk, f[c]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] += __shfl_xor_sync(0xffffffffu, f[c], o);
    if (lane != 0) return;
    if (fref) wF_over_ncomp *= fw[atom_conf[k]];
    float l = 0.f;
    for (int c = 0; c < 3; c++) {
        F[3 * (size_t)k + c] = f[c];
        if (fref) {
            const float r = f[c] - fref[3 * (size_t)k + c];
            rho[3 * (size_t)k + c] = 2.f * wF_over_ncomp * r;
            l = fmaf(r, r, l);
        }
    }
    if (fref) lossF[t] = wF_over_ncomp * l;
}

// v_i = dL/du_i = sum_s J_is (rho_i - rho_j); a warp per atom, a lane per descriptor
__global__ void __launch_bounds__(256) k_nn_vvec(const int* __restrict__ list, int a0, int na,
                                                 const int* __restrict__ slot_start, const int* __restrict__ slot_j,
                                                 const float* __restrict__ J, const float* __restrict__ rho,
                                                 float* __restrict__ V) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= na) return;
    const int i = list[a0 + t];
    const int s0 = slot_start[i], s1 = slot_start[i + 1];
    float v = 0.f;
    const float ri[3] = {rho[3 * (size_t)i], rho[3 * (size_t)i + 1], rho[3 * (size_t)i + 2]};
#pragma unroll 2
    for (int s = s0; s < s1; s++) {
        const int j = slot_j[s];
        const float* Js = J + (size_t)s * 3 * NN_DESC + lane;
#pragma unroll
        for (int c = 0; c < 3; c++) v = fmaf(Js[c * NN_DESC], ri[c] - rho[3 * (size_t)j + c], v);
    }
    V[(size_t)i * NN_DESC + lane] = v;
}

// sum of a feature over the chunk's atoms: four a thread, then over the eight lanes along the atoms
__device__ __forceinline__ float nt_sum(float4 v) {
    float s = ((v.x + v.y) + v.z) + v.w;
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// out[r][c] = sum over the chunk's atoms of P[r] X[c] + Q[r] Y[c], rows
// to + NT_TO o, columns tc + 8 k, both products of an atom before the next atom's
template <int NCOL, int COLS>
__device__ __forceinline__ void nt_outer(const float* P, const float* X, const float* Q, const float* Y,
                                         float* __restrict__ out) {
    const int tc = threadIdx.x & 7, to = threadIdx.x >> 3;
    float acc[NT_R][NCOL];
#pragma unroll
    for (int o = 0; o < NT_R; o++)
#pragma unroll
        for (int k = 0; k < NCOL; k++) acc[o][k] = 0.f;
#pragma unroll 1
    for (int a = 0; a < NN_CHUNK; a += 4) {
        float4 pr[NT_R], qr[NT_R];
#pragma unroll
        for (int o = 0; o < NT_R; o++) {
            pr[o] = *reinterpret_cast<const float4*>(P + (to + NT_TO * o) * NT_AS + a);
            qr[o] = *reinterpret_cast<const float4*>(Q + (to + NT_TO * o) * NT_AS + a);
        }
#pragma unroll
        for (int k = 0; k < NCOL; k++) {
            const float4 x = *reinterpret_cast<const float4*>(X + (tc + 8 * k) * NT_AS + a);
            const float4 y = *reinterpret_cast<const float4*>(Y + (tc + 8 * k) * NT_AS + a);
#pragma unroll
            for (int o = 0; o < NT_R; o++) {
                float v = acc[o][k];
                v = fmaf(qr[o].x, y.x, fmaf(pr[o].x, x.x, v));
                v = fmaf(qr[o].y, y.y, fmaf(pr[o].y, x.y, v));
                v = fmaf(qr[o].z, y.z, fmaf(pr[o].z, x.z, v));
                acc[o][k] = fmaf(qr[o].w, y.w, fmaf(pr[o].w, x.w, v));
            }
        }
    }
#pragma unroll
    for (int o = 0; o < NT_R; o++)
#pragma unroll
        for (int k = 0; k < NCOL; k++) out[(to + NT_TO * o) * COLS + tc + 8 * k] = acc[o][k];
}

// The loss terms' sum in FP64, by one block.
__device__ __forceinline__ void nt_loss(const float* __restrict__ lossE, int nE, const float* __restrict__ lossF,
                                        int nF, double* red, double* __restrict__ loss) {
    // four sums a thread: the latency of the FP64 adds, not their number, sets this block's time
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k = threadIdx.x; k < nE; k += 4 * NT_THREADS)
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] += k + q * NT_THREADS < nE ? (double)__ldg(lossE + k + q * NT_THREADS) : 0.0;
    for (int k = threadIdx.x; k < nF; k += 4 * NT_THREADS)
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] += k + q * NT_THREADS < nF ? (double)__ldg(lossF + k + q * NT_THREADS) : 0.0;
    red[threadIdx.x] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    for (int off = NT_THREADS / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[0] = red[0];
}

// Partial dL/dw of a chunk of atoms: the energy term (weight e = dL/dE_i) and
// the force term d(u . v)/dw (u = dE/dG, v = dL/du) by a forward tangent
// dz1 = W1 v~ followed by reverse mode through the tangent computation, then
// the outer products over the chunk, all from shared memory.  One block more
// sums the loss meanwhile.
__global__ void __launch_bounds__(NT_THREADS) k_nn_grad(const float* __restrict__ w, const float* __restrict__ Gt,
                                                        const float* __restrict__ V, NNDescParams p,
                                                        const float* __restrict__ acts, const int* __restrict__ list,
                                                        const float* __restrict__ ew,
                                                        const int* __restrict__ ew_index, int a0, int na,
                                                        float* __restrict__ partial, const float* __restrict__ lossE,
                                                        int nE, const float* __restrict__ lossF,
                                                        double* __restrict__ loss) {
    extern __shared__ __align__(16) float sm[];
    if (blockIdx.x * NN_CHUNK >= na) {  // the block past the chunks
        nt_loss(lossE, nE, lossF, na, reinterpret_cast<double*>(sm), loss);
        return;
    }
    const NTWeights q = nt_load_weights(w, sm);
    float* G = sm + NT_W_FLOATS;
    float* VT = G + NN_DESC * NT_AS;
    float* A1 = VT + NN_DESC * NT_AS;
    float* DA1 = A1 + NN_H * NT_AS;
    float* D1 = DA1 + NN_H * NT_AS;
    float* Z1 = D1 + NN_H * NT_AS;   // first the part of r1 that needs dz1
    float* Z2 = Z1 + NN_H * NT_AS;
    float* D2 = Z2 + NN_H * NT_AS;
    float* R2 = D2 + NN_H * NT_AS;
    float* e = R2 + NN_H * NT_AS;    // NN_CHUNK
    const int t0 = blockIdx.x * NN_CHUNK, cnt = min(NN_CHUNK, na - t0);
    list += a0 + t0;
    float* out = partial + (size_t)blockIdx.x * NN_PARAMS;
    nt_load_rows<false>(Gt, nullptr, list, cnt, G);
    nt_load_rows<true>(V, p.isig, list, cnt, VT);
    if (threadIdx.x < NN_CHUNK) {
        const int atom = threadIdx.x < cnt ? list[threadIdx.x] : 0;
        float v = threadIdx.x < cnt ? ew[ew_index ? ew_index[atom] : atom] : 0.f;
        e[threadIdx.x] = v;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) out[NN_OFF_B3] = v;
    }
    __syncthreads();
    const int ta = threadIdx.x & 7, to = threadIdx.x >> 3;
    const float* act = acts + (size_t)blockIdx.x * NT_ACTS * NN_CHUNK + 4 * ta;
    const float4 e4 = *reinterpret_cast<const float4*>(e + 4 * ta);
    // absent atoms of the last chunk: the forward pass gave them a1 = tanh(b1)
    // and so on; their tangents and weights are zero here, and the terms that
    // survive (d1, d2 against zero inputs or tangents) multiply zeros
    float z[NT_R][4];
    nt_zero(z);
    nt_rows<NN_DESC, NT_W1S>(q.W1, VT, to, ta, z);
#pragma unroll
    for (int o = 0; o < NT_R; o++) {
        const int j = to + NT_TO * o;
        const float4 a1 = *reinterpret_cast<const float4*>(act + j * NN_CHUNK);
        const float4 sd = *reinterpret_cast<const float4*>(act + (2 * NN_H + j) * NN_CHUNK);
        float4 da, d1, r;
        const auto one = [](float a, float s, float dz, float& da_, float& d1_, float& r_) {
            const float s1 = 1.f - a * a;
            da_ = s1 * dz;
            d1_ = s * s1;
            r_ = s * dz * (-2.f * a * s1);
        };
        one(a1.x, sd.x, z[o][0], da.x, d1.x, r.x);
        one(a1.y, sd.y, z[o][1], da.y, d1.y, r.y);
        one(a1.z, sd.z, z[o][2], da.z, d1.z, r.z);
        one(a1.w, sd.w, z[o][3], da.w, d1.w, r.w);
        nt_at(A1, j, ta) = a1;
        nt_at(DA1, j, ta) = da;
        nt_at(D1, j, ta) = d1;
        nt_at(Z1, j, ta) = r;
    }
    __syncthreads();
    nt_zero(z);
    nt_rows<NN_H, NT_W2S>(q.W2, DA1, to, ta, z);
#pragma unroll
    for (int o = 0; o < NT_R; o++) {
        const int j = to + NT_TO * o;
        const float w3 = q.w3[j];
        const float4 a2 = *reinterpret_cast<const float4*>(act + (NN_H + j) * NN_CHUNK);
        float4 d2, r2, z2, g3;
        const auto one = [&](float a, float dz, float ei, float& d2_, float& r2_, float& z2_, float& g3_) {
            const float s2 = 1.f - a * a;
            d2_ = w3 * s2;
            r2_ = w3 * dz * (-2.f * a * s2);
            z2_ = ei * d2_ + r2_;
            g3_ = ei * a + s2 * dz;
        };
        one(a2.x, z[o][0], e4.x, d2.x, r2.x, z2.x, g3.x);
        one(a2.y, z[o][1], e4.y, d2.y, r2.y, z2.y, g3.y);
        one(a2.z, z[o][2], e4.z, d2.z, r2.z, z2.z, g3.z);
        one(a2.w, z[o][3], e4.w, d2.w, r2.w, z2.w, g3.w);
        nt_at(D2, j, ta) = d2;
        nt_at(R2, j, ta) = r2;
        nt_at(Z2, j, ta) = z2;
        const float gw3 = nt_sum(g3), gb2 = nt_sum(z2);
        if (ta == 0) {
            out[NN_OFF_W3 + j] = gw3;
            out[NN_OFF_B2 + j] = gb2;
        }
    }
    __syncthreads();
    nt_zero(z);
    nt_cols<NT_R, NT_W2S>(q.W2, R2, to, ta, z);
#pragma unroll
    for (int c = 0; c < NT_R; c++) {
        const int j = NT_R * to + c;
        const float4 a1 = nt_at(A1, j, ta), d1 = nt_at(D1, j, ta), r = nt_at(Z1, j, ta);
        const float4 z1 = make_float4(e4.x * d1.x + (z[c][0] * (1.f - a1.x * a1.x) + r.x),
                                      e4.y * d1.y + (z[c][1] * (1.f - a1.y * a1.y) + r.y),
                                      e4.z * d1.z + (z[c][2] * (1.f - a1.z * a1.z) + r.z),
                                      e4.w * d1.w + (z[c][3] * (1.f - a1.w * a1.w) + r.w));
        nt_at(Z1, j, ta) = z1;
        const float gb1 = nt_sum(z1);
        if (ta == 0) out[NN_OFF_B1 + j] = gb1;
    }
    __syncthreads();
    nt_outer<8, NN_H>(Z2, A1, D2, DA1, out + NN_OFF_W2);
    nt_outer<4, NN_DESC>(Z1, G, D1, VT, out + NN_OFF_W1);
}

// One Adam step's factors; on = 0: leave the weights alone.
struct NTAdam {
    int on;
    float lr, b1, b2, eps;
};

// The chunks' partial gradients summed in FP64 (each of NT_SPLIT threads a
// run of the chunks, the runs in order), the gradient stored and the weights
// stepped.
constexpr int NT_SPLIT = 8;
constexpr int NT_FINAL_BLOCKS = (NN_PARAMS + 31) / 32;

__global__ void __launch_bounds__(32 * NT_SPLIT) k_nn_step(const float* __restrict__ partial, int nchunks,
                                                           float* __restrict__ grad, NTAdam ad, float* __restrict__ w,
                                                           float* __restrict__ m, float* __restrict__ v) {
    __shared__ double red[32 * NT_SPLIT];
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    double s = 0.0;
    const int k = blockIdx.x * 32 + lane;
    const int per = (nchunks + NT_SPLIT - 1) / NT_SPLIT, c0 = part * per, c1 = min(nchunks, c0 + per);
    if (k < NN_PARAMS) {
#pragma unroll 8
        for (int c = c0; c < c1; c++) s += f2d_exact(__ldg(partial + (size_t)c * NN_PARAMS + k));  // no FP64 conversion
    }
    red[threadIdx.x] = s;
    __syncthreads();
    if (part != 0 || k >= NN_PARAMS) return;
    for (int q = 1; q < NT_SPLIT; q++) s += red[q * 32 + lane];
    const float gk = (float)s;
    grad[k] = gk;
    if (!ad.on) return;
    const float mk = ad.b1 * m[k] + (1.f - ad.b1) * gk;
    const float vk = ad.b2 * v[k] + (1.f - ad.b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    w[k] -= ad.lr * mk / (sqrtf(vk) + ad.eps);
}

// The atoms of the configurations in the epoch's order, back to back.
__global__ void k_nn_order(const int* __restrict__ clist, const int* __restrict__ at,
                           const int* __restrict__ conf_start, int* __restrict__ list) {
    const int c = clist[blockIdx.x], a = conf_start[c], n = conf_start[c + 1] - a;
    for (int k = threadIdx.x; k < n; k += blockDim.x) list[at[blockIdx.x] + k] = a + k;
}

}  // namespace omdg

// ====================================================================== C ABI
using namespace omdg;

static int nn_fail(omdg_nn* t, int code, const std::string& msg) {
    if (t) t->err = msg;
    return code;
}

static int nn_cuda(omdg_nn* t, cudaError_t e, const char* what) {
    if (e == cudaSuccess) return OMDG_OK;
    return nn_fail(t, OMDG_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

static int nn_status(omdg_nn* t) {
    unsigned st = 0;
    cudaError_t e = cudaMemcpyAsync(&st, t->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    if (e != cudaSuccess) return nn_cuda(t, e, "status");
    if (!st) return OMDG_OK;
    unsigned zero = 0;
    cudaMemcpy(t->d_status, &zero, sizeof(unsigned), cudaMemcpyHostToDevice);
    if (st & ERR_TIMEOUT) return nn_fail(t, OMDG_ECUDA, "tensor-core kernel wait timed out");
    if (st & ERR_NBR_OVERFLOW) return nn_fail(t, OMDG_ESTATE, "asymmetric neighbour slots");
    return nn_fail(t, OMDG_ECUDA, "device status word set");
}

static void nn_free_data(omdg_nn* t) {
    cudaFree(t->d_fw);
    cudaFree(t->d_eatom);
    cudaFree(t->d_ewa);
    t->d_fw = t->d_eatom = t->d_ewa = nullptr;
    void* ptrs[] = {t->d_conf_start, t->d_atom_conf, t->d_x,     t->d_L,      t->d_eref,    t->d_fref,   t->d_slot_start,
                    t->d_slot_j,     t->d_slot_rev,  t->d_slot_d, t->d_G,     t->d_Gt,      t->d_J,      t->d_E,
                    t->d_u,          t->d_F,         t->d_rho,   t->d_vvec,   t->d_ew,      t->d_lossE,  t->d_lossF,
                    t->d_acts,       t->d_partial,   t->d_list,  t->d_clist};
    for (void* p : ptrs) cudaFree(p);
    t->d_conf_start = t->d_atom_conf = t->d_slot_start = t->d_slot_j = t->d_slot_rev = t->d_list = t->d_clist = nullptr;
    t->d_x = t->d_L = nullptr;
    t->d_eref = t->d_fref = t->d_G = t->d_Gt = t->d_J = t->d_E = t->d_u = t->d_F = t->d_rho = t->d_vvec = nullptr;
    t->d_ew = t->d_lossE = t->d_lossF = t->d_acts = t->d_partial = nullptr;
    t->d_slot_d = nullptr;
    t->nconf = 0;
    t->natoms = t->nslots = 0;
    t->cap_batch_atoms = t->cap_clist = 0;
}

template <typename T>
static cudaError_t dalloc(T** p, size_t count) {
    return cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * std::max<size_t>(count, 1));
}

extern "C" {

int omdg_nn_create(omdg_nn** out, int device) {
    if (!out) return OMDG_EINVAL;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return OMDG_ECUDA;
    omdg_nn* t = new omdg_nn();
    t->device = device;
    cudaSetDevice(device);
    cudaDeviceGetAttribute(&t->num_sms, cudaDevAttrMultiProcessorCount, device);
    cudaError_t e = cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = dalloc(&t->d_status, 1);
    if (e == cudaSuccess) e = cudaMemset(t->d_status, 0, sizeof(unsigned));
    if (e == cudaSuccess) e = dalloc(&t->d_params, NN_PARAMS);
    if (e == cudaSuccess) e = dalloc(&t->d_adam_m, NN_PARAMS);
    if (e == cudaSuccess) e = dalloc(&t->d_adam_v, NN_PARAMS);
    if (e == cudaSuccess) e = dalloc(&t->d_grad, NN_PARAMS);
    if (e != cudaSuccess) {
        delete t;
        return OMDG_ECUDA;
    }
    nn_default_descriptors(t->model.dp);
    for (int d = 0; d < NN_DESC; d++) t->model.sigma[d] = 1.f;
    t->model.w.assign(NN_PARAMS, 0.f);
    *out = t;
    return OMDG_OK;
}

int omdg_nn_destroy(omdg_nn* t) {
    if (!t) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    nn_free_data(t);
    void* ptrs[] = {t->d_status, t->d_params, t->d_adam_m, t->d_adam_v, t->d_grad, t->d_loss};
    for (void* p : ptrs) cudaFree(p);
    nn_net_free(t->net);
    cudaStreamDestroy(t->stream);
    delete t;
    return OMDG_OK;
}

const char* omdg_nn_last_error(omdg_nn* t) { return t ? t->err.c_str() : "null network"; }

int omdg_nn_set_weights(omdg_nn* t, const float* params, long count) {
    if (!t || !params || count != NN_PARAMS) return t ? nn_fail(t, OMDG_EINVAL, "expected 6337 parameters") : OMDG_EINVAL;
    cudaSetDevice(t->device);
    t->model.w.assign(params, params + NN_PARAMS);
    t->have_weights = true;
    t->adam_t = 0;
    cudaError_t e = cudaMemcpyAsync(t->d_params, params, sizeof(float) * NN_PARAMS, cudaMemcpyHostToDevice, t->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(t->d_adam_m, 0, sizeof(float) * NN_PARAMS, t->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(t->d_adam_v, 0, sizeof(float) * NN_PARAMS, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    return nn_cuda(t, e, "set weights");
}

int omdg_nn_get_weights(omdg_nn* t, float* params, long count) {
    if (!t || !params || count != NN_PARAMS) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    cudaError_t e = cudaMemcpy(params, t->d_params, sizeof(float) * NN_PARAMS, cudaMemcpyDeviceToHost);
    return nn_cuda(t, e, "get weights");
}

int omdg_nn_set_normalization(omdg_nn* t, const float* mu, const float* sigma, const float* gmin, const float* gmax) {
    if (!t || !mu || !sigma) return OMDG_EINVAL;
    for (int d = 0; d < NN_DESC; d++) {
        if (!(sigma[d] > 0.f)) return nn_fail(t, OMDG_EINVAL, "sigma must be positive");
        t->model.dp.mu[d] = mu[d];
        t->model.sigma[d] = sigma[d];
        t->model.dp.isig[d] = 1.f / sigma[d];
        t->model.dp.gmin[d] = gmin ? gmin[d] : -INFINITY;
        t->model.dp.gmax[d] = gmax ? gmax[d] : INFINITY;
    }
    if (t->natoms > 0) {
        cudaSetDevice(t->device);
        const long q = t->natoms * NN_DESC;
        k_nn_normalize<<<(unsigned)((q + 255) / 256), 256, 0, t->stream>>>(t->model.dp, t->natoms, t->d_G, t->d_Gt);
        return nn_cuda(t, cudaStreamSynchronize(t->stream), "normalise");
    }
    return OMDG_OK;
}

int omdg_nn_get_normalization(omdg_nn* t, float* mu, float* sigma, float* gmin, float* gmax) {
    if (!t) return OMDG_EINVAL;
    for (int d = 0; d < NN_DESC; d++) {
        if (mu) mu[d] = t->model.dp.mu[d];
        if (sigma) sigma[d] = t->model.sigma[d];
        if (gmin) gmin[d] = t->model.dp.gmin[d];
        if (gmax) gmax[d] = t->model.dp.gmax[d];
    }
    return OMDG_OK;
}

int omdg_nn_save(omdg_nn* t, const char* path) {
    if (!t || !path) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    int rc = omdg_nn_get_weights(t, t->model.w.data(), NN_PARAMS);
    if (rc) return rc;
    return nn_model_save(path, t->model, t->err);
}

int omdg_nn_load(omdg_nn* t, const char* path) {
    if (!t || !path) return OMDG_EINVAL;
    NNModel m;
    int rc = nn_model_load(path, m, t->err);
    if (rc) return rc;
    rc = omdg_nn_set_normalization(t, m.dp.mu, m.sigma, m.dp.gmin, m.dp.gmax);
    if (rc) return rc;
    t->model.dp = m.dp;
    return omdg_nn_set_weights(t, m.w.data(), NN_PARAMS);
}

int omdg_nn_set_descriptors(omdg_nn* t, const float* rs, const float* eta_r, const int* zeta, const float* lambda,
                            const float* eta_a) {
    if (!t || !rs || !eta_r || !zeta || !lambda || !eta_a) return OMDG_EINVAL;
    if (t->natoms > 0) return nn_fail(t, OMDG_ESTATE, "set the descriptors before the dataset");
    NNDescParams& p = t->model.dp;
    for (int k = 0; k < NN_RAD; k++) {
        if (!(eta_r[k] >= 0.f)) return nn_fail(t, OMDG_EINVAL, "radial eta must be >= 0");
        p.rs[k] = rs[k];
        p.eta_r[k] = eta_r[k];
    }
    for (int m = 0; m < NN_ANG; m++) {
        if (zeta[m] < 1 || zeta[m] > 16) return nn_fail(t, OMDG_EINVAL, "zeta must be an integer in [1, 16]");
        if (!(eta_a[m] >= 0.f)) return nn_fail(t, OMDG_EINVAL, "angular eta must be >= 0");
        p.zeta[m] = zeta[m];
        p.lam[m] = lambda[m];
        p.eta_a[m] = eta_a[m];
        p.pref[m] = (float)std::pow(2.0, 1.0 - zeta[m]);
    }
    return OMDG_OK;
}

int omdg_nn_set_cutoff(omdg_nn* t, float rc, float rin) {
    if (!t) return OMDG_EINVAL;
    if (t->natoms > 0) return nn_fail(t, OMDG_ESTATE, "set the cutoff before the dataset");
    if (!nn_set_cutoff(t->model.dp, rc, rin)) return nn_fail(t, OMDG_EINVAL, "the cutoff needs 0 <= rin < rc");
    return OMDG_OK;
}

int omdg_nn_set_dataset(omdg_nn* t, int nconf, const int* natoms, const double* x, const double* box_len,
                        const double* energy, const double* forces) {
    if (!t || nconf <= 0 || !natoms || !x || !box_len || !energy || !forces) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    nn_free_data(t);
    const double rc = t->model.dp.rc;
    std::vector<int> start(nconf + 1, 0), atom_conf;
    for (int c = 0; c < nconf; c++) {
        if (natoms[c] <= 0) return nn_fail(t, OMDG_EINVAL, "configuration without atoms");
        for (int a = 0; a < 3; a++)
            if (!(box_len[3 * c + a] >= 2.0 * rc))
                return nn_fail(t, OMDG_EINVAL, "every box length must be at least twice the descriptor cutoff");
        start[c + 1] = start[c] + natoms[c];
        atom_conf.insert(atom_conf.end(), natoms[c], c);
    }
    const long n = start[nconf];
    std::vector<float> eref(nconf), fref(3 * (size_t)n);
    for (int c = 0; c < nconf; c++) eref[c] = (float)energy[c];
    for (long q = 0; q < 3 * n; q++) fref[q] = (float)forces[q];
    cudaError_t e = dalloc(&t->d_conf_start, nconf + 1);
    if (e == cudaSuccess) e = dalloc(&t->d_atom_conf, n);
    if (e == cudaSuccess) e = dalloc(&t->d_x, 3 * n);
    if (e == cudaSuccess) e = dalloc(&t->d_L, 3 * (size_t)nconf);
    if (e == cudaSuccess) e = dalloc(&t->d_eref, nconf);
    if (e == cudaSuccess) e = dalloc(&t->d_fref, 3 * n);
    if (e == cudaSuccess) e = dalloc(&t->d_fw, nconf);
    if (e == cudaSuccess) e = dalloc(&t->d_slot_start, n + 1);
    if (e == cudaSuccess) e = dalloc(&t->d_G, n * NN_DESC);
    if (e == cudaSuccess) e = dalloc(&t->d_Gt, n * NN_DESC);
    if (e == cudaSuccess) e = dalloc(&t->d_E, n);
    if (e == cudaSuccess) e = dalloc(&t->d_u, n * NN_DESC);
    if (e == cudaSuccess) e = dalloc(&t->d_F, 3 * n);
    if (e == cudaSuccess) e = dalloc(&t->d_rho, 3 * n);
    if (e == cudaSuccess) e = dalloc(&t->d_vvec, n * NN_DESC);
    if (e == cudaSuccess) e = dalloc(&t->d_ew, nconf);
    if (e == cudaSuccess) e = dalloc(&t->d_list, n);
    if (e != cudaSuccess) return nn_cuda(t, e, "dataset allocation");
    cudaStream_t s = t->stream;
    cudaMemcpyAsync(t->d_conf_start, start.data(), sizeof(int) * (nconf + 1), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(t->d_atom_conf, atom_conf.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(t->d_x, x, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(t->d_L, box_len, sizeof(double) * 3 * nconf, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(t->d_eref, eref.data(), sizeof(float) * nconf, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(t->d_fref, fref.data(), sizeof(float) * 3 * n, cudaMemcpyHostToDevice, s);
    t->fms.assign(nconf, 0.f);
    for (int c = 0; c < nconf; c++) {
        double q = 0;
        for (long a = 3L * start[c]; a < 3L * start[c + 1]; a++) q += (double)forces[a] * forces[a];
        t->fms[c] = (float)(q / (3.0 * natoms[c]));
    }
    std::vector<float> ones(nconf, 1.f);
    cudaMemcpyAsync(t->d_fw, ones.data(), sizeof(float) * nconf, cudaMemcpyHostToDevice, s);
    const unsigned blocks = (unsigned)((n + 127) / 128);
    int* d_count = t->d_slot_start;  // counts first, then converted to starts on the host
    k_nn_count<<<blocks, 128, 0, s>>>(n, t->d_atom_conf, t->d_conf_start, t->d_x, t->d_L, rc * rc, d_count);
    std::vector<int> cnt(n + 1, 0);
    e = cudaMemcpyAsync(cnt.data(), d_count, sizeof(int) * n, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return nn_cuda(t, e, "neighbour count");
    std::vector<int> sstart(n + 1, 0);
    for (long i = 0; i < n; i++) {
        if (cnt[i] > NN_MAXN) return nn_fail(t, OMDG_ESTATE, "an atom has more than 24 neighbours inside the cutoff");
        sstart[i + 1] = sstart[i] + cnt[i];
    }
    const long ns = sstart[n];
    e = dalloc(&t->d_slot_j, ns);
    if (e == cudaSuccess) e = dalloc(&t->d_slot_rev, ns);
    if (e == cudaSuccess) e = dalloc(&t->d_slot_d, ns);
    if (e == cudaSuccess) e = dalloc(&t->d_J, (size_t)ns * 3 * NN_DESC);
    if (e != cudaSuccess) return nn_cuda(t, e, "slot allocation");
    cudaMemcpyAsync(t->d_slot_start, sstart.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice, s);
    k_nn_fill<<<blocks, 128, 0, s>>>(n, t->d_atom_conf, t->d_conf_start, t->d_x, t->d_L, rc * rc, t->d_slot_start,
                                     t->d_slot_j, t->d_slot_d);
    k_nn_rev<<<blocks, 128, 0, s>>>(n, t->d_slot_start, t->d_slot_j, t->d_slot_rev, t->d_status);
    k_nn_train_desc<<<blocks, 128, 0, s>>>(t->model.dp, n, t->d_slot_start, t->d_slot_d, t->d_G, t->d_J);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return nn_cuda(t, e, "descriptors");
    t->nconf = nconf;
    t->natoms = n;
    t->nslots = ns;
    t->conf_start = start;
    int rc2 = nn_status(t);
    if (rc2) return rc2;
    return omdg_nn_set_normalization(t, t->model.dp.mu, t->model.sigma, t->model.dp.gmin, t->model.dp.gmax);
}

// relative != 0: each configuration's force residual is weighted by the mean
// square reference force over the dataset divided by its own, so that every
// configuration counts by its relative force error; 0: plain mean square.
int omdg_nn_set_force_weighting(omdg_nn* t, int relative) {
    if (!t || t->nconf == 0) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    std::vector<float> w(t->nconf, 1.f);
    if (relative) {
        double mean = 0;
        for (float q : t->fms) mean += q;
        mean /= t->nconf;
        for (int c = 0; c < t->nconf; c++) w[c] = t->fms[c] > 0.f ? (float)(mean / t->fms[c]) : 1.f;
    }
    cudaError_t e = cudaMemcpyAsync(t->d_fw, w.data(), sizeof(float) * t->nconf, cudaMemcpyHostToDevice, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    return nn_cuda(t, e, "force weights");
}

// Per-atom reference energies: the energy term of the loss becomes
// wE mean_i (E_i - E_i^ref)^2 over the batch atoms; NULL returns to the
// per-configuration total-energy term.
int omdg_nn_set_atom_energies(omdg_nn* t, const double* e_atom) {
    if (!t || t->natoms == 0) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    cudaFree(t->d_eatom);
    cudaFree(t->d_ewa);
    t->d_eatom = t->d_ewa = nullptr;
    if (!e_atom) return OMDG_OK;
    std::vector<float> h(e_atom, e_atom + t->natoms);
    cudaError_t e = dalloc(&t->d_eatom, t->natoms);
    if (e == cudaSuccess) e = dalloc(&t->d_ewa, t->natoms);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(t->d_eatom, h.data(), sizeof(float) * t->natoms, cudaMemcpyHostToDevice, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    return nn_cuda(t, e, "atom energies");
}

int omdg_nn_descriptors(omdg_nn* t, float* G, long count) {
    if (!t || !G || count != t->natoms * NN_DESC) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    return nn_cuda(t, cudaMemcpy(G, t->d_G, sizeof(float) * count, cudaMemcpyDeviceToHost), "descriptors");
}

// Mean, standard deviation and range of every descriptor over the dataset.
int omdg_nn_normalize_from_dataset(omdg_nn* t) {
    if (!t || t->natoms == 0) return OMDG_EINVAL;
    std::vector<float> G(t->natoms * NN_DESC);
    int rc = omdg_nn_descriptors(t, G.data(), (long)G.size());
    if (rc) return rc;
    float mu[NN_DESC], sg[NN_DESC], lo[NN_DESC], hi[NN_DESC];
    for (int d = 0; d < NN_DESC; d++) {
        double s = 0, s2 = 0;
        float a = INFINITY, b = -INFINITY;
        for (long i = 0; i < t->natoms; i++) {
            const double v = G[i * NN_DESC + d];
            s += v;
            s2 += v * v;
            a = std::min(a, (float)v);
            b = std::max(b, (float)v);
        }
        const double m = s / t->natoms;
        const double var = std::max(0.0, s2 / t->natoms - m * m);
        mu[d] = (float)m;
        // a descriptor that does not vary over the dataset keeps scale 1
        const double sd = std::sqrt(var);
        sg[d] = (float)(sd > 1e-6 * std::max(std::fabs(m), 1e-30) ? sd : 1.0);
        lo[d] = a;
        hi[d] = b;
    }
    return omdg_nn_set_normalization(t, mu, sg, lo, hi);
}

static int ensure_batch(omdg_nn* t, long atoms) {
    if (atoms <= t->cap_batch_atoms) return OMDG_OK;
    cudaFree(t->d_lossE);
    cudaFree(t->d_lossF);
    cudaFree(t->d_acts);
    cudaFree(t->d_partial);
    const long chunks = (atoms + NN_CHUNK - 1) / NN_CHUNK;
    cudaError_t e = dalloc(&t->d_lossE, std::max<long>(t->nconf, atoms));
    if (e == cudaSuccess) e = dalloc(&t->d_lossF, atoms);
    if (e == cudaSuccess) e = dalloc(&t->d_acts, (size_t)chunks * NT_ACTS * NN_CHUNK);
    if (e == cudaSuccess) e = dalloc(&t->d_partial, (size_t)chunks * NN_PARAMS);
    if (e != cudaSuccess) return nn_cuda(t, e, "batch allocation");
    t->cap_batch_atoms = atoms;
    return OMDG_OK;
}

static void nn_kernel_attributes() {
    cudaFuncSetAttribute(k_nn_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(float) * NT_FWD_FLOATS);
    cudaFuncSetAttribute(k_nn_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(float) * NT_GRAD_FLOATS);
}

// Loss and gradient over the configurations clist[c0 .. c0 + nb) whose atoms
// are list[a0 .. a0 + na); leaves dL/dw in d_grad and L in loss, and steps the
// weights when ad says so.
static int nn_loss_grad(omdg_nn* t, const int* clist, int c0, int nb, long a0, long na, double wE, double wF,
                        const NTAdam& ad, double* loss) {
    int rc = ensure_batch(t, na);
    if (rc) return rc;
    cudaStream_t s = t->stream;
    const NNDescParams& p = t->model.dp;
    nn_kernel_attributes();
    const int chunks = (int)((na + NN_CHUNK - 1) / NN_CHUNK);
    const unsigned wb = (unsigned)((na + 7) / 8);  // blocks of eight warps, an atom each
    k_nn_fwd<<<chunks, NT_THREADS, sizeof(float) * NT_FWD_FLOATS, s>>>(
        t->d_params, t->d_Gt, p, t->d_list, (int)a0, (int)na, t->d_E, t->d_u, t->d_acts, t->d_eatom, (float)wE,
        t->d_ewa, t->d_lossE);
    if (!t->d_eatom)
        k_nn_conf_energy<<<nb, 256, 0, s>>>(clist, c0, nb, t->d_conf_start, t->d_E, t->d_eref, (float)wE, t->d_ew,
                                            t->d_lossE);
    k_nn_force<<<wb, 256, 0, s>>>(t->d_list, (int)a0, (int)na, t->d_slot_start, t->d_slot_j, t->d_slot_rev, t->d_J,
                                  t->d_u, t->d_fref, (float)(wF / (3.0 * na)), t->d_fw, t->d_atom_conf, t->d_F,
                                  t->d_rho, t->d_lossF);
    k_nn_vvec<<<wb, 256, 0, s>>>(t->d_list, (int)a0, (int)na, t->d_slot_start, t->d_slot_j, t->d_J, t->d_rho,
                                 t->d_vvec);
    k_nn_grad<<<chunks + 1, NT_THREADS, sizeof(float) * NT_GRAD_FLOATS, s>>>(
        t->d_params, t->d_Gt, t->d_vvec, p, t->d_acts, t->d_list, t->d_eatom ? t->d_ewa : t->d_ew,
        t->d_eatom ? nullptr : t->d_atom_conf, (int)a0, (int)na, t->d_partial, t->d_lossE,
        t->d_eatom ? (int)na : nb, t->d_lossF, loss);
    k_nn_step<<<NT_FINAL_BLOCKS, 32 * NT_SPLIT, 0, s>>>(t->d_partial, chunks, t->d_grad, ad, t->d_params, t->d_adam_m,
                                                        t->d_adam_v);
    return nn_cuda(t, cudaGetLastError(), "training step");
}

// The configuration orders of `epochs` epochs (confs, back to back) to the
// device; conf_atoms0 gives where each configuration's atoms begin in its
// epoch's atom order, which nn_order writes.
static int upload_orders(omdg_nn* t, const std::vector<int>& confs, int epochs, std::vector<int>& conf_atoms0) {
    const size_t n = confs.size(), per = n / epochs;
    std::vector<int> up(confs);
    up.resize(2 * n);
    conf_atoms0.assign((per + 1) * epochs, 0);
    for (int ep = 0; ep < epochs; ep++) {
        int* at = conf_atoms0.data() + (per + 1) * ep;
        for (size_t k = 0; k < per; k++) {
            const int c = confs[per * ep + k];
            up[n + per * ep + k] = at[k];
            at[k + 1] = at[k] + (t->conf_start[c + 1] - t->conf_start[c]);
        }
    }
    if ((long)up.size() > t->cap_clist) {
        cudaFree(t->d_clist);
        t->d_clist = nullptr;
        t->cap_clist = 0;
        cudaError_t e = dalloc(&t->d_clist, up.size());
        if (e != cudaSuccess) return nn_cuda(t, e, "batch order");
        t->cap_clist = (long)up.size();
    }
    cudaError_t e = cudaMemcpyAsync(t->d_clist, up.data(), sizeof(int) * up.size(), cudaMemcpyHostToDevice, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    return nn_cuda(t, e, "batch order");
}

// The atom order of one uploaded epoch (n configurations in all epochs, per of them in each).
static void nn_order(omdg_nn* t, size_t n, size_t per, int ep) {
    k_nn_order<<<(unsigned)per, 256, 0, t->stream>>>(t->d_clist + per * ep, t->d_clist + n + per * ep, t->d_conf_start,
                                                    t->d_list);
}

static int ensure_losses(omdg_nn* t, long n) {
    if (n <= t->cap_loss) return OMDG_OK;
    cudaFree(t->d_loss);
    t->d_loss = nullptr;
    t->cap_loss = 0;
    cudaError_t e = dalloc(&t->d_loss, n);
    if (e != cudaSuccess) return nn_cuda(t, e, "loss allocation");
    t->cap_loss = n;
    return OMDG_OK;
}

int omdg_nn_gradient(omdg_nn* t, int conf0, int nconf, double wE, double wF, double* loss, float* grad) {
    if (!t || conf0 < 0 || nconf <= 0 || conf0 + nconf > t->nconf) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    std::vector<int> confs(nconf);
    std::iota(confs.begin(), confs.end(), conf0);
    std::vector<int> ca;
    int rc = upload_orders(t, confs, 1, ca);
    if (!rc) rc = ensure_losses(t, 1);
    if (rc) return rc;
    nn_order(t, confs.size(), confs.size(), 0);
    if ((rc = nn_loss_grad(t, t->d_clist, 0, nconf, 0, ca[nconf], wE, wF, NTAdam{}, t->d_loss))) return rc;
    cudaError_t e = cudaSuccess;
    if (loss) e = cudaMemcpyAsync(loss, t->d_loss, sizeof(double), cudaMemcpyDeviceToHost, t->stream);
    if (grad && e == cudaSuccess)
        e = cudaMemcpyAsync(grad, t->d_grad, sizeof(float) * NN_PARAMS, cudaMemcpyDeviceToHost, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    if (e != cudaSuccess) return nn_cuda(t, e, "gradient");
    return nn_status(t);
}

int omdg_nn_train(omdg_nn* t, int epochs, int batch_confs, double lr, double lr_final, double wE, double wF,
                  unsigned seed, double* epoch_loss) {
    if (!t || epochs <= 0 || batch_confs <= 0 || !(lr > 0) || !(lr_final > 0) || t->nconf == 0) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    std::mt19937 rng(seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    std::vector<int> confs(t->nconf), orders, ca;
    std::iota(confs.begin(), confs.end(), 0);
    // epochs are queued in groups (orders of up to 2^20 configurations); the
    // host waits, and reads the batches' losses, once per group
    const int nbatch = (t->nconf + batch_confs - 1) / batch_confs;
    const int group = std::max(1, std::min(epochs, (1 << 20) / t->nconf));
    std::vector<double> losses((size_t)group * nbatch);
    int rc = ensure_losses(t, (long)losses.size());
    if (rc) return rc;
    for (int e0 = 0; e0 < epochs; e0 += group) {
        const int ne = std::min(group, epochs - e0);
        orders.clear();
        for (int k = 0; k < ne; k++) {
            std::shuffle(confs.begin(), confs.end(), rng);
            orders.insert(orders.end(), confs.begin(), confs.end());
        }
        if ((rc = upload_orders(t, orders, ne, ca))) return rc;
        for (int k = 0; k < ne; k++) {
            const int ep = e0 + k;
            // cosine decay from lr (first epoch) to lr_final (last epoch)
            const double lr_ep =
                epochs > 1 ? lr_final + 0.5 * (lr - lr_final) * (1.0 + std::cos(M_PI * ep / (epochs - 1))) : lr;
            const int* at = ca.data() + (size_t)(t->nconf + 1) * k;
            nn_order(t, orders.size(), t->nconf, k);
            for (int c0 = 0, b = 0; c0 < t->nconf; c0 += batch_confs, b++) {
                const int nb = std::min(batch_confs, t->nconf - c0);
                t->adam_t++;
                const double bc1 = 1.0 - std::pow((double)b1, (double)t->adam_t);
                const double bc2 = 1.0 - std::pow((double)b2, (double)t->adam_t);
                const float lr_t = (float)(lr_ep * std::sqrt(bc2) / bc1);
                rc = nn_loss_grad(t, t->d_clist + (size_t)t->nconf * k, c0, nb, at[c0], at[c0 + nb] - at[c0], wE, wF,
                                  NTAdam{1, lr_t, b1, b2, eps}, t->d_loss + (size_t)nbatch * k + b);
                if (rc) return rc;
            }
        }
        cudaError_t e = cudaSuccess;
        if (epoch_loss)
            e = cudaMemcpyAsync(losses.data(), t->d_loss, sizeof(double) * (size_t)ne * nbatch,
                                cudaMemcpyDeviceToHost, t->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
        if (e != cudaSuccess) return nn_cuda(t, e, "training");
        for (int k = 0; epoch_loss && k < ne; k++) {
            double sum = 0.0;
            for (int b = 0; b < nbatch; b++) sum += losses[(size_t)nbatch * k + b];
            epoch_loss[e0 + k] = sum / std::max(1, nbatch);
        }
    }
    rc = nn_status(t);
    if (rc) return rc;
    return omdg_nn_get_weights(t, t->model.w.data(), NN_PARAMS);
}

// Energies per atom and forces of configurations [conf0, conf0 + nconf) with
// the tensor-core network (BF16 weights and activations, FP32 accumulation).
int omdg_nn_predict(omdg_nn* t, int conf0, int nconf, int fp32, double* energy_per_atom, double* forces) {
    if (!t || conf0 < 0 || nconf <= 0 || conf0 + nconf > t->nconf) return OMDG_EINVAL;
    cudaSetDevice(t->device);
    int rc = omdg_nn_get_weights(t, t->model.w.data(), NN_PARAMS);
    if (rc) return rc;
    if ((rc = nn_net_upload(t->net, t->model, t->stream, t->err))) return rc;
    std::vector<int> confs(nconf);
    std::iota(confs.begin(), confs.end(), conf0);
    std::vector<int> ca;
    if ((rc = upload_orders(t, confs, 1, ca))) return rc;
    nn_order(t, confs.size(), confs.size(), 0);
    const long a0 = t->conf_start[conf0], na = t->conf_start[conf0 + nconf] - a0;
    cudaError_t e = cudaSuccess;
    if (fp32) {
        nn_kernel_attributes();
        k_nn_fwd<<<(unsigned)((na + NN_CHUNK - 1) / NN_CHUNK), NT_THREADS, sizeof(float) * NT_FWD_FLOATS, t->stream>>>(
            t->d_params, t->d_Gt, t->model.dp, t->d_list, 0, (int)na, t->d_E, t->d_u, nullptr, nullptr, 0.f, nullptr,
            nullptr);
        e = cudaGetLastError();
    } else {
        e = nn_mlp_launch(t->net, t->d_Gt + a0 * NN_DESC, (int)na, t->d_E + a0, t->d_u + a0 * NN_DESC, t->d_status,
                          t->num_sms, t->stream);
    }
    if (e != cudaSuccess) return nn_cuda(t, e, "network");
    k_nn_force<<<(unsigned)((na + 7) / 8), 256, 0, t->stream>>>(t->d_list, 0, (int)na, t->d_slot_start, t->d_slot_j, t->d_slot_rev, t->d_J,
                                          t->d_u, nullptr, 0.f, nullptr, nullptr, t->d_F, nullptr, nullptr);
    std::vector<float> E(na), F(3 * na);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(E.data(), t->d_E + a0, sizeof(float) * na, cudaMemcpyDeviceToHost, t->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(F.data(), t->d_F + 3 * a0, sizeof(float) * 3 * na, cudaMemcpyDeviceToHost, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    if (e != cudaSuccess) return nn_cuda(t, e, "predict");
    if ((rc = nn_status(t))) return rc;
    for (long i = 0; i < na; i++) {
        if (energy_per_atom) energy_per_atom[i] = E[i];
        if (forces)
            for (int c = 0; c < 3; c++) forces[3 * i + c] = F[3 * i + c];
    }
    return OMDG_OK;
}

}  // extern "C"
