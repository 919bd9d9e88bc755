// Spectral initialisation on the device: chebyshev_eigenvectors (src/spectral.cpp:141-241), the Chebyshev-filtered
// subspace iteration with Rayleigh-Ritz of the reference, in FP64 as the reference computes it. The block X is
// n x p, row major (p <= 8 columns), as the reference holds it.
//
// Kernels:
//  * step_kernel, one degree of the filter in one launch: the product with the lazy normalised adjacency (a group of
//    lanes per row, one per column, each summing the row's entries in order, as src/spectral.cpp:34-48), the deflation
//    of the trivial eigenvector t per component, and the three-term recurrence. The projection of M Y on t is that of Y on
//    u = M^T t, which the step before has summed while it wrote Y (per-component sums by block reductions and FP64
//    atomics): no pass between the product and the recurrence. On the graph's own degrees u is t but for inv_sqrt_deg's
//    rounding, and is held as u / t - 1 in single precision (to 1e-11 of t), read where it is used (read with the row's
//    other values the step took 45 us instead of 37). Where it is not (other scale factors, a directed graph), or an
//    edge joins two components, the steps take the product and the rest in two launches (finish_kernel). The block is
//    kept twice, as it is and with its rows scaled by D^-1/2 (what the next product gathers);
//  * the p x p products X^T X and X^T Z summed over the rows inside the kernels that write X or Z, the blocks' partial
//    sums added in a fixed order by the last block;
//  * two passes of Cholesky orthonormalisation (X <- X R^-1 with X^T X = R^T R, which is Gram-Schmidt of the columns in
//    exact arithmetic; the second pass restores the orthogonality the first leaves); a block too near to rank deficient
//    for it goes column by column;
//  * the rotation by the Ritz vectors with the residuals. The p x p factorisations and eigenproblem run on the host.
// Bound by the gathers of the products (one 8 p byte row per entry from L2) and their index reads. At 200k rows of 25
// entries, p = 4: 37 us per degree (136 G gathered rows/s) against 65 as five passes (product 48, component sums 4.6, deflation
// 6.4, recurrence 4.8), and 4 host round trips per outer iteration against 33.
#include "spectral.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

namespace mgb {
namespace {

constexpr int kSpecThreads = 256;
constexpr int kStepBlocks = 8;   // blocks per SM of the product: its sums cost one atomic per block and column

// blocks of the reductions (their partials go to the host) and of the row-parallel kernels (one row per thread)
int spec_blocks(int64_t rows) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((rows + kSpecThreads - 1) / kSpecThreads, 4 * kNumSMs));
}
int row_blocks(int64_t rows) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((rows + kSpecThreads - 1) / kSpecThreads, 64 * kNumSMs));
}

// the weight of node i on the trivial eigenvector: 1 / sd_i (0 for isolated nodes)
__device__ __forceinline__ double trivial_of(float sd) { return sd > 0.f ? 1.0 / (double)sd : 0.0; }

// lanes per row of the product: the power of two >= P
template <int P> constexpr int kLanes = P <= 2 ? 2 : (P <= 4 ? 4 : 8);

// the sum of one value per thread over a block's threads of the same column (threadIdx.x % G); result in threads < G
template <int G>
__device__ __forceinline__ double column_block_sum(double x, double (*red)[G]) {
#pragma unroll
    for (int o = 16; o >= G; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane < G) red[warp][lane] = x;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < G)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w][threadIdx.x];
    return t;
}

// running per-component sums of one column: rows of one component follow one another as a rule, so a thread adds to
// memory when the component changes, and a block whose threads end on one component once per column
struct ComponentSum {
    double sum = 0.0;
    int comp = -1;
    __device__ __forceinline__ void add(double x, int c, double* __restrict__ proj, int P, int k) {
        if (c != comp) {
            if (comp >= 0) atomicAdd(&proj[(int64_t)comp * P + k], sum);
            comp = c;
            sum = 0.0;
        }
        sum += x;
    }
};

// G lanes per row: thread's column k = threadIdx.x % G (k < P counts)
template <int P, int G>
__device__ __forceinline__ void flush_component(const ComponentSum& cs, double* __restrict__ proj, int k, double (*red)[G]) {
    __shared__ int any;
    if (threadIdx.x == 0) any = -1;
    __syncthreads();
    if (cs.comp >= 0) any = cs.comp;   // any one of them
    __syncthreads();
    const int c = any;
    if (__syncthreads_and(cs.comp < 0 || cs.comp == c)) {
        const double t = column_block_sum<G>(cs.comp >= 0 ? cs.sum : 0.0, red);
        if (c >= 0 && threadIdx.x < P) atomicAdd(&proj[(int64_t)c * P + threadIdx.x], t);
    } else if (cs.comp >= 0 && k < P) {
        atomicAdd(&proj[(int64_t)cs.comp * P + k], cs.sum);
    }
}

// the last block to finish adds the blocks' partial sums part[b][q], q < Q, in block order into out[q]
template <int Q>
__device__ __forceinline__ void sum_partials(const double* __restrict__ part, unsigned* __restrict__ counter,
                                             double* __restrict__ out) {
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int q = threadIdx.x >> 3; q < Q; q += blockDim.x >> 3) {   // 8 threads per entry, then their sums in order
        double t = 0.0;
        for (unsigned b = threadIdx.x & 7; b < gridDim.x; b += 8) t += __ldcg(&part[(size_t)b * Q + q]);
        const unsigned m = 0xffu << (threadIdx.x & 24);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(m, t, o);
        if ((threadIdx.x & 7) == 0) out[q] = t;
    }
    if (threadIdx.x == 0) *counter = 0u;
}

// One step Yout = (Z - c Yin) s - ss X with Z = M Yin deflated, M = (I + D^-1/2 A D^-1/2) / 2. Vin = D^-1/2 Yin is what
// the product gathers, Vout the same of Yout; X may be Yout (each entry is read before it is written). proj_in holds the
// per-component sums of t Yin, proj_out (zero before) receives those of t Yout, proj_next is set to zero for the step
// after. GRAM: part / counter / gram receive the p x p product Yin^T Yout. du: the sums are those of t (1 + du) Yout, as
// the next product wants them (zeros: of t Yout).
template <int P, bool GRAM>
__global__ void __launch_bounds__(kSpecThreads) step_kernel(
    const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices, const float* __restrict__ data,
    const float* __restrict__ sd, const int32_t* __restrict__ comp, const double* __restrict__ tnorm, int64_t n,
    const float* __restrict__ du, int64_t n_proj, const double* __restrict__ Yin, const double* __restrict__ Vin,
    const double* X, double* Yout, double* __restrict__ Vout, double c, double s, double ss, const double* __restrict__ proj_in,
    double* __restrict__ proj_out, double* __restrict__ proj_next, double* __restrict__ part,
    unsigned* __restrict__ counter, double* __restrict__ gram) {
    constexpr int G = kLanes<P>;
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ double red[kSpecThreads / 32][G];
    const int lane = threadIdx.x & 31, k = lane % G, base = lane - k;
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x / G);
    const int64_t g0 = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / G;   // the warp's first group
    for (int64_t z = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; z < n_proj; z += (int64_t)gridDim.x * blockDim.x)
        proj_next[z] = 0.0;
    ComponentSum cs;
    double h[GRAM ? P : 1];
#pragma unroll
    for (int a = 0; a < (GRAM ? P : 1); ++a) h[a] = 0.0;
    int last = -1;          // the component whose projection coefficient is at hand
    double pr = 0.0;
    for (int64_t gw = g0; gw < n; gw += groups) {
        const int64_t i = gw + lane / G;
        const bool row = i < n, mine = row && k < P;
        const int32_t e0 = row ? indptr[i] : 0, e1 = row ? indptr[i + 1] : 0;
        const float sdi = row ? sd[i] : 0.f;
        const int cc = row ? comp[i] : -1;
        const double y = mine ? Yin[i * P + k] : 0.0;
        const double xo = mine && ss != 0.0 ? X[i * P + k] : 0.0;
        // the group's lanes read 2 G entries at once, one trip ahead; each lane gathers its column of every entry, all
        // of a trip's before the first is used
        const int trips = __reduce_max_sync(kAll, (e1 - e0 + 2 * G - 1) / (2 * G));
        int32_t col[2];
        float w[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int32_t at = e0 + q * G + k;
            col[q] = at < e1 ? __ldg(&indices[at]) : 0;
            w[q] = at < e1 ? __ldg(&data[at]) : 0.f;
        }
        if (mine && cc != last) {
            last = cc;
            const double tn = tnorm[cc];
            pr = tn > 0.0 ? proj_in[(int64_t)cc * P + k] / tn : 0.0;
        }
        double acc = 0.0;
        for (int r = 0; r < trips; ++r) {
            const int32_t at = e0 + r * 2 * G;
            double v[2 * G];
            float wu[2 * G];
#pragma unroll
            for (int u = 0; u < 2 * G; ++u) {
                const int32_t cu = __shfl_sync(kAll, col[u / G], base + u % G);
                wu[u] = __shfl_sync(kAll, w[u / G], base + u % G);
                v[u] = at + u < e1 && k < P ? __ldg(&Vin[(int64_t)cu * P + k]) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int32_t nx = at + 2 * G + q * G + k;
                col[q] = nx < e1 ? __ldg(&indices[nx]) : 0;
                w[q] = nx < e1 ? __ldg(&data[nx]) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 2 * G; ++u)
                if (at + u < e1) acc += (double)wu[u] * v[u];
        }
        double out = 0.0;
        if (mine) {
            const double t = trivial_of(sdi);
            const double z = 0.5 * (y + (double)sdi * acc) - t * pr;
            out = (z - c * y) * s;
            if (ss != 0.0) out -= ss * xo;
            Yout[i * P + k] = out;
            Vout[i * P + k] = (double)sdi * out;
            cs.add((t + t * (double)du[i]) * out, cc, proj_out, P, k);
        }
        if constexpr (GRAM) {
#pragma unroll
            for (int a = 0; a < P; ++a) h[a] += __shfl_sync(kAll, y, base + a) * out;
        }
    }
    flush_component<P, G>(cs, proj_out, k, red);
    if constexpr (GRAM) {
#pragma unroll
        for (int a = 0; a < P; ++a) {
            const double t = column_block_sum<G>(h[a], red);
            if (threadIdx.x < P) part[((size_t)blockIdx.x * P + a) * P + threadIdx.x] = t;
        }
        sum_partials<P * P>(part, counter, gram);
    }
}

// tnorm[c] = the component's sum of t_i^2
__global__ void __launch_bounds__(kSpecThreads) trivial_norm_kernel(const float* __restrict__ sd,
                                                                    const int32_t* __restrict__ comp, int64_t n,
                                                                    double* __restrict__ tnorm) {
    __shared__ double red[kSpecThreads / 32][1];
    ComponentSum cs;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double t = trivial_of(sd[i]);
        cs.add(t * t, comp[i], tnorm, 1, 0);
    }
    flush_component<1, 1>(cs, tnorm, 0, red);
}

// u = M^T t: u_j = (t_j + sd_j sum_i a_ij sd_i t_i) / 2, by one warp per row; `u` holds t / 2 before. *open: an edge joins
// two components, for which the projections have no such weights.
__global__ void __launch_bounds__(kSpecThreads) half_trivial_kernel(const float* __restrict__ sd, int64_t n, double* __restrict__ u) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        u[i] = 0.5 * trivial_of(sd[i]);
}
__global__ void __launch_bounds__(kSpecThreads) adjoint_kernel(const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                                               const float* __restrict__ data, const float* __restrict__ sd,
                                                               const int32_t* __restrict__ comp, int64_t n,
                                                               int n_comp, double* __restrict__ u, int* __restrict__ open) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    bool crosses = false;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const double st = (double)sd[i] * trivial_of(sd[i]);
        if (st == 0.0) continue;
        const int c = comp[i];
        const int32_t e1 = indptr[i + 1];
        for (int32_t e = indptr[i] + lane; e < e1; e += 32) {
            const int32_t j = indices[e];
            const double x = 0.5 * (double)sd[j] * ((double)data[e] * st);
            if (x == 0.0) continue;
            if (n_comp == 1 || comp[j] == c) atomicAdd(&u[j], x);
            else crosses = true;
        }
    }
    if (crosses) *open = 1;
}
// u / t - 1 as it is held, *open where that is no small number
__global__ void __launch_bounds__(kSpecThreads) ratio_kernel(const float* __restrict__ sd, const double* __restrict__ u, int64_t n,
                                                             float* __restrict__ du, int* __restrict__ open) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double t = trivial_of(sd[i]);
        const double r = t > 0.0 ? u[i] / t - 1.0 : (u[i] == 0.0 ? 0.0 : INFINITY);
        du[i] = (float)r;
        if (!(fabs(r) < 1e-4)) *open = 1;
    }
}

template <int P>
struct Coef {
    double v[P * P];
};

// the sums of P columns, one thread per row
template <int P>
__device__ __forceinline__ void flush_rows(ComponentSum (&cs)[P], double* __restrict__ proj, double (*red)[1]) {
    __shared__ int any;
    if (threadIdx.x == 0) any = -1;
    __syncthreads();
    if (cs[0].comp >= 0) any = cs[0].comp;
    __syncthreads();
    const int c = any;
    const bool one = __syncthreads_and(cs[0].comp < 0 || cs[0].comp == c) != 0;
#pragma unroll
    for (int k = 0; k < P; ++k) {
        if (one) {
            const double t = column_block_sum<1>(cs[k].comp >= 0 ? cs[k].sum : 0.0, red);
            if (threadIdx.x == 0 && c >= 0) atomicAdd(&proj[(int64_t)c * P + k], t);
        } else if (cs[k].comp >= 0) {
            atomicAdd(&proj[(int64_t)cs[k].comp * P + k], cs[k].sum);
        }
    }
}

// The rest of a step whose product Z = M Yin stands by itself: Yout = (Z deflated - c Yin) s - ss X, with proj_in the
// per-component sums of t Z; the other outputs as step_kernel's (proj_out those of t Yout).
template <int P, bool GRAM>
__global__ void __launch_bounds__(kSpecThreads) finish_kernel(const float* __restrict__ sd, const int32_t* __restrict__ comp,
                                                              const double* __restrict__ tnorm, int64_t n,
                                                              const double* __restrict__ Z, const double* __restrict__ Yin,
                                                              const double* X, double* Yout, double* __restrict__ Vout,
                                                              double c, double s, double ss, const double* __restrict__ proj_in,
                                                              double* __restrict__ proj_out, double* __restrict__ part,
                                                              unsigned* __restrict__ counter, double* __restrict__ gram) {
    __shared__ double red[kSpecThreads / 32][1];
    double acc[GRAM ? P * P : 1];
#pragma unroll
    for (int q = 0; q < (GRAM ? P * P : 1); ++q) acc[q] = 0.0;
    ComponentSum cs[P];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double sdi = (double)sd[i], t = trivial_of(sd[i]);
        const int cc = comp[i];
        const double tn = tnorm[cc];
        double y[P], out[P];
#pragma unroll
        for (int k = 0; k < P; ++k) {
            y[k] = Yin[i * P + k];
            const double z = Z[i * P + k] - t * (tn > 0.0 ? proj_in[(int64_t)cc * P + k] / tn : 0.0);
            out[k] = (z - c * y[k]) * s;
            if (ss != 0.0) out[k] -= ss * X[i * P + k];
            Yout[i * P + k] = out[k];
            Vout[i * P + k] = sdi * out[k];
            cs[k].add(t * out[k], cc, proj_out, P, k);
        }
        if constexpr (GRAM) {
#pragma unroll
            for (int a = 0; a < P; ++a)
#pragma unroll
                for (int q = 0; q < P; ++q) acc[a * P + q] += y[a] * out[q];
        }
    }
    flush_rows<P>(cs, proj_out, red);
    if constexpr (GRAM) {
#pragma unroll
        for (int q = 0; q < P * P; ++q) {
            const double t = column_block_sum<1>(acc[q], red);
            if (threadIdx.x == 0) part[(size_t)blockIdx.x * P * P + q] = t;
        }
        sum_partials<P * P>(part, counter, gram);
    }
}

// The rows of a P-column block, one thread per row (compile-time switches):
//  WIDEN    X from the caller's float block
//  DEFLATE  X -= t proj_in / tnorm
//  APPLY    X <- X T (column c = sum_k X_k T[k][c])
//  GRAM     gram = X^T X of what was written
//  SUMS     V = D^-1/2 X and proj_out = per-component sums of t (1 + du) X
//  RESID    resid[c] = sum of ((Z T)_ic - theta_c X_ic)^2
constexpr int kWiden = 1, kDeflate = 2, kApply = 4, kGram = 8, kSums = 16, kResid = 32;

template <int P, int USE>
__global__ void __launch_bounds__(kSpecThreads) rows_kernel(const float* __restrict__ in, double* __restrict__ X,
                                                            const double* __restrict__ Z, int64_t n, Coef<P> T, Coef<P> theta,
                                                            const float* __restrict__ sd, const int32_t* __restrict__ comp,
                                                            const double* __restrict__ tnorm, const float* __restrict__ du,
                                                            const double* __restrict__ proj_in, double* __restrict__ V,
                                                            double* __restrict__ proj_out, double* __restrict__ part,
                                                            unsigned* __restrict__ counter, double* __restrict__ out) {
    constexpr int Q = (USE & kGram) ? P * P : ((USE & kResid) ? P : 1);
    __shared__ double red[kSpecThreads / 32][1];
    double acc[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) acc[q] = 0.0;
    ComponentSum cs[(USE & kSums) ? P : 1];
    int last = -1;          // the component whose projection coefficients are at hand
    double pr[(USE & kDeflate) ? P : 1];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double x[P], z[P];
#pragma unroll
        for (int k = 0; k < P; ++k) x[k] = (USE & kWiden) ? (double)in[i * P + k] : X[i * P + k];
        const float sdi = (USE & (kDeflate | kSums)) ? sd[i] : 0.f;
        const double t = trivial_of(sdi);
        const int c = (USE & (kDeflate | kSums)) ? comp[i] : 0;
        if constexpr ((USE & kDeflate) != 0) {
            if (c != last) {
                last = c;
                const double tn = tnorm[c];
#pragma unroll
                for (int k = 0; k < P; ++k) pr[k] = tn > 0.0 ? proj_in[(int64_t)c * P + k] / tn : 0.0;
            }
#pragma unroll
            for (int k = 0; k < P; ++k) x[k] -= t * pr[k];
        }
        if constexpr ((USE & kApply) != 0) {
            double y[P];
#pragma unroll
            for (int a = 0; a < P; ++a) {
                double sum = 0.0;
#pragma unroll
                for (int k = 0; k < P; ++k) sum += x[k] * T.v[k * P + a];
                y[a] = sum;
            }
#pragma unroll
            for (int k = 0; k < P; ++k) x[k] = y[k];
        }
        if constexpr ((USE & kResid) != 0) {
#pragma unroll
            for (int k = 0; k < P; ++k) z[k] = Z[i * P + k];
#pragma unroll
            for (int a = 0; a < P; ++a) {
                double sum = 0.0;
#pragma unroll
                for (int k = 0; k < P; ++k) sum += z[k] * T.v[k * P + a];
                const double d = sum - theta.v[a] * x[a];
                acc[a] += d * d;
            }
        }
#pragma unroll
        for (int k = 0; k < P; ++k) X[i * P + k] = x[k];
        if constexpr ((USE & kSums) != 0) {
            const double ws = t + t * (double)du[i];
#pragma unroll
            for (int k = 0; k < P; ++k) {
                if (V) V[i * P + k] = (double)sdi * x[k];
                cs[k].add(ws * x[k], c, proj_out, P, k);
            }
        }
        if constexpr ((USE & kGram) != 0) {
#pragma unroll
            for (int r = 0; r < P; ++r)
#pragma unroll
                for (int q = 0; q < P; ++q) acc[r * P + q] += x[r] * x[q];
        }
    }
    if constexpr ((USE & kSums) != 0) flush_rows<P>(cs, proj_out, red);
    if constexpr ((USE & (kGram | kResid)) != 0) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double t = column_block_sum<1>(acc[q], red);
            if (threadIdx.x == 0) part[(size_t)blockIdx.x * Q + q] = t;
        }
        sum_partials<Q>(part, counter, out);
    }
}

// column k of X: X_k <- (X_k - sum_{j < k} coef_j X_j) * scale
template <int P>
__global__ void __launch_bounds__(kSpecThreads) column_update_kernel(double* __restrict__ X, int64_t n, int k,
                                                                     Coef<P> coef, double scale) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double x = X[i * P + k];
        for (int j = 0; j < k; ++j) x -= coef.v[j] * X[i * P + j];
        X[i * P + k] = x * scale;
    }
}

__global__ void narrow_kernel(const double* __restrict__ in, float* __restrict__ out, int64_t count) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

// the smallest and the largest component label
__global__ void label_range_kernel(const int32_t* __restrict__ comp, int64_t n, int32_t* __restrict__ range) {
    int32_t lo = INT32_MAX, hi = INT32_MIN;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        lo = min(lo, comp[i]);
        hi = max(hi, comp[i]);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) { atomicMin(&range[0], lo); atomicMax(&range[1], hi); }
}

// the solver for a block of P columns; the steps and the stopping rule of src/spectral.cpp:172-238
template <int P>
struct Solver {
    const int32_t* indptr; const int32_t* indices; const float* data; const float* sd; const int32_t* comp;
    int64_t n; int64_t n_proj; int blocks; int sblocks; cudaStream_t s;
    double* proj[3]; int at = 0;          // per-component sums of t X: proj[at] those of the current block
    const double* tnorm; double* part; unsigned* counter; double* sums; double* host;
    const float* du; int open = 0;        // u / t - 1, then n zeros; u is no such thing (read with the first sums)
    const double* no_norm; double* Z;     // zeros in the place of tnorm; the product of a step in two launches

    double* now() { return proj[at]; }
    double* next() { return proj[(at + 1) % 3]; }
    double* after() { return proj[(at + 2) % 3]; }

    // waits for `count` sums of the last kernel
    const double* read(int count) {
        MGB_CUDA(cudaMemcpyAsync(host, sums, sizeof(double) * (size_t)count, cudaMemcpyDeviceToHost, s));
        MGB_CUDA(cudaStreamSynchronize(s));
        return host;
    }
    // the p x p sums, with the open flag behind them
    const double* read_flagged() {
        const double* h = read(P * P + 1);
        open = reinterpret_cast<const int*>(h + P * P)[1];
        return h;
    }
    template <int USE>
    void rows(double* X, const double* Z, const Coef<P>& T, const Coef<P>& theta, double* V, const float* in = nullptr) {
        const float* w = in ? du + n : du;   // the caller's block is deflated next, the others multiplied
        if (USE & kSums) MGB_CUDA(cudaMemsetAsync(next(), 0, sizeof(double) * (size_t)n_proj, s));
        rows_kernel<P, USE><<<blocks, kSpecThreads, 0, s>>>(in, X, Z, n, T, theta, sd, comp, tnorm, w, now(), V, next(), part,
                                                           counter, sums);
        MGB_LAUNCH_CHECK();
        if (USE & kSums) at = (at + 1) % 3;
    }
    // Yout = ((M Yin deflated) - c Yin) s - ss X; proj moves on (the next target was zeroed by the step before, or here);
    // last: Yout is deflated next, not multiplied
    template <bool GRAM>
    void step(const double* Yin, const double* Vin, const double* X, double* Yout, double* Vout, double c, double sc,
              double ss, bool clear, bool last) {
        if (open) {
            MGB_CUDA(cudaMemsetAsync(next(), 0, sizeof(double) * (size_t)n_proj, s));
            step_kernel<P, false><<<sblocks, kSpecThreads, 0, s>>>(indptr, indices, data, sd, comp, no_norm, n, du + n, n_proj, Yin, Vin,
                                                                  nullptr, Z, Vout, 0.0, 1.0, 0.0, now(), next(), after(), part,
                                                                  counter, sums);
            MGB_LAUNCH_CHECK();
            finish_kernel<P, GRAM><<<blocks, kSpecThreads, 0, s>>>(sd, comp, tnorm, n, Z, Yin, X, Yout, Vout, c, sc, ss, next(),
                                                                   after(), part, counter, sums);
            MGB_LAUNCH_CHECK();
            at = (at + 2) % 3;
            return;
        }
        if (clear) MGB_CUDA(cudaMemsetAsync(next(), 0, sizeof(double) * (size_t)n_proj, s));
        step_kernel<P, GRAM><<<sblocks, kSpecThreads, 0, s>>>(indptr, indices, data, sd, comp, tnorm, n, last ? du + n : du, n_proj, Yin, Vin, X,
                                                             Yout, Vout, c, sc, ss, now(), next(), after(), part, counter, sums);
        MGB_LAUNCH_CHECK();
        at = (at + 1) % 3;
    }

    // R^-1 for X^T X = R^T R (R upper triangular with a positive diagonal); false where a pivot is too small
    static bool inverse_factor(const double* Gm, Coef<P>& T) {
        double R[P][P] = {};
        for (int j = 0; j < P; ++j) {
            for (int i = 0; i <= j; ++i) {
                double v = Gm[i * P + j];
                for (int k = 0; k < i; ++k) v -= R[k][i] * R[k][j];
                if (i < j) R[i][j] = v / R[i][i];
                else {
                    if (!(v > 1e-10 * Gm[j * P + j]) || !(v > 1e-300)) return false;
                    R[j][j] = std::sqrt(v);
                }
            }
        }
        for (int q = 0; q < P * P; ++q) T.v[q] = 0.0;
        for (int j = 0; j < P; ++j) {
            T.v[j * P + j] = 1.0 / R[j][j];
            for (int i = j - 1; i >= 0; --i) {
                double v = 0.0;
                for (int k = i + 1; k <= j; ++k) v += R[i][k] * T.v[k * P + j];
                T.v[i * P + j] = -v / R[i][i];
            }
        }
        return true;
    }
    static Coef<P> identity() {
        Coef<P> I{};
        for (int k = 0; k < P; ++k) I.v[k * P + k] = 1.0;
        return I;
    }
    // X deflated and its columns orthonormalised, each against the ones before it, twice over (the reference's two
    // passes of Gram-Schmidt); V = D^-1/2 X and the per-component sums of the result
    void orthonormalize(double* X, double* V) {
        rows<kDeflate | kGram>(X, nullptr, Coef<P>{}, Coef<P>{}, nullptr);
        Coef<P> T;
        if (inverse_factor(read_flagged(), T)) {
            rows<kApply | kGram>(X, nullptr, T, Coef<P>{}, nullptr);
            if (inverse_factor(read(P * P), T)) {
                rows<kApply | kSums>(X, nullptr, T, Coef<P>{}, V);
                return;
            }
        }
        columns(X);
        rows<kApply | kSums>(X, nullptr, identity(), Coef<P>{}, V);
    }
    // column by column: the projections of a column on the earlier ones taken together (classical Gram-Schmidt, the
    // second pass restoring the orthogonality the first leaves), then its norm; a column of norm 0 stays 0
    void columns(double* X) {
        for (int pass = 0; pass < 2; ++pass)
            for (int k = 0; k < P; ++k) {
                Coef<P> c{};
                if (k > 0) {
                    rows<kGram>(X, nullptr, Coef<P>{}, Coef<P>{}, nullptr);
                    const double* Gm = read(P * P);
                    for (int j = 0; j < k; ++j) c.v[j] = Gm[(size_t)k * P + j];
                    column_update_kernel<P><<<blocks, kSpecThreads, 0, s>>>(X, n, k, c, 1.0);
                    MGB_LAUNCH_CHECK();
                }
                rows<kGram>(X, nullptr, Coef<P>{}, Coef<P>{}, nullptr);
                const double nrm = read(P * P)[(size_t)k * P + k];
                const double inv = nrm > 1e-300 ? 1.0 / std::sqrt(nrm) : 0.0;
                column_update_kernel<P><<<blocks, kSpecThreads, 0, s>>>(X, n, k, Coef<P>{}, inv);
                MGB_LAUNCH_CHECK();
            }
    }
    // Rayleigh-Ritz: Z = M X deflated, H = X^T Z (its upper triangle mirrored), H = V diag(theta) V^T, X and Z
    // rotated by V; returns the largest residual norm |Z_c - theta_c X_c| over the wanted columns. Vx: D^-1/2 X in and
    // out, Vz scratch.
    double rayleigh_ritz(double* X, double* Vx, double* Z, double* Vz, int n_wanted, std::vector<double>& theta) {
        step<true>(X, Vx, nullptr, Z, Vz, 0.0, 1.0, 0.0, true, true);
        const double* h = read(P * P);
        std::vector<double> H(h, h + P * P);
        for (int a = 0; a < P; ++a)
            for (int b = a + 1; b < P; ++b) H[(size_t)b * P + a] = H[(size_t)a * P + b];
        std::vector<double> V;
        symmetric_eigen(H, P, theta, V);
        Coef<P> v{}, th{};
        for (int q = 0; q < P * P; ++q) v.v[q] = V[q];
        for (int c = 0; c < P; ++c) th.v[c] = theta[c];
        rows<kApply | kResid | kSums>(X, Z, v, th, Vx);
        const double* r = read(P);
        double worst = 0.0;
        for (int c = 0; c < n_wanted; ++c) worst = std::max(worst, std::sqrt(r[c]));
        return worst;
    }

    void run(float* Xout, int n_wanted, int degree, int max_iter, double tol, SpecWork& w) {
        const int64_t cnt = n * P;
        const size_t bytes = sizeof(double) * (size_t)cnt;
        double* X = static_cast<double*>(w.X.ensure(bytes));
        double* Y = static_cast<double*>(w.Y.ensure(bytes));
        double* Vx = static_cast<double*>(w.Z.ensure(bytes));
        double* Vy = static_cast<double*>(w.Ynew.ensure(bytes));
        rows<kWiden | kSums>(X, nullptr, Coef<P>{}, Coef<P>{}, nullptr, Xout);
        orthonormalize(X, Vx);   // (waits for the stream)
        if (open) Z = static_cast<double*>(w.M.ensure(bytes));
        std::vector<double> theta;
        double res = rayleigh_ritz(X, Vx, Y, Vy, n_wanted, theta);
        double prev_sum = -1.0;
        for (int it = 0; it < max_iter; ++it) {
            // stop when the residual is small against the gap after the wanted Ritz values (floored at 1e-3), or
            // when the wanted Ritz values no longer move (src/spectral.cpp:196-203)
            const double gap = std::max(theta[n_wanted - 1] - theta[n_wanted], 1e-3);
            double sum = 0.0;
            for (int c = 0; c < n_wanted; ++c) sum += theta[c];
            const bool stagnant = prev_sum >= 0 && std::fabs(sum - prev_sum) < 1e-9 * (double)n_wanted;
            if (res < tol * gap || res < 1e-9 || stagnant) break;
            prev_sum = sum;
            // the Chebyshev filter damping [0, alpha] (the scaled three-term recurrence of Zhou and Saad,
            // src/spectral.cpp:205-231); X and Y hold the previous iterate and the current one in turn
            double alpha = theta[P - 1];
            alpha = std::min(alpha, theta[n_wanted - 1] - 0.5 * gap);
            alpha = std::max(alpha, 1e-3);
            const double a0 = std::min(1.0, theta[0] + 1e-9);
            const double e = 0.5 * alpha, cc = 0.5 * alpha;
            const double sigma1 = e / (a0 - cc);
            double sigma = sigma1;
            step<false>(X, Vx, nullptr, Y, Vy, cc, sigma1 / e, 0.0, true, false);
            for (int k = 2; k <= degree; ++k) {
                const double sigma_new = 1.0 / (2.0 / sigma1 - sigma);
                step<false>(Y, Vy, X, X, Vx, cc, 2.0 * sigma_new / e, sigma * sigma_new, false, k == degree);
                std::swap(X, Y);
                std::swap(Vx, Vy);
                sigma = sigma_new;
            }
            std::swap(X, Y);
            std::swap(Vx, Vy);
            orthonormalize(X, Vx);
            res = rayleigh_ritz(X, Vx, Y, Vy, n_wanted, theta);
        }
        narrow_kernel<<<row_blocks(cnt), kSpecThreads, 0, s>>>(X, Xout, cnt);
        MGB_LAUNCH_CHECK();
        MGB_CUDA(cudaStreamSynchronize(s));
    }
};

template <int P>
void run_solver(const int32_t* indptr, const int32_t* indices, const float* data, int64_t n, const float* sd,
                const int32_t* comp, int n_comp, float* X, int n_wanted, int degree, int max_iter, double tol,
                SpecWork& w, cudaStream_t s) {
    Solver<P> sv;
    sv.indptr = indptr; sv.indices = indices; sv.data = data; sv.sd = sd; sv.comp = comp;
    sv.n = n; sv.n_proj = (int64_t)n_comp * P; sv.s = s;
    sv.blocks = spec_blocks(n);
    sv.sblocks = (int)std::max<int64_t>(1, std::min<int64_t>((n * kLanes<P> + kSpecThreads - 1) / kSpecThreads,
                                                             (int64_t)kStepBlocks * kNumSMs));
    double* proj = static_cast<double*>(w.proj.ensure(sizeof(double) * 3 * (size_t)sv.n_proj));
    for (int q = 0; q < 3; ++q) sv.proj[q] = proj + q * sv.n_proj;
    double* tn = static_cast<double*>(w.tnorm.ensure(2 * sizeof(double) * (size_t)n_comp));
    sv.no_norm = tn + n_comp;
    // the block partials, the sums and the last-block counter
    const size_t parts = (size_t)std::max(sv.blocks, sv.sblocks) * P * P;
    sv.part = static_cast<double*>(w.part.ensure(sizeof(double) * (parts + P * P + 1)));
    sv.sums = sv.part + parts;
    sv.counter = reinterpret_cast<unsigned*>(sv.sums + P * P);   // and the open flag
    int* open = reinterpret_cast<int*>(sv.counter) + 1;
    double host[P * P + 1];
    sv.host = host;
    MGB_CUDA(cudaMemsetAsync(sv.counter, 0, sizeof(double), s));
    MGB_CUDA(cudaMemsetAsync(tn, 0, 2 * sizeof(double) * (size_t)n_comp, s));
    trivial_norm_kernel<<<sv.blocks, kSpecThreads, 0, s>>>(sd, comp, n, tn);
    MGB_LAUNCH_CHECK();
    sv.tnorm = tn;
    double* u = static_cast<double*>(w.u.ensure((sizeof(double) + 2 * sizeof(float)) * (size_t)n));
    float* du = reinterpret_cast<float*>(u + n);   // n ratios, n zeros (sums of t X)
    MGB_CUDA(cudaMemsetAsync(du + n, 0, sizeof(float) * (size_t)n, s));
    half_trivial_kernel<<<row_blocks(n), kSpecThreads, 0, s>>>(sd, n, u);
    MGB_LAUNCH_CHECK();
    adjoint_kernel<<<row_blocks(n * 32), kSpecThreads, 0, s>>>(indptr, indices, data, sd, comp, n, n_comp, u, open);
    MGB_LAUNCH_CHECK();
    ratio_kernel<<<row_blocks(n), kSpecThreads, 0, s>>>(sd, u, n, du, open);
    MGB_LAUNCH_CHECK();
    sv.du = du;
    sv.run(X, n_wanted, degree, max_iter, tol, w);
}

}  // namespace

// cyclic Jacobi rotations (Golub and Van Loan, Matrix Computations, section 8.5): each sweep zeroes the off-diagonal
// entries (i, j), i < j, in row order with the rotation whose tangent is the smaller root of
// t^2 + 2 theta t - 1 = 0, theta = (a_jj - a_ii) / (2 a_ij); sweeps stop once the squared off-diagonal sum is
// below 1e-22, as the reference's solver stops (src/spectral.cpp:87-123)
void symmetric_eigen(std::vector<double> A, int p, std::vector<double>& vals, std::vector<double>& V) {
    V.assign((size_t)p * p, 0.0);
    for (int i = 0; i < p; ++i) V[(size_t)i * p + i] = 1.0;
    auto at = [&](int r, int c) -> double& { return A[(size_t)r * p + c]; };
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0;
        for (int i = 0; i < p; ++i)
            for (int j = i + 1; j < p; ++j) off += at(i, j) * at(i, j);
        if (off < 1e-22) break;
        for (int i = 0; i < p; ++i)
            for (int j = i + 1; j < p; ++j) {
                const double aij = at(i, j);
                if (std::fabs(aij) < 1e-300) continue;
                const double theta = (at(j, j) - at(i, i)) / (2.0 * aij);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
                const double c = 1.0 / std::sqrt(t * t + 1.0), sn = t * c;
                for (int r = 0; r < p; ++r) {   // A <- A J (columns i and j)
                    const double x = at(r, i), y = at(r, j);
                    at(r, i) = c * x - sn * y;
                    at(r, j) = sn * x + c * y;
                }
                for (int r = 0; r < p; ++r) {   // A <- J^T A (rows i and j)
                    const double x = at(i, r), y = at(j, r);
                    at(i, r) = c * x - sn * y;
                    at(j, r) = sn * x + c * y;
                }
                for (int r = 0; r < p; ++r) {   // V <- V J
                    const double x = V[(size_t)r * p + i], y = V[(size_t)r * p + j];
                    V[(size_t)r * p + i] = c * x - sn * y;
                    V[(size_t)r * p + j] = sn * x + c * y;
                }
            }
    }
    std::vector<int> order(p);
    for (int i = 0; i < p; ++i) order[i] = i;
    std::vector<double> d(p);
    for (int i = 0; i < p; ++i) d[i] = at(i, i);
    std::sort(order.begin(), order.end(), [&](int a, int b) { return d[a] > d[b]; });
    vals.resize(p);
    std::vector<double> W((size_t)p * p);
    for (int c = 0; c < p; ++c) {
        vals[c] = d[order[c]];
        for (int r = 0; r < p; ++r) W[(size_t)r * p + c] = V[(size_t)r * p + order[c]];
    }
    V.swap(W);
}

void label_range_dev(const int32_t* comp, int64_t n, int32_t range[2], SpecWork& w, cudaStream_t s) {
    int32_t* d = static_cast<int32_t*>(w.tnorm.ensure(2 * sizeof(int32_t)));
    range[0] = INT32_MAX; range[1] = INT32_MIN;
    MGB_CUDA(cudaMemcpyAsync(d, range, 2 * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    label_range_kernel<<<spec_blocks(n), kSpecThreads, 0, s>>>(comp, n, d);
    MGB_LAUNCH_CHECK();
    MGB_CUDA(cudaMemcpyAsync(range, d, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    MGB_CUDA(cudaStreamSynchronize(s));
}

void chebyshev_eigenvectors_dev(const int32_t* indptr, const int32_t* indices, const float* data, int64_t n,
                                const float* sd, const int32_t* comp, int n_comp, float* X, int p, int n_wanted,
                                int degree, int max_iter, double tol, SpecWork& w, cudaStream_t s) {
    switch (p) {
        case 2: run_solver<2>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        case 3: run_solver<3>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        case 4: run_solver<4>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        case 5: run_solver<5>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        case 6: run_solver<6>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        case 7: run_solver<7>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        case 8: run_solver<8>(indptr, indices, data, n, sd, comp, n_comp, X, n_wanted, degree, max_iter, tol, w, s); break;
        default: throw Error(MG_ERR_NOT_SUPPORTED, "the device solver takes 2 to 8 columns");
    }
}

}  // namespace mgb
