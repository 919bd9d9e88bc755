// The fuzzy neighbour graph on the device.
//
// smooth_knn (src/graph.cpp:29-78): one thread per row. The row's distance sum (FP64) and rho, then the bisection
// of sigma until sum_j exp(-(d_j - rho) / sigma) is within 1e-5 of log2(n_neighbors) * bandwidth, in the
// reference's order of float operations; the floor of sigma at 1e-3 times the row's (or, for rho = 0, the whole
// array's) mean distance; then the memberships. exp is evaluated in FP64 and rounded to float: the reference's
// expf (glibc) agrees with that rounding on all but about 1e-4 of the float inputs, so a bisection decision
// differs only when a sum lands within an ulp of the target and sigma moves by about an ulp.
//
// Fuzzy union (magnet/knn.py:215-230): scipy's csr_matrix((vals, (rows, ind))) sums duplicate columns of a row and
// eliminate_zeros drops zero memberships; T = A^T; P = mix (A + T - A o T) + (1 - mix) (A o T), float32 as scipy
// evaluates it, zeros dropped, columns sorted. On the device:
//   1. each row of A sorted by column (stable; a bitonic network over 16 or 32 lanes for rows that fit), duplicates
//      summed in row order, zeros dropped, the column counts of T taken on the way;
//   2. T by a counting scatter: an exclusive scan of the counts, atomic slots, (row, value) as one 8-byte store;
//   3. per row, by a warp, A's and T's entries sorted together by column in the lanes' registers and equal columns
//      joined, counted, scanned into indptr, then written. Rows of more than 512 entries (hubs) have their T part
//      sorted by row first (a bitonic network in shared memory, heapsort past 512 entries) and are merged by a thread.
// Bound by the scattered stores and atomics of T and by issue in the sorts: 0.49 ms at 300k rows of 14 neighbours (rows
// 0.05, T 0.08, counting 0.13, writing 0.15) where one thread per row took 0.76 (rows 0.13, T 0.10, its sort 0.19,
// counting 0.05, writing 0.23), its reads and writes a row apart between threads.
// This file is compiled without FMA contraction (-fmad=false), so each product and sum rounds on its own as in
// the reference's x86-64 build and numpy.
#include "graph.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

namespace mgb {

namespace {

constexpr int kThreads = 256;

int grid_for(int64_t work, int per_block = kThreads) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((work + per_block - 1) / per_block, 16LL * kNumSMs));
}

__device__ __forceinline__ float exp_rounded(float x) { return (float)exp((double)x); }

// ---------------------------------------------------------------------------------------------- smooth_knn
__global__ void sigma_kernel(const float* __restrict__ D, int64_t n, int k, float target, int n_iter,
                             float* __restrict__ sigma, float* __restrict__ rho, double* __restrict__ part) {
    __shared__ double red[kThreads / 32];
    double block_sum = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float* d = D + i * k;
        double rowsum = 0.0;
        float r = 0.f;
        bool has = false;
        for (int j = 0; j < k; ++j) {
            rowsum += d[j];
            if (!has && d[j] > 0.f) { r = d[j]; has = true; }
        }
        block_sum += rowsum;
        float lo = 0.f, hi = INFINITY, mid = 1.f, sg = 1.f;
        bool done = false;
        for (int it = 0; it < n_iter; ++it) {
            float psum = 0.f;
            for (int j = 0; j < k; ++j) {
                const float dmr = d[j] - r;
                psum += dmr > 0.f ? exp_rounded(-dmr / mid) : 1.f;
            }
            if (fabsf(psum - target) < 1e-5f) { sg = mid; done = true; break; }
            if (psum > target) { hi = mid; mid = (lo + hi) * 0.5f; }
            else { lo = mid; mid = isinf(hi) ? mid * 2.f : (lo + hi) * 0.5f; }
        }
        if (!done) sg = mid;
        const float mean_row = (float)(rowsum / k);
        if (r > 0.f) sg = fmaxf(sg, 1e-3f * mean_row);
        sigma[i] = sg;
        rho[i] = r;
    }
    // the block's share of the whole array's distance sum
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) block_sum += __shfl_xor_sync(0xffffffffu, block_sum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = block_sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        part[blockIdx.x] = t;
    }
}

__global__ void membership_kernel(const float* __restrict__ D, int64_t n, int k, const float* __restrict__ sigma,
                                  const float* __restrict__ rho, const double* __restrict__ part, int n_part,
                                  float* __restrict__ out) {
    __shared__ float mean_all;
    if (threadIdx.x < 32) {   // one warp, a fixed order (one thread walking 1172 partials took most of the kernel's time)
        double t = 0.0;
        for (int b = threadIdx.x; b < n_part; b += 32) t += part[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) mean_all = (float)(t / (double)(n * k));
    }
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float r = rho[i];
        float sg = sigma[i];
        if (!(r > 0.f)) sg = fmaxf(sg, 1e-3f * mean_all);
        const float* d = D + i * k;
        float* o = out + i * k;
        for (int j = 0; j < k; ++j) {
            const float dmr = d[j] - r;
            o[j] = dmr > 0.f ? exp_rounded(-dmr / sg) : 1.f;
        }
    }
}

// ---------------------------------------------------------------------------------------------- fuzzy union
// step 1: row i of A into slot i * k: sorted by column (stable), duplicates summed in row order, zeros dropped; alen[i] =
// entries kept; tcnt[c] counts column c. Out-of-range columns set *bad (the row is left empty).
// Rows of up to L entries, L lanes per row, one entry per lane.
template <int L>
__global__ void __launch_bounds__(kThreads) a_lanes_kernel(const int32_t* __restrict__ ind, const float* __restrict__ vals,
                                                           int64_t n_rows, int k, int64_t n, int32_t* __restrict__ acol,
                                                           float* __restrict__ aval, int32_t* __restrict__ alen,
                                                           int32_t* __restrict__ tcnt, int* __restrict__ bad) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, l = lane % L, base = lane - l;
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x / L);
    const int64_t g0 = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / L;   // the warp's first group
    for (int64_t gw = g0; gw < n_rows; gw += groups) {
        const int64_t i = gw + lane / L;
        const bool row = i < n_rows, in = row && l < k;
        // key: the column, then the place in the row (a stable order); lanes past the row sort behind everything
        uint64_t key = ~0ull;
        float x = 0.f;
        bool wrong = false;
        if (in) {
            const int32_t col = ind[i * k + l];
            x = vals[i * k + l];
            wrong = col < 0 || col >= n;
            key = ((uint64_t)(uint32_t)col << 32) | (uint32_t)l;
        }
        const unsigned wrongs = (__ballot_sync(kAll, wrong) >> base) & (L == 32 ? kAll : ((1u << L) - 1u));
        if (wrong) atomicExch(bad, 1);
#pragma unroll
        for (int k2 = 2; k2 <= L; k2 <<= 1)
#pragma unroll
            for (int j = k2 >> 1; j > 0; j >>= 1) {
                const uint64_t ok = __shfl_xor_sync(kAll, key, j);
                const float ox = __shfl_xor_sync(kAll, x, j);
                const bool lower = (l & j) == 0, up = (l & k2) == 0;   // this lane keeps the smaller / larger one
                if ((ok < key) == (lower == up)) { key = ok; x = ox; }
            }
        const int32_t col = (int32_t)(key >> 32);
        const bool real = key != ~0ull && wrongs == 0;
        const int32_t before = __shfl_up_sync(kAll, col, 1);
        bool head = real && (l == 0 || before != col);
        const unsigned dup = __ballot_sync(kAll, real && !head);
        if (dup) {   // duplicates: each head adds the entries behind it, in row order
            const unsigned heads = __ballot_sync(kAll, head);
            for (int o = 1; o < L; ++o) {
                const float nx = __shfl_down_sync(kAll, x, o);
                const int at = lane + o;
                const bool mine = head && l + o < L && at < 32 && ((dup >> at) & 1u) &&
                                  (heads & ((2u << at) - 1u) & ~((2u << lane) - 1u)) == 0u;
                if (mine) x += nx;
            }
        }
        head = head && x != 0.f;
        const unsigned kept = (__ballot_sync(kAll, head) >> base) & (L == 32 ? kAll : ((1u << L) - 1u));
        if (head) {
            const int64_t at = i * k + __popc(kept & ((1u << l) - 1u));
            acol[at] = col;
            aval[at] = x;
            atomicAdd(&tcnt[col], 1);
        }
        if (row && l == 0) alen[i] = __popc(kept);
    }
}

// longer rows: one thread per row, insertion sort in place
__global__ void a_rows_kernel(const int32_t* __restrict__ ind, const float* __restrict__ vals, int64_t n_rows,
                              int k, int64_t n, int32_t* __restrict__ acol, float* __restrict__ aval,
                              int32_t* __restrict__ alen, int32_t* __restrict__ tcnt, int* __restrict__ bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_rows; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t* c = acol + i * k;
        float* v = aval + i * k;
        bool wrong = false;
        for (int j = 0; j < k; ++j) {
            const int32_t col = ind[i * k + j];
            if (col < 0 || col >= n) { wrong = true; break; }
            const float x = vals[i * k + j];
            int p = j;
            while (p > 0 && c[p - 1] > col) { c[p] = c[p - 1]; v[p] = v[p - 1]; --p; }
            c[p] = col; v[p] = x;
        }
        alen[i] = 0;
        if (wrong) { atomicExch(bad, 1); continue; }
        int m = 0;
        for (int j = 0; j < k;) {
            const int32_t col = c[j];
            float x = v[j];
            int e = j + 1;
            for (; e < k && c[e] == col; ++e) x += v[e];
            if (x != 0.f) { c[m] = col; v[m] = x; ++m; atomicAdd(&tcnt[col], 1); }
            j = e;
        }
        alen[i] = m;
    }
}

// step 2: entry (i, col) of A into T's row col, (row, value bits) in one store; 16 lanes per row of A
__global__ void __launch_bounds__(kThreads) t_fill_kernel(const int32_t* __restrict__ acol, const float* __restrict__ aval,
                                                          const int32_t* __restrict__ alen, int64_t n_rows, int k,
                                                          const int64_t* __restrict__ tptr, int32_t* __restrict__ tcur,
                                                          int2* __restrict__ t) {
    const int l = threadIdx.x & 15;
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x / 16);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 16; i < n_rows; i += groups) {
        const int len = alen[i];
        for (int j = l; j < len; j += 16) {
            const int32_t col = acol[i * k + j];
            const int64_t pos = tptr[col] + atomicAdd(&tcur[col], 1);
            t[pos] = make_int2((int32_t)i, __float_as_int(aval[i * k + j]));
        }
    }
}

__device__ void sift_down(int2* t, int64_t root, int64_t end) {
    while (2 * root + 1 < end) {
        int64_t child = 2 * root + 1;
        if (child + 1 < end && t[child + 1].x > t[child].x) ++child;
        if (t[root].x >= t[child].x) return;
        const int2 v = t[root]; t[root] = t[child]; t[child] = v;
        root = child;
    }
}

// step 3a: the T part of rows that a warp's registers do not hold (A and T entries > kWarpRow), sorted by row index
// (the keys of a row are distinct), one warp per row. Up to kSortMax entries: a bitonic network over the row padded to
// a power of two in the warp's own shared-memory region; longer rows (hub nodes chosen by very many): heapsort in
// place by the warp's first lane.
constexpr int kWarpRow = 512;
constexpr int kSortWarps = 8;
constexpr int kSortMax = 512;

__global__ void __launch_bounds__(32 * kSortWarps) t_sort_kernel(const int64_t* __restrict__ tptr, int64_t n,
                                                                 const int32_t* __restrict__ alen, int64_t n_rows,
                                                                 int2* __restrict__ t) {
    __shared__ int2 sh[kSortWarps][kSortMax];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int2* K = sh[wib];
    // each warp looks at 32 rows at once and sorts the long ones among them
    const int64_t warps = (int64_t)gridDim.x * kSortWarps;
    for (int64_t r0 = ((int64_t)blockIdx.x * kSortWarps + wib) * 32; r0 < n; r0 += warps * 32) {
        const int64_t mine = r0 + lane;
        const int64_t len = mine < n ? tptr[mine + 1] - tptr[mine] : 0;
        unsigned todo = __ballot_sync(0xffffffffu, len > 1 && len + (mine < n_rows ? alen[mine] : 0) > kWarpRow);
        while (todo) {
            const int64_t r = r0 + __ffs(todo) - 1;
            todo &= todo - 1u;
            int2* row = t + tptr[r];
            const int64_t m = tptr[r + 1] - tptr[r];
            if (m > kSortMax) {
                if (lane == 0) {
                    for (int64_t s0 = m / 2 - 1; s0 >= 0; --s0) sift_down(row, s0, m);
                    for (int64_t e = m - 1; e > 0; --e) {
                        const int2 v = row[0]; row[0] = row[e]; row[e] = v;
                        sift_down(row, 0, e);
                    }
                }
                __syncwarp();
                continue;
            }
            int P = 32;
            while (P < m) P <<= 1;
            for (int q = lane; q < P; q += 32) K[q] = q < m ? row[q] : make_int2(INT32_MAX, 0);
            __syncwarp();
            for (int k2 = 2; k2 <= P; k2 <<= 1) {
                for (int j = k2 >> 1; j > 0; j >>= 1) {
                    for (int q = lane; q < P; q += 32) {
                        const int u = q ^ j;
                        if (u > q) {
                            const bool ascending = (q & k2) == 0;
                            if ((K[q].x > K[u].x) == ascending) { const int2 v = K[q]; K[q] = K[u]; K[u] = v; }
                        }
                    }
                    __syncwarp();
                }
            }
            for (int q = lane; q < m; q += 32) row[q] = K[q];
            __syncwarp();
        }
    }
}

// P's entry from A's a and T's t (has_a / has_t: present); scipy's float32 order
__device__ __forceinline__ float union_value(bool has_a, float a, bool has_t, float t, float mix, float one_minus_mix) {
    if (has_a && has_t) {
        const float prod = a * t;
        const float d = (a + t) - prod;
        return d * mix + prod * one_minus_mix;
    }
    return (has_a ? a : t) * mix;
}

// step 3b: row i of the union from A's and T's rows i, one warp per row; counted, or written at uptr[i].
// R registers per lane: entries 32 c + lane, sorted ascending by key 2 column + (1 for T).
template <bool WRITE, int R>
__device__ __forceinline__ int union_row(const int32_t* __restrict__ ac, const float* __restrict__ av, int la,
                                         const int2* __restrict__ t, int lt, float mix, float one_minus_mix, int lane,
                                         int32_t* __restrict__ indices, float* __restrict__ data) {
    constexpr unsigned kAll = 0xffffffffu;
    uint32_t key[R];
    float x[R];
#pragma unroll
    for (int c = 0; c < R; ++c) {
        const int q = c * 32 + lane;
        key[c] = 0xffffffffu;   // behind every entry (a column is below 2^31 - 1)
        x[c] = 0.f;
        if (q < la) {
            key[c] = 2u * (uint32_t)ac[q];
            x[c] = av[q];
        } else if (q < la + lt) {
            const int2 e = t[q - la];
            key[c] = 2u * (uint32_t)e.x + 1u;
            x[c] = __int_as_float(e.y);
        }
    }
#pragma unroll
    for (int k2 = 2; k2 <= 32 * R; k2 <<= 1)
#pragma unroll
        for (int j = k2 >> 1; j > 0; j >>= 1) {
            if (j >= 32) {   // between a lane's registers
#pragma unroll
                for (int c = 0; c < R; ++c)
                    if (((c * 32) & j) == 0) {
                        const int d = c + j / 32;
                        const bool up = ((c * 32 + lane) & k2) == 0;
                        if ((key[c] > key[d]) == up) {
                            const uint32_t tk = key[c]; key[c] = key[d]; key[d] = tk;
                            const float tx = x[c]; x[c] = x[d]; x[d] = tx;
                        }
                    }
            } else {
#pragma unroll
                for (int c = 0; c < R; ++c) {
                    const uint32_t ok = __shfl_xor_sync(kAll, key[c], j);
                    const float ox = __shfl_xor_sync(kAll, x[c], j);
                    const bool lower = (lane & j) == 0, up = ((c * 32 + lane) & k2) == 0;
                    if ((ok < key[c]) == (lower == up)) { key[c] = ok; x[c] = ox; }
                }
            }
        }
    int count = 0;
#pragma unroll
    for (int c = 0; c < R; ++c) {
        // the entry after and the one before this one
        uint32_t nk = __shfl_down_sync(kAll, key[c], 1);
        float nx = __shfl_down_sync(kAll, x[c], 1);
        const uint32_t fk = c + 1 < R ? __shfl_sync(kAll, key[c + 1 < R ? c + 1 : c], 0) : 0xffffffffu;
        const float fx = c + 1 < R ? __shfl_sync(kAll, x[c + 1 < R ? c + 1 : c], 0) : 0.f;
        if (lane == 31) { nk = fk; nx = fx; }
        uint32_t pk = __shfl_up_sync(kAll, key[c], 1);
        const uint32_t lk = c > 0 ? __shfl_sync(kAll, key[c > 0 ? c - 1 : 0], 31) : 0xffffffffu;
        if (lane == 0) pk = lk;
        const bool real = key[c] != 0xffffffffu;
        const bool is_t = (key[c] & 1u) != 0u;
        const bool joined = real && is_t && pk == key[c] - 1u;   // T's half of a column that A has too
        const bool pair = real && !is_t && nk == key[c] + 1u;
        float v = 0.f;
        if (real && !joined) v = union_value(!is_t, x[c], pair || is_t, pair ? nx : x[c], mix, one_minus_mix);
        const bool keep = real && !joined && v != 0.f;
        const unsigned m = __ballot_sync(kAll, keep);
        if (WRITE && keep) {
            const int at = count + __popc(m & ((1u << lane) - 1u));
            indices[at] = (int32_t)(key[c] >> 1);
            data[at] = v;
        }
        count += __popc(m);
    }
    return count;
}

template <bool WRITE>
__global__ void __launch_bounds__(kThreads) union_kernel(const int32_t* __restrict__ acol, const float* __restrict__ aval,
                                                         const int32_t* __restrict__ alen, int64_t n_rows, int k,
                                                         const int64_t* __restrict__ tptr, const int2* __restrict__ t,
                                                         int64_t n, float mix, float one_minus_mix,
                                                         int32_t* __restrict__ ucnt, const int64_t* __restrict__ uptr,
                                                         int32_t* __restrict__ indices, float* __restrict__ data) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const int la = i < n_rows ? alen[i] : 0;
        const int32_t* ac = acol + i * k;
        const float* av = aval + i * k;
        const int64_t t0 = tptr[i], lt = tptr[i + 1] - t0;
        const int64_t out = WRITE ? uptr[i] : 0;
        int cnt = 0;
        if (la + lt <= 32) {
            cnt = union_row<WRITE, 1>(ac, av, la, t + t0, (int)lt, mix, one_minus_mix, lane, indices + out, data + out);
        } else if (la + lt <= 64) {
            cnt = union_row<WRITE, 2>(ac, av, la, t + t0, (int)lt, mix, one_minus_mix, lane, indices + out, data + out);
        } else if (la + lt <= 128) {
            cnt = union_row<WRITE, 4>(ac, av, la, t + t0, (int)lt, mix, one_minus_mix, lane, indices + out, data + out);
        } else if (la + lt <= 256) {
            cnt = union_row<WRITE, 8>(ac, av, la, t + t0, (int)lt, mix, one_minus_mix, lane, indices + out, data + out);
        } else if (la + lt <= kWarpRow) {
            cnt = union_row<WRITE, 16>(ac, av, la, t + t0, (int)lt, mix, one_minus_mix, lane, indices + out, data + out);
        } else {
            continue;   // union_long_kernel's
        }
        if (!WRITE && lane == 0) ucnt[i] = cnt;
    }
}

// the rows past kWarpRow entries, both parts sorted: one thread's merge per row
template <bool WRITE>
__global__ void union_long_kernel(const int32_t* __restrict__ acol, const float* __restrict__ aval,
                                  const int32_t* __restrict__ alen, int64_t n_rows, int k, const int64_t* __restrict__ tptr,
                                  const int2* __restrict__ t, int64_t n, float mix, float one_minus_mix,
                                  int32_t* __restrict__ ucnt, const int64_t* __restrict__ uptr,
                                  int32_t* __restrict__ indices, float* __restrict__ data) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int la = i < n_rows ? alen[i] : 0;
        int64_t ta = tptr[i];
        const int64_t te = tptr[i + 1];
        if (la + (te - ta) <= kWarpRow) continue;
        const int32_t* ac = acol + i * k;
        const float* av = aval + i * k;
        int64_t at = WRITE ? uptr[i] : 0;
        int ja = 0, cnt = 0;
        while (ja < la || ta < te) {
            const int32_t ca = ja < la ? ac[ja] : INT32_MAX;
            const int32_t ct = ta < te ? t[ta].x : INT32_MAX;
            const int32_t col = ca < ct ? ca : ct;
            const bool has_a = ca == col, has_t = ct == col;
            const float x = union_value(has_a, has_a ? av[ja] : 0.f, has_t, has_t ? __int_as_float(t[ta].y) : 0.f, mix,
                                        one_minus_mix);
            if (has_a) ++ja;
            if (has_t) ++ta;
            if (x != 0.f) {
                if (WRITE) { indices[at] = col; data[at] = x; ++at; }
                ++cnt;
            }
        }
        if (!WRITE) ucnt[i] = cnt;
    }
}

// ---------------------------------------------------------------------------------------------- scan
constexpr int kScanTile = 2048;   // elements per block in the first pass

// per tile: exclusive scan of in[] into out[] (int64) and the tile's total into sums[]
__global__ void __launch_bounds__(1024) scan_tiles_kernel(const int32_t* __restrict__ in, int64_t n,
                                                          int64_t* __restrict__ out, int64_t* __restrict__ sums) {
    __shared__ int64_t sh[1024];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    const int t = threadIdx.x;
    const int64_t i0 = base + 2 * t, i1 = i0 + 1;
    const int64_t x0 = i0 < n ? in[i0] : 0, x1 = i1 < n ? in[i1] : 0;
    sh[t] = x0 + x1;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {   // Hillis-Steele inclusive scan of the pair sums
        const int64_t v = t >= o ? sh[t - o] : 0;
        __syncthreads();
        sh[t] += v;
        __syncthreads();
    }
    const int64_t before = t > 0 ? sh[t - 1] : 0;
    if (i0 < n) out[i0] = before;
    if (i1 < n) out[i1] = before + x0;
    if (t == 1023) sums[blockIdx.x] = sh[1023];
}

// one block: exclusive scan of the tile totals (in place), then the grand total into out[n]
__global__ void __launch_bounds__(1024) scan_sums_kernel(int64_t* __restrict__ sums, int n_tiles,
                                                         int64_t* __restrict__ out, int64_t n) {
    __shared__ int64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < n_tiles; b0 += 1024) {
        __shared__ int64_t sh[1024];
        const int t = threadIdx.x;
        const int64_t x = b0 + t < n_tiles ? sums[b0 + t] : 0;
        sh[t] = x;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {
            const int64_t v = t >= o ? sh[t - o] : 0;
            __syncthreads();
            sh[t] += v;
            __syncthreads();
        }
        if (b0 + t < n_tiles) sums[b0 + t] = carry + sh[t] - x;
        __syncthreads();
        if (t == 0) carry += sh[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[n] = carry;
}

__global__ void scan_add_kernel(int64_t* __restrict__ out, int64_t n, const int64_t* __restrict__ sums) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] += sums[i / kScanTile];
}

// out[0..n] = exclusive scan of in[0..n) and the total
void exclusive_scan(const int32_t* in, int64_t n, int64_t* out, DevBuf& tmp, cudaStream_t s) {
    const int64_t tiles = std::max<int64_t>(1, (n + kScanTile - 1) / kScanTile);
    int64_t* sums = static_cast<int64_t*>(tmp.ensure(sizeof(int64_t) * tiles));
    if (n > 0) {
        scan_tiles_kernel<<<(unsigned)tiles, 1024, 0, s>>>(in, n, out, sums);
        MGB_LAUNCH_CHECK();
    } else {
        MGB_CUDA(cudaMemsetAsync(sums, 0, sizeof(int64_t), s));
    }
    scan_sums_kernel<<<1, 1024, 0, s>>>(sums, (int)tiles, out, n);
    MGB_LAUNCH_CHECK();
    if (n > 0) {
        scan_add_kernel<<<grid_for(n), kThreads, 0, s>>>(out, n, sums);
        MGB_LAUNCH_CHECK();
    }
}

__global__ void narrow_kernel(const int64_t* __restrict__ in, int64_t n, int32_t* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (int32_t)in[i];
}

// ------------------------------------------------------------------------------------------------ transform schedule
// The edge schedule of MAGNET.transform (magnet/__init__.py:907-912) for m new rows of k neighbours, one block:
// freq_i = min(1, s w_i) with s such that sum(freq) = samples_per_node * m (magnet/__init__.py:51-66), the edges with
// freq >= 1 / n_epochs kept in row order with head n_train + row, their neighbour as tail and eps = 1 / freq.
// The reference sorts the weights and walks the breakpoints of the piecewise-linear sum; here Newton's iteration on it
// does: s <- (target - k) / (sum of the unsaturated weights), k the weights saturated at s, from s = target / sum up.
// The sum of min(1, s w) is concave and piecewise linear, so the iterates rise to the root and stay on its segment once
// they reach it: k no longer grows, after 5 to 10 rounds (a bisection to the last ulp took about 60 for a request and
// 170 for a fit). Sums are FP64 reductions in a fixed order, so the result is the same from call to call; it differs
// from the host's sorted cumulative sum only by FP64 rounding.
constexpr int kSchedThreads = 1024;

__device__ __forceinline__ double block_sum_d(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
    return t;
}

__global__ void __launch_bounds__(kSchedThreads) transform_schedule_kernel(
    const float* __restrict__ w, const int64_t* __restrict__ ind, int64_t n, int k, int64_t n_train, double target,
    double min_freq, int32_t* __restrict__ head, int32_t* __restrict__ tail, float* __restrict__ eps,
    int64_t* __restrict__ n_kept) {
    __shared__ double red[kSchedThreads / 32];
    __shared__ int64_t scan[kSchedThreads / 32];
    __shared__ int64_t carry;
    // sum and positive count
    double sum = 0.0, npos = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = (double)w[i];
        sum += v;
        if (v > 0.0) npos += 1.0;
    }
    sum = block_sum_d(sum, red);
    npos = block_sum_d(npos, red);
    // s: all ones when n <= target (the reference returns ones, zero weights included); saturating every positive
    // weight when they are too few (the reference's s = 1 / max(w_min, 1e-300)); else the exact solution
    bool ones = (double)n <= target;
    double s = 0.0;
    if (!ones && npos <= target) {
        s = 1e300;
    } else if (!ones) {
        s = target / sum;
        double saturated = -1.0;
        for (int it = 0; it < 200; ++it) {
            double cnt = 0.0, rest = 0.0;
            for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
                const double v = (double)w[i];
                if (s * v > 1.0) cnt += 1.0; else rest += v;
            }
            cnt = block_sum_d(cnt, red);
            rest = block_sum_d(rest, red);
            if (cnt <= saturated || !(rest > 0.0)) break;
            saturated = cnt;
            s = (target - cnt) / rest;
        }
    }
    // the kept edges in row order: a block-wide exclusive scan of the keep flags, 1024 edges at a time
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t base = 0; base < n; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        double freq = 0.0;
        bool keep = false;
        if (i < n) {
            freq = ones ? 1.0 : fmin(1.0, s * (double)w[i]);
            keep = freq >= min_freq;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) scan[warp] = __popc(bal);
        __syncthreads();
        if (threadIdx.x == 0) {
            int64_t acc = 0;
            for (int j = 0; j < (int)(blockDim.x >> 5); ++j) { const int64_t t = scan[j]; scan[j] = acc; acc += t; }
            red[0] = (double)acc;   // this tile's count
        }
        __syncthreads();
        if (keep) {
            const int64_t pos = carry + scan[warp] + __popc(bal & ((1u << lane) - 1u));
            head[pos] = (int32_t)(n_train + i / k);
            tail[pos] = (int32_t)ind[i];
            eps[pos] = (float)(1.0 / freq);
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += (int64_t)red[0];
        __syncthreads();
    }
    if (threadIdx.x == 0) *n_kept = carry;
}

// ------------------------------------------------------------------------------------------------ fit schedule
// The solve of s for a fit's weights in rounds of one grid-wide pass each (the iteration above): the blocks' partial
// sums are added by the last block, which takes the step; rounds past the end of the iteration do nothing. A 300k-row
// fit's solve takes 13 launches (55 us) and one host round trip; the bisection took 176 of each (4 ms).
constexpr int kSchedBlocks = 4 * kNumSMs;

struct SchedState {
    double s, saturated;   // the iterate; the weights saturated at the one before
    int done, ones;        // the iteration has ended; all frequencies are 1
    unsigned counter, pad;
};

// FIRST: the sum and the positive count, which settle the special cases and the first iterate
template <bool FIRST>
__global__ void __launch_bounds__(kThreads) sched_round_kernel(const float* __restrict__ w, int64_t n, double target,
                                                               double2* __restrict__ part, SchedState* __restrict__ st) {
    __shared__ double2 red[kThreads / 32];
    __shared__ int is_last;
    const bool done = FIRST ? false : st->done != 0;   // written before this launch
    if (done) return;
    const double s = FIRST ? 0.0 : st->s;
    double a = 0.0, b = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = (double)w[i];
        if (FIRST) { a += v; if (v > 0.0) b += 1.0; }
        else if (s * v > 1.0) b += 1.0;
        else a += v;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) red[warp] = make_double2(a, b);
    __syncthreads();
    if (threadIdx.x == 0) {
        double2 t = make_double2(0.0, 0.0);
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { t.x += red[k].x; t.y += red[k].y; }
        part[blockIdx.x] = t;
        __threadfence();
        is_last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last || warp != 0) return;
    __threadfence();
    a = 0.0; b = 0.0;
    for (unsigned q = lane; q < gridDim.x; q += 32) { const double2 v = __ldcg(&part[q]); a += v.x; b += v.y; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane != 0) return;
    st->counter = 0u;
    if (FIRST) {
        // all ones when n <= target (zero weights included); every positive weight saturated when they are too few
        st->ones = (double)n <= target ? 1 : 0;
        st->done = st->ones || b <= target ? 1 : 0;
        st->s = st->done ? 1e300 : target / a;
        st->saturated = -1.0;
    } else if (b <= st->saturated || !(a > 0.0)) {
        st->done = 1;
    } else {
        st->saturated = b;
        st->s = (target - b) / a;
    }
}

__device__ __forceinline__ double sched_freq(double v, double s, bool ones) { return ones ? 1.0 : fmin(1.0, s * v); }

// one warp per row: its kept entries counted, or written in order from off[row] on
template <bool WRITE>
__global__ void __launch_bounds__(kThreads) sched_rows_kernel(const int32_t* __restrict__ indptr,
                                                              const int32_t* __restrict__ indices,
                                                              const float* __restrict__ w, int64_t n_rows,
                                                              const SchedState* __restrict__ st, double min_freq,
                                                              int32_t* __restrict__ cnt, const int64_t* __restrict__ off,
                                                              int32_t* __restrict__ head, int32_t* __restrict__ tail,
                                                              float* __restrict__ eps) {
    const int lane = threadIdx.x & 31;
    const double s = st->s;
    const bool ones = st->ones != 0;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += warps) {
        const int32_t e0 = indptr[r], e1 = indptr[r + 1];
        int64_t at = WRITE ? off[r] : 0;
        int total = 0;
        for (int32_t b = e0; b < e1; b += 32) {
            const int32_t e = b + lane;
            const double f = e < e1 ? sched_freq((double)w[e], s, ones) : 0.0;
            const bool keep = e < e1 && f >= min_freq;
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (WRITE && keep) {
                const int64_t pos = at + __popc(m & ((1u << lane) - 1u));
                head[pos] = (int32_t)r;
                tail[pos] = indices[e];
                eps[pos] = (float)(1.0 / f);
            }
            at += __popc(m);
            total += __popc(m);
        }
        if (!WRITE && lane == 0) cnt[r] = total;
    }
}

}  // namespace

void exclusive_scan_i32(const int32_t* in, int64_t n, int64_t* out, DevBuf& tmp, cudaStream_t s) {
    exclusive_scan(in, n, out, tmp, s);
}

void smooth_knn_dev(const float* dist, int64_t n_rows, int k, float target, int n_iter, float* out, GraphWork& w,
                    cudaStream_t s) {
    if (n_rows == 0 || k == 0) return;
    float* sigma = static_cast<float*>(w.sigma.ensure(sizeof(float) * n_rows));
    float* rho = static_cast<float*>(w.rho.ensure(sizeof(float) * n_rows));
    const int blocks = grid_for(n_rows);
    double* part = static_cast<double*>(w.part.ensure(sizeof(double) * blocks));
    sigma_kernel<<<blocks, kThreads, 0, s>>>(dist, n_rows, k, target, n_iter, sigma, rho, part);
    MGB_LAUNCH_CHECK();
    membership_kernel<<<blocks, kThreads, 0, s>>>(dist, n_rows, k, sigma, rho, part, blocks, out);
    MGB_LAUNCH_CHECK();
}

int64_t fuzzy_union_dev(const int32_t* ind, const float* vals, int64_t n_rows, int k, int64_t n, float mix,
                        float one_minus_mix, int32_t* indptr, int32_t* indices, float* data, int64_t cap,
                        GraphWork& w, cudaStream_t s) {
    const int64_t ek = std::max<int64_t>(n_rows * k, 1);
    int32_t* acol = static_cast<int32_t*>(w.acol.ensure(sizeof(int32_t) * ek));
    float* aval = static_cast<float*>(w.aval.ensure(sizeof(float) * ek));
    int32_t* alen = static_cast<int32_t*>(w.alen.ensure(sizeof(int32_t) * std::max<int64_t>(n_rows, 1)));
    int32_t* tcnt = static_cast<int32_t*>(w.tcnt.ensure(sizeof(int32_t) * std::max<int64_t>(n, 1)));
    int32_t* tcur = static_cast<int32_t*>(w.tcur.ensure(sizeof(int32_t) * std::max<int64_t>(n, 1)));
    int64_t* tptr = static_cast<int64_t*>(w.tptr.ensure(sizeof(int64_t) * (n + 1)));
    int2* t = static_cast<int2*>(w.trow.ensure(sizeof(int2) * ek));
    int32_t* ucnt = static_cast<int32_t*>(w.ucnt.ensure(sizeof(int32_t) * std::max<int64_t>(n, 1)));
    int* bad = static_cast<int*>(w.flag.ensure(sizeof(int)));
    int64_t* uptr = static_cast<int64_t*>(w.uptr.ensure(sizeof(int64_t) * (n + 1)));
    MGB_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s));
    MGB_CUDA(cudaMemsetAsync(tcnt, 0, sizeof(int32_t) * std::max<int64_t>(n, 1), s));
    MGB_CUDA(cudaMemsetAsync(tcur, 0, sizeof(int32_t) * std::max<int64_t>(n, 1), s));
    if (n_rows > 0 && k > 0) {
        // lanes per row while the row fits them: 16 (two rows a warp) or 32
        if (k <= 16) a_lanes_kernel<16><<<grid_for(n_rows * 16), kThreads, 0, s>>>(ind, vals, n_rows, k, n, acol, aval, alen, tcnt, bad);
        else if (k <= 32) a_lanes_kernel<32><<<grid_for(n_rows * 32), kThreads, 0, s>>>(ind, vals, n_rows, k, n, acol, aval, alen, tcnt, bad);
        else a_rows_kernel<<<grid_for(n_rows), kThreads, 0, s>>>(ind, vals, n_rows, k, n, acol, aval, alen, tcnt, bad);
        MGB_LAUNCH_CHECK();
        int h_bad = 0;
        MGB_CUDA(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
        MGB_CUDA(cudaStreamSynchronize(s));
        require(h_bad == 0, "neighbour index out of range");
    } else {
        MGB_CUDA(cudaMemsetAsync(alen, 0, sizeof(int32_t) * std::max<int64_t>(n_rows, 1), s));
    }
    exclusive_scan(tcnt, n, tptr, w.scan, s);
    if (n_rows > 0 && k > 0) {
        t_fill_kernel<<<grid_for(n_rows * 16), kThreads, 0, s>>>(acol, aval, alen, n_rows, k, tptr, tcur, t);
        MGB_LAUNCH_CHECK();
    }
    if (n > 0) {
        t_sort_kernel<<<(int)std::min<int64_t>((n + 32 * kSortWarps - 1) / (32 * kSortWarps), 8LL * kNumSMs),
                        32 * kSortWarps, 0, s>>>(tptr, n, alen, n_rows, t);
        MGB_LAUNCH_CHECK();
        union_kernel<false><<<grid_for(n * 32), kThreads, 0, s>>>(acol, aval, alen, n_rows, k, tptr, t, n, mix, one_minus_mix,
                                                                  ucnt, nullptr, nullptr, nullptr);
        MGB_LAUNCH_CHECK();
        union_long_kernel<false><<<grid_for(n), kThreads, 0, s>>>(acol, aval, alen, n_rows, k, tptr, t, n, mix, one_minus_mix,
                                                                  ucnt, nullptr, nullptr, nullptr);
        MGB_LAUNCH_CHECK();
    }
    exclusive_scan(ucnt, n, uptr, w.scan, s);
    int64_t nnz = 0;
    MGB_CUDA(cudaMemcpyAsync(&nnz, uptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MGB_CUDA(cudaStreamSynchronize(s));
    require(nnz <= cap, "output capacity too small for the union");
    require(nnz <= INT32_MAX, "the union has more than 2^31 - 1 entries");
    if (n > 0) {
        union_kernel<true><<<grid_for(n * 32), kThreads, 0, s>>>(acol, aval, alen, n_rows, k, tptr, t, n, mix, one_minus_mix,
                                                                 nullptr, uptr, indices, data);
        MGB_LAUNCH_CHECK();
        union_long_kernel<true><<<grid_for(n), kThreads, 0, s>>>(acol, aval, alen, n_rows, k, tptr, t, n, mix, one_minus_mix,
                                                                 nullptr, uptr, indices, data);
        MGB_LAUNCH_CHECK();
    }
    narrow_kernel<<<grid_for(n + 1), kThreads, 0, s>>>(uptr, n + 1, indptr);
    MGB_LAUNCH_CHECK();
    MGB_CUDA(cudaStreamSynchronize(s));
    return nnz;
}

int64_t transform_schedule_dev(const float* w, const int64_t* ind, int64_t m, int k, int64_t n_train,
                               double samples_per_node, int n_epochs, int32_t* head, int32_t* tail, float* eps,
                               GraphWork& gw, cudaStream_t s) {
    const int64_t n = m * (int64_t)k;
    int64_t* cnt = static_cast<int64_t*>(gw.sched.ensure(sizeof(int64_t)));
    transform_schedule_kernel<<<1, kSchedThreads, 0, s>>>(w, ind, n, k, n_train, samples_per_node * (double)m,
                                                          1.0 / (double)n_epochs, head, tail, eps, cnt);
    MGB_LAUNCH_CHECK();
    int64_t kept = 0;
    MGB_CUDA(cudaMemcpyAsync(&kept, cnt, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MGB_CUDA(cudaStreamSynchronize(s));
    return kept;
}

int64_t edge_schedule_dev(const int32_t* indptr, const int32_t* indices, const float* w, int64_t n, int64_t nnz,
                          double samples_per_node, int n_epochs, int32_t* head, int32_t* tail, float* eps,
                          GraphWork& gw, cudaStream_t s) {
    if (nnz <= 0) return 0;
    const double target = samples_per_node * (double)n;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((nnz + kThreads - 1) / kThreads, kSchedBlocks));
    char* base = static_cast<char*>(gw.s_part.ensure(sizeof(SchedState) + sizeof(double2) * kSchedBlocks));
    SchedState* st = reinterpret_cast<SchedState*>(base);
    double2* part = reinterpret_cast<double2*>(base + sizeof(SchedState));
    int32_t* cnt = static_cast<int32_t*>(gw.s_flag.ensure(sizeof(int32_t) * (size_t)n));
    int64_t* off = static_cast<int64_t*>(gw.s_off.ensure(sizeof(int64_t) * (size_t)(n + 1)));
    MGB_CUDA(cudaMemsetAsync(st, 0, sizeof(SchedState), s));
    sched_round_kernel<true><<<blocks, kThreads, 0, s>>>(w, nnz, target, part, st);
    MGB_LAUNCH_CHECK();
    const double min_freq = 1.0 / (double)n_epochs;
    const int rb = (int)std::max<int64_t>(1, std::min<int64_t>((n * 32 + kThreads - 1) / kThreads, 32LL * kNumSMs));
    int64_t kept = 0;
    for (int rounds = 0;;) {
        // a dozen rounds ahead of the host's look at the state: most solves end within them
        for (int q = 0; q < 12; ++q, ++rounds) {
            sched_round_kernel<false><<<blocks, kThreads, 0, s>>>(w, nnz, target, part, st);
            MGB_LAUNCH_CHECK();
        }
        sched_rows_kernel<false><<<rb, kThreads, 0, s>>>(indptr, indices, w, n, st, min_freq, cnt, nullptr, nullptr, nullptr,
                                                         nullptr);
        MGB_LAUNCH_CHECK();
        exclusive_scan_i32(cnt, n, off, gw.s_tmp, s);
        SchedState h;
        MGB_CUDA(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
        MGB_CUDA(cudaMemcpyAsync(&kept, off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        MGB_CUDA(cudaStreamSynchronize(s));
        if (h.done || rounds >= 204) break;
    }
    sched_rows_kernel<true><<<rb, kThreads, 0, s>>>(indptr, indices, w, n, st, min_freq, nullptr, off, head, tail, eps);
    MGB_LAUNCH_CHECK();
    return kept;
}

}  // namespace mgb
