// Query kNN on the device: knn_search of src/nndescent.cpp:585-690 (the beam search of new rows over the training
// rows' neighbour graph that MAGNET.transform runs, magnet/knn.py:131-152).
//
// Per query the reference keeps a max-heap of the best `ef` rows found (res), a min-heap of rows still to expand
// (cand) and a visited stamp per row; it starts from the n_entry landmarks closest to the query (or n_entry random
// rows without landmarks), then repeatedly expands the closest candidate's graph row until the closest candidate is
// farther than the ef-th result. Here one warp runs one query with the same steps:
//  * the distances of a graph row's neighbours (or of the landmarks), up to 32 at a time, are computed in the
//    reference's squared-distance order (sqdist.cuh), so every distance equals the reference's bit for bit. In the
//    AVX-512 order four lanes share a row, each holding four of the sixteen sums, so a row arrives as 64-byte pieces
//    and a batch of 32 rows of 64 features in one round of reads;
//  * the visited marks are a bit per training row in a bitset owned by the warp (test-and-set with atomicOr, the
//    row's neighbours at once, while their distances are read; the rows of a CSR row are distinct), cleared after the
//    query from its visit list;
//  * both heaps are one list, the best ef rows by distance in the lanes' registers with a mark on the expanded ones:
//    a row pushed on cand is pushed on res too, and one that has dropped out of res is no closer than the ef-th result
//    for good, so cand's next is the closest row of the list without a mark, and the search ends when there is none (the
//    reference would still expand a dropped row that ties with the ef-th result).
//    Rows that cannot enter are dropped by all lanes at once; the others enter one by one in the row's order, as the
//    reference's loop takes them, by a ballot and a shift.
// The expansion order and the result set therefore follow the reference's exactly whenever no two distances tie
// (ties may be broken differently by the reference's heaps). The results are sorted by (distance, row).
// Bound by the latency of the walk: about 65 expansions one after another per query. One lane's heap operations in
// shared memory and a distance's four dependent rounds of reads took most of it before: 0.88 ms for 48 queries and
// 6.2 ms for 4096 (60k and 200k rows of 64 features, ef 64); 0.39 and 1.69 ms now.
#include "common.cuh"
#include "sqdist.cuh"
#include "graph.cuh"
#include <vector>
#include <algorithm>
#include <string>

namespace mgb {

namespace {

constexpr int kSearchWarps = 4;        // queries in flight per block
constexpr int kMaxEf = 256;            // result list capacity (ef)
// Rows a query may have pushed and not expanded; one that counts more is reported as not supported. The list needs no
// such limit: it is what a heap of candidates held, and the calls that were refused for it stay refused.
constexpr int kCandCap = 2048;
constexpr int kVisitCap = 8192;        // visit list per warp; past it the warp clears its whole bitset
constexpr int kSearchPerSm = 16;       // queries in flight per SM at most: their bitsets (n / 8 bytes each) share the L2
constexpr int kEntryTop = 8;           // entry landmarks a lane keeps in registers; more are taken one by one
constexpr unsigned kFull = 0xffffffffu;
constexpr int32_t kExpanded = INT32_MIN;   // mark bit on a listed row

__device__ __forceinline__ bool pair_less(float da, int32_t ia, float db, int32_t ib) {
    return da < db || (da == db && ia < ib);
}

struct SearchArgs {
    const float* X; int64_t n; int d;
    const int32_t* gptr; const int32_t* gidx;
    const int32_t* land; int64_t n_land;
    const int32_t* entries;            // m x n_entry random entry rows (no landmarks), else null
    const float* Q; int64_t m;
    int k, ef, n_entry;
    int32_t* out_i; float* out_d;
    uint32_t* bits; int64_t bit_words;   // per warp slot: bit_words words
    int32_t* visits;                      // per warp slot: kVisitCap rows
    float* ldist;                         // per warp slot: n_land distances (n_entry > kEntryTop only)
    int* overflow;                        // queries that held more than kCandCap rows to expand
    int stage;                            // queries are staged in shared memory
};

// the best ef rows seen, ascending by (distance, row): position 32 c + lane in register c
template <int CH>
struct BestList {
    float d[CH];
    int32_t i[CH];
    int n = 0;
    __device__ __forceinline__ void clear() {
        n = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) { d[c] = INFINITY; i[c] = kExpanded | INT32_MAX; }
    }
    __device__ __forceinline__ float at(int pos) const {
        float v = 0.f;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const float t = __shfl_sync(kFull, d[c], pos & 31);
            if (c == (pos >> 5)) v = t;
        }
        return v;
    }
    // row j at distance dj enters at its place by (distance, row); the ef-th drops out when the list is full
    __device__ __forceinline__ void insert(float dj, int32_t j, int ef, int lane) {
        int pos = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) pos += __popc(__ballot_sync(kFull, c * 32 + lane < n && pair_less(d[c], i[c] & INT32_MAX, dj, j)));
#pragma unroll
        for (int c = CH - 1; c >= 0; --c) {
            float ud = __shfl_up_sync(kFull, d[c], 1);
            int32_t ui = __shfl_up_sync(kFull, i[c], 1);
            if (c > 0) {
                const float pd = __shfl_sync(kFull, d[c > 0 ? c - 1 : 0], 31);
                const int32_t pi = __shfl_sync(kFull, i[c > 0 ? c - 1 : 0], 31);
                if (lane == 0) { ud = pd; ui = pi; }
            }
            const int at_ = c * 32 + lane;
            if (at_ == pos) { d[c] = dj; i[c] = j; }
            else if (at_ > pos && at_ < ef) { d[c] = ud; i[c] = ui; }
        }
        if (n < ef) ++n;
    }
    // the closest row not expanded, marked now; -1 when there is none
    __device__ __forceinline__ int32_t take(int lane) {
        int32_t row = -1;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const unsigned open = __ballot_sync(kFull, c * 32 + lane < n && i[c] >= 0);
            if (row < 0 && open) {
                const int src = __ffs(open) - 1;
                row = __shfl_sync(kFull, i[c], src);
                if (lane == src) i[c] |= kExpanded;
            }
        }
        return row;
    }
};

// the squared distances of up to 32 rows (row j of lane l, -1: none) to the query in q, each in its lane
template <int ORDER, bool VEC>
__device__ __forceinline__ float batch_distance(const SearchArgs& a, const float* __restrict__ q, int32_t j, int lane) {
    if constexpr (ORDER != 0) {
        return j >= 0 ? sqdist<ORDER>(q, a.X + (int64_t)j * a.d, a.d) : 0.f;
    } else {
        // lane l of a quad holds sums 4l .. 4l + 3 of the sixteen; quad r of pass g has row 8 g + r
        const int sub = lane & 3, quad = lane >> 2;
        const int blocks = a.d / 16;
        float4 acc[4];
        const float* row[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int32_t jj = __shfl_sync(kFull, j, 8 * g + quad);
            row[g] = jj >= 0 ? a.X + (int64_t)jj * a.d : nullptr;
            acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll 4
        for (int b = 0; b < blocks; ++b) {
            const int at = 16 * b + 4 * sub;
            float4 x[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                x[g] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (row[g]) {
                    if (VEC) x[g] = __ldg(reinterpret_cast<const float4*>(row[g] + at));
                    else x[g] = make_float4(__ldg(row[g] + at), __ldg(row[g] + at + 1), __ldg(row[g] + at + 2), __ldg(row[g] + at + 3));
                }
            }
            const float4 qv = VEC ? *reinterpret_cast<const float4*>(q + at) : make_float4(q[at], q[at + 1], q[at + 2], q[at + 3]);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float df = __fsub_rn(qv.x, x[g].x); acc[g].x = __fmaf_rn(df, df, acc[g].x);
                df = __fsub_rn(qv.y, x[g].y); acc[g].y = __fmaf_rn(df, df, acc[g].y);
                df = __fsub_rn(qv.z, x[g].z); acc[g].z = __fmaf_rn(df, df, acc[g].z);
                df = __fsub_rn(qv.w, x[g].w); acc[g].w = __fmaf_rn(df, df, acc[g].w);
            }
        }
        float mine = 0.f;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            // sums 8 + k onto k (lanes 2, 3 onto 0, 1), 4 + k onto k (lane 1 onto 0), then (0 + 2) + (1 + 3)
            float t[4] = {acc[g].x, acc[g].y, acc[g].z, acc[g].w};
#pragma unroll
            for (int o = 2; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < 4; ++c) t[c] = __fadd_rn(__shfl_xor_sync(kFull, t[c], o), t[c]);
            float s = __fadd_rn(__fadd_rn(t[0], t[2]), __fadd_rn(t[1], t[3]));
            if (row[g])
                for (int i = 16 * blocks; i < a.d; ++i) { const float df = __fsub_rn(q[i], __ldg(row[g] + i)); s = __fmaf_rn(df, df, s); }
            const float r = __shfl_sync(kFull, s, 4 * (lane & 7));
            if ((lane >> 3) == g) mine = r;
        }
        return mine;
    }
}

template <int ORDER, int CH, bool VEC>
__global__ void __launch_bounds__(32 * kSearchWarps) search_kernel(SearchArgs a) {
    extern __shared__ float query_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float* const staged = a.stage ? query_smem + (size_t)wib * a.d : nullptr;
    const int64_t slot = (int64_t)blockIdx.x * kSearchWarps + wib;
    const int64_t slots = (int64_t)gridDim.x * kSearchWarps;
    uint32_t* bits = a.bits + slot * a.bit_words;
    int32_t* visits = a.visits + slot * kVisitCap;
    float* ldist = a.ldist + slot * a.n_land;
    for (int64_t q = slot; q < a.m; q += slots) {
        const float* qv = a.Q + q * a.d;
        if (staged) {
            for (int t = lane; t < a.d; t += 32) staged[t] = qv[t];
            __syncwarp();
            qv = staged;
        }
        BestList<CH> best;
        best.clear();
        int ncand = 0, nvis = 0;
        bool overflow = false;
        // rows of one batch (up to 32, one per lane, -1 none) in the reference's order: visited test-and-set and
        // distance, then the sequential decisions of consider()
        auto consider_batch = [&](int32_t j) {
            bool fresh = false;
            if (j >= 0) {
                const uint32_t bit = 1u << (j & 31);
                fresh = (atomicOr(&bits[j >> 5], bit) & bit) == 0u;
            }
            const float dd = batch_distance<ORDER, VEC>(a, qv, j, lane);
            const unsigned fm = __ballot_sync(kFull, fresh);
            if (fresh) {
                const int r = nvis + __popc(fm & ((1u << lane) - 1u));
                if (r < kVisitCap) visits[r] = j;
            }
            nvis += __popc(fm);
            // the ef-th distance only falls, so a row that cannot enter now cannot enter later
            float worst = best.n < a.ef ? INFINITY : best.at(a.ef - 1);
            unsigned mm = __ballot_sync(kFull, fresh && (best.n < a.ef || dd < worst));
            while (mm) {
                const int src = __ffs(mm) - 1;
                mm &= mm - 1u;
                const float dj = __shfl_sync(kFull, dd, src);
                const int32_t jj = __shfl_sync(kFull, j, src);
                if (best.n < a.ef || dj < worst) {
                    best.insert(dj, jj, a.ef, lane);
                    worst = best.n < a.ef ? INFINITY : best.at(a.ef - 1);
                    if (ncand < kCandCap) ++ncand;
                    else overflow = true;
                }
            }
        };
        // entry points
        if (a.n_land > 0) {
            const int take = (int)((int64_t)a.n_entry < a.n_land ? (int64_t)a.n_entry : a.n_land);
            const bool few = take <= kEntryTop;
            // each lane's closest landmarks by (distance, row), ascending
            float td[kEntryTop];
            int32_t ti[kEntryTop];
#pragma unroll
            for (int t = 0; t < kEntryTop; ++t) { td[t] = INFINITY; ti[t] = INT32_MAX; }
            for (int64_t l0 = 0; l0 < a.n_land; l0 += 32) {
                const int64_t l = l0 + lane;
                const int32_t j = l < a.n_land ? a.land[l] : -1;
                const float dl = batch_distance<ORDER, VEC>(a, qv, j, lane);
                if (!few) { if (j >= 0) ldist[l] = dl; continue; }
                if (j >= 0) {
                    float cd = dl;
                    int32_t ci = j;
#pragma unroll
                    for (int t = 0; t < kEntryTop; ++t)
                        if (cd == td[t] && ci == ti[t]) {   // a landmark given twice counts once
                            cd = INFINITY; ci = INT32_MAX;
                        } else if (pair_less(cd, ci, td[t], ti[t])) {
                            const float sd = td[t]; const int32_t si = ti[t];
                            td[t] = cd; ti[t] = ci; cd = sd; ci = si;
                        }
                }
            }
            __syncwarp();
            float last_d = -INFINITY;
            int32_t last_i = -1;
            for (int e = 0; e < take; ++e) {
                // the next (distance, row) pair after the last one taken: the partial_sort of the reference
                float bd = INFINITY;
                int32_t bi = INT32_MAX;
                if (few) {
                    bd = td[0]; bi = ti[0];
                } else {
                    for (int64_t l = lane; l < a.n_land; l += 32) {
                        const float dl = ldist[l];
                        const int32_t il = a.land[l];
                        if (pair_less(last_d, last_i, dl, il) && pair_less(dl, il, bd, bi)) { bd = dl; bi = il; }
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float od = __shfl_xor_sync(kFull, bd, o);
                    const int32_t oi = __shfl_xor_sync(kFull, bi, o);
                    if (pair_less(od, oi, bd, bi)) { bd = od; bi = oi; }
                }
                if (few && td[0] == bd && ti[0] == bi) {   // the lane it came from moves on (so do lanes with a copy)
#pragma unroll
                    for (int t = 0; t + 1 < kEntryTop; ++t) { td[t] = td[t + 1]; ti[t] = ti[t + 1]; }
                    td[kEntryTop - 1] = INFINITY; ti[kEntryTop - 1] = INT32_MAX;
                }
                last_d = bd; last_i = bi;
                consider_batch(lane == 0 && bi != INT32_MAX ? bi : -1);
            }
        } else {
            for (int e = 0; e < a.n_entry; ++e) consider_batch(lane == 0 ? a.entries[q * a.n_entry + e] : -1);
        }
        // expansions
        for (;;) {
            const int32_t row = best.take(lane);
            if (row < 0) break;
            --ncand;
            const int32_t b = a.gptr[row], e = a.gptr[row + 1];
            for (int32_t j0 = b; j0 < e; j0 += 32) consider_batch(j0 + lane < e ? a.gidx[j0 + lane] : -1);
        }
        if (overflow && lane == 0) atomicAdd(a.overflow, 1);
        // the first k of the list
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int at = c * 32 + lane;
            if (at < a.k) {
                a.out_i[q * a.k + at] = at < best.n ? (best.i[c] & INT32_MAX) : -1;
                a.out_d[q * a.k + at] = at < best.n ? best.d[c] : INFINITY;
            }
        }
        // clear this query's visited bits for the next one
        __syncwarp();
        if (nvis <= kVisitCap) {
            for (int v = lane; v < nvis; v += 32) bits[visits[v] >> 5] = 0u;
        } else {
            for (int64_t w = lane; w < a.bit_words; w += 32) bits[w] = 0u;
        }
        __syncwarp();
    }
}

struct SearchWork {
    DevBuf bits, visits, ldist, flag, entries;
    int64_t bits_bytes = 0;
};
thread_local SearchWork g_search;

using SearchKernel = void (*)(SearchArgs);

// the list's registers by ef; rows read as 16 bytes per lane when every row of X and Q is 16-byte aligned
template <int ORDER, bool VEC>
SearchKernel search_for_ef(int ef) {
    return ef <= 64 ? search_kernel<ORDER, 2, VEC> : (ef <= 128 ? search_kernel<ORDER, 4, VEC> : search_kernel<ORDER, 8, VEC>);
}

}  // namespace

void knn_search_dev(const float* X, int64_t n, int d, const int32_t* gptr, const int32_t* gidx, const int32_t* land,
                    int64_t n_land, const int32_t* entries_host, const float* Q, int64_t m, int k, int ef,
                    int n_entry, int order, int32_t* out_i, float* out_d, cudaStream_t s) {
    if (m == 0) return;
    const bool vec = d % 4 == 0 && reinterpret_cast<uintptr_t>(X) % 16 == 0 && reinterpret_cast<uintptr_t>(Q) % 16 == 0;
    const SearchKernel kernel = order == 0 ? (vec ? search_for_ef<0, true>(ef) : search_for_ef<0, false>(ef))
                              : order == 1 ? search_for_ef<1, false>(ef)
                                           : search_for_ef<2, false>(ef);
    const bool stage = (size_t)d * sizeof(float) * kSearchWarps <= 32768;
    const size_t smem = stage ? (size_t)d * sizeof(float) * kSearchWarps : 0;
    int per_sm = 0;
    MGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * kSearchWarps, smem));
    per_sm = std::max(1, std::min(per_sm, kSearchPerSm / kSearchWarps));
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((m + kSearchWarps - 1) / kSearchWarps,
                                                                  (int64_t)per_sm * kNumSMs));
    const int64_t slots = blocks * kSearchWarps;
    const int64_t words = (n + 31) / 32;
    SearchWork& w = g_search;
    const int64_t need = slots * words * (int64_t)sizeof(uint32_t);
    if (need > w.bits_bytes || !w.bits.p) {
        w.bits.ensure((size_t)need);
        MGB_CUDA(cudaMemsetAsync(w.bits.p, 0, (size_t)need, s));   // kept zero by every query after
        w.bits_bytes = need;
    }
    w.visits.ensure(sizeof(int32_t) * (size_t)slots * kVisitCap);
    w.ldist.ensure(n_entry > kEntryTop ? sizeof(float) * (size_t)std::max<int64_t>(1, slots * n_land) : sizeof(float));
    int* flag = static_cast<int*>(w.flag.ensure(sizeof(int)));
    MGB_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));
    const int32_t* entries = nullptr;
    if (n_land == 0) {
        int32_t* e = static_cast<int32_t*>(w.entries.ensure(sizeof(int32_t) * (size_t)m * n_entry));
        MGB_CUDA(cudaMemcpyAsync(e, entries_host, sizeof(int32_t) * (size_t)m * n_entry, cudaMemcpyHostToDevice, s));
        entries = e;
    }
    SearchArgs a{X, n, d, gptr, gidx, land, n_land, entries, Q, m, k, ef, n_entry, out_i, out_d,
                 w.bits.as<uint32_t>(), words, w.visits.as<int32_t>(), w.ldist.as<float>(), flag, stage ? 1 : 0};
    kernel<<<(unsigned)blocks, 32 * kSearchWarps, smem, s>>>(a);
    MGB_LAUNCH_CHECK();
    int h = 0;
    MGB_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    MGB_CUDA(cudaStreamSynchronize(s));
    if (h) throw Error(MG_ERR_NOT_SUPPORTED, std::to_string(h) + " queries needed more than " +
                                                 std::to_string(kCandCap) + " candidates; lower ef");
}

int knn_search_max_ef() { return kMaxEf; }

}  // namespace mgb
