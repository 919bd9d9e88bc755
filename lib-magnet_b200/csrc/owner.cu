// Owner mode of optimize_layout (parallel = 1): src/layout.cpp:118-276 with OWNER = true, :300-330 (owner epochs),
// :441-463 (chunks), :31-40 (the owner attraction scale 1.5).
//
// The reference splits the nodes at the edge quantiles into n_chunks = min(4096, max(1, E / 4096)) chunks (edges
// sorted by head). In epoch e, chunk k draws from its own stream stream_seed(seed, e, k) over its edges in order,
// moves only its own heads u (no step on the tail or on the partners) and reads every other position from the
// layout as it was at the start of the epoch; with the reverse mid pairs, u also takes, after each edge, the pulls
// of the nodes that chose it. The result is a function of the inputs alone, whatever the thread count.
//
// On the device the schedule and the draws of a batch of epochs run ahead of the positions, because they depend on
// them only through a negative at distance 0 exactly (src/layout.cpp:181), which draws dim extra uniforms:
//  1. schedule, one thread per edge: advances eons / eonns over the batch's epochs as the reference does and records
//     each epoch's negatives count per sampled edge;
//  2. chain, one thread or warp per (epoch, chunk): consumes the chunk's stream in edge order as the edge loop would (n_neg
//     draws, the mid-range test and walk, the reverse-pull draws), recording at each head's first sampled edge the
//     stream state where its draws start. It reads no position.
// Then each epoch, from a read buffer into a write buffer that swap from epoch to epoch (two copies of the layout, of
// which only rows with edges are ever written):
//  3. node pass: replays every head's edges as the reference does from the head's recorded state (other positions
//     from the read buffer, its own in registers) and writes its row. A negative at distance 0 marks the node's
//     chunk, since the states recorded after it are then off by dim draws;
//  4. fallback, one thread per chunk, doing work for marked chunks only: replays the whole chunk serially from the
//     chunk's seed.
// Epochs without mid-range pulls in 2-d under the power kernel and the sgd optimizer (every transform) run steps 3
// and 4 of a whole batch in one cooperative launch with a grid barrier between epochs (owner_epochs_kernel); other
// epochs launch the two steps one by one, Adam's with its state and the layout copied aside first.
// This file is compiled without FMA contraction (-fmad=false): every product and sum rounds on its own, as in
// the reference's plain x86-64 build. The power kernel with b = rep_b = 1 under the sgd optimizer uses +, *, / and
// sqrt only and reproduces the reference bit for bit; powf, expf, tanhf and coshf may differ from the host libm
// in the last place.
#include "sgd.cuh"
#include <algorithm>
#include <climits>

namespace mgb {

namespace {

constexpr int32_t kNotSampled = INT32_MIN;   // n_neg record of an edge skipped this epoch
constexpr float kOwnerAttraction = 1.5f;     // OWNER_ATT, src/layout.cpp:40

struct OwnerDev {
    const int64_t* own; const int64_t* eown; int n_chunks;   // first node / first edge of each chunk (+1 entry)
    const int64_t* row;                                       // first edge of each node (n + 1 entries)
    const int32_t* rev_indptr; const int32_t* rev_indices;    // reverse mid pairs or NULL
    int32_t* n_neg;                                           // per edge: this epoch's negatives, kNotSampled
    uint64_t* state;                                          // stream state of a head, at its first edge
    int* dirty;                                               // per chunk: a distance-0 negative was drawn
    const float* Yr;                                          // the layout at the start of the epoch
    const float* snap_m; const float* snap_v; const int32_t* snap_t;   // the Adam state at the start
};

// the mid-range partner of edge (u, v) (src/layout.cpp:225-249), after the mid_rate test succeeded
__device__ __forceinline__ int32_t mid_partner(const SgdDev& c, Rng& r, int64_t u, int32_t v) {
    int32_t w = v;
    if (c.jump_indptr) {
        const int L = c.walk_lens ? c.walk_lens[v] : c.walk_len;
        for (int h = 0; h < L; ++h) {
            const int32_t js = c.jump_indptr[w], je = c.jump_indptr[w + 1];
            if (je > js && r.uniform() < c.mid_jump) {
                w = c.jump_indices[js + (int32_t)r.below((uint32_t)(je - js))];
            } else {
                const int32_t s0 = c.indptr[w], e0 = c.indptr[w + 1];
                if (e0 <= s0) break;
                w = c.indices[s0 + (int32_t)r.below((uint32_t)(e0 - s0))];
            }
        }
    } else if (c.mid_pairs) {
        w = c.mid_pairs[u * c.n_mid + r.below((uint32_t)c.n_mid)];
    } else {
        const int L = c.walk_lens ? c.walk_lens[v] : c.walk_len;
        for (int h = 0; h < L; ++h) {
            const int32_t s0 = c.indptr[w], e0 = c.indptr[w + 1];
            if (e0 <= s0) break;
            w = c.indices[s0 + (int32_t)r.below((uint32_t)(e0 - s0))];
        }
    }
    return w;
}

// apply_step (src/layout.cpp:90-116) on a row held in registers; the Adam state of u belongs to this thread
template <int DM>
__device__ __forceinline__ void owner_step(const SgdDev& c, float* yu, const float* g, float alpha, int64_t u,
                                           int dim) {
    float step[DM];
    if (c.optimizer == 1) {
        const int32_t t = ++c.adam_t[u];
        const float c1 = 1.0f - powf(c.beta1, (float)t), c2 = 1.0f - powf(c.beta2, (float)t);
        float* m = c.adam_m + u * dim;
        float* v = c.adam_v + u * dim;
        for (int d = 0; d < dim; ++d) {
            m[d] = c.beta1 * m[d] + (1.0f - c.beta1) * g[d];
            v[d] = c.beta2 * v[d] + (1.0f - c.beta2) * g[d] * g[d];
            step[d] = alpha * (m[d] / c1) / (sqrtf(v[d] / c2) + 1e-7f);
        }
    } else {
#pragma unroll
        for (int d = 0; d < DM; ++d)
            if (d < dim) step[d] = alpha * g[d];
    }
    const float cap = 4.0f * alpha;
    if (c.clip_mode == 1) {
        float n2 = 0.0f;
#pragma unroll
        for (int d = 0; d < DM; ++d)
            if (d < dim) n2 += step[d] * step[d];
        if (n2 > cap * cap) {
            const float f = cap / sqrtf(n2);
#pragma unroll
            for (int d = 0; d < DM; ++d)
                if (d < dim) step[d] *= f;
        }
    } else {
#pragma unroll
        for (int d = 0; d < DM; ++d)
            if (d < dim) step[d] = step[d] > cap ? cap : (step[d] < -cap ? -cap : step[d]);
    }
#pragma unroll
    for (int d = 0; d < DM; ++d)
        if (d < dim) yu[d] += step[d];
}

// What a thread whose work others wait for at a grid barrier tells them: one count per 256 units of work (a draw, an edge,
// a copied value, a listing; at most a few microseconds each), so the count moves at least every millisecond or so.
struct Beat {
    unsigned* at;
    unsigned done = 0;
    __device__ __forceinline__ void tick() {
        if ((++done & 255u) == 0u) atomicAdd(at, 1u);
    }
};
struct NoBeat {   // of a launch in which nobody waits
    __device__ __forceinline__ void tick() {}
};

// The edges of head node u in one epoch, from stream state `state`; returns the state after them. The row is read
// from the snapshot and written back to Y (when u may move). `jitter` is set when a negative lands at distance 0.
template <int D, class B>
__device__ uint64_t owner_node(const SgdDev& c, const OwnerDev& o, int64_t u, uint64_t state, float alpha,
                               float mid_w, bool& jitter, B& beat) {
    constexpr int DM = D ? D : kMaxDim;
    const int dim = D ? D : c.dim;
    Rng r(0);
    r.s = state;
    const bool move_u = u >= c.n_fixed;
    const float inv_n_mid = c.n_mid > 0 ? 1.0f / (float)c.n_mid : 0.0f;
    float yu[DM], diff[DM], gu[DM], gk[DM];
#pragma unroll
    for (int d = 0; d < DM; ++d)
        if (d < dim) yu[d] = o.Yr[u * dim + d];
    const int64_t row1 = o.row[u + 1];
    for (int64_t w0 = o.row[u]; w0 < row1; w0 += 64) {
        // the sampled edges of a window of 64 as a bit mask, taken in edge order
        const int cnt = (int)(row1 - w0 < 64 ? row1 - w0 : 64);
        beat.tick();
        uint64_t mask = 0;
        for (int t = 0; t < cnt; ++t)
            if (o.n_neg[w0 + t] != kNotSampled) mask |= 1ull << t;
        while (mask) {
            const int64_t i = w0 + (__ffsll((long long)mask) - 1);
            mask &= mask - 1;
            const int n_neg = o.n_neg[i];
            beat.tick();
            const int32_t v = c.tail[i];
            const float* yv = o.Yr + (int64_t)v * dim;
            float d2 = 0.0f;
#pragma unroll
            for (int d = 0; d < DM; ++d)
                if (d < dim) { gu[d] = 0.0f; diff[d] = yu[d] - yv[d]; d2 += diff[d] * diff[d]; }
            const float b_u = c.node_b ? c.node_b[u] : c.b;
            const float b_uv = c.node_b ? 0.5f * (c.node_b[u] + c.node_b[v]) : c.b;
            const float pw_v = (c.b_is_one && !c.node_b) ? d2 : (d2 > 0.0f ? powf(d2, b_uv) : 0.0f);
            // attraction along the edge, the head only, scaled by 1.5
            if (d2 > 0.0f) {
                float coeff;
                if (c.kernel == 0) coeff = -kOwnerAttraction * c.exaggeration * 2.0f * c.a * b_uv * pw_v / (d2 * (c.a * pw_v + 1.0f));
                else if (c.kernel == 1) coeff = -kOwnerAttraction * c.exaggeration * 2.0f * c.a;
                else if (c.kernel == 2) { const float dd = sqrtf(d2); coeff = -kOwnerAttraction * c.exaggeration * c.a * tanhf(c.a * dd) / dd; }
                else coeff = -kOwnerAttraction * c.exaggeration * 2.0f * c.a * (1.0f + tanhf(c.a * d2));
#pragma unroll
                for (int d = 0; d < DM; ++d)
                    if (d < dim) gu[d] += coeff * diff[d];
            }
            // repulsion from the negatives, read from the snapshot
            for (int p = 0; p < n_neg; ++p) {
                const int32_t k = (int32_t)r.below((uint32_t)c.n);
                beat.tick();
                if (k == u) continue;
                const float* yk = o.Yr + (int64_t)k * dim;
                float dd = 0.0f;
#pragma unroll
                for (int d = 0; d < DM; ++d)
                    if (d < dim) { diff[d] = yu[d] - yk[d]; dd += diff[d] * diff[d]; }
                if (dd > 0.0f) {
                    float coeff;
                    if (c.kernel == 0) {
                        if (c.node_b && c.rep_coupled) { const float pw = powf(dd, b_u); coeff = 2.0f * b_u * c.repulsion_strength / ((0.001f + dd) * (c.a * pw + 1.0f)); }
                        else { const float pw = c.rep_b_is_one ? dd : powf(dd, c.rep_b); coeff = c.two_b / ((0.001f + dd) * (c.rep_a * pw + 1.0f)); }
                    } else if (c.kernel == 1) {
                        const float q = expf(-c.a * dd);
                        coeff = c.repulsion_strength * 2.0f * c.a * q / fmaxf(1.0f - q, 1e-3f);
                    } else if (c.kernel == 2) {
                        const float rr = sqrtf(dd); const float q = 1.0f / coshf(c.a * rr);
                        coeff = c.repulsion_strength * c.a * q * tanhf(c.a * rr) / (rr * fmaxf(1.0f - q, 1e-3f));
                    } else {
                        const float th = fmaxf(tanhf(c.a * dd), 1e-3f);
                        coeff = c.repulsion_strength * 2.0f * c.a * (1.0f - th * th) / th;
                    }
#pragma unroll
                    for (int d = 0; d < DM; ++d)
                        if (d < dim) gu[d] += coeff * diff[d];
                } else {
                    jitter = true;
                    for (int d = 0; d < dim; ++d) gu[d] += (r.uniform() - 0.5f) * 1e-3f / fmaxf(alpha, 1e-6f);
                }
            }
            // mid-range partner, read from the snapshot
            if (mid_w > 0.0f && r.uniform() < c.mid_rate) {
                const int32_t w = mid_partner(c, r, u, v);
                if (w != u) {
                    const float* yw = o.Yr + (int64_t)w * dim;
#pragma unroll
                    for (int d = 0; d < DM; ++d)
                        if (d < dim) { const float g = -mid_w * (yu[d] - yw[d]); gu[d] += g; }
                }
            }
            if (move_u) owner_step<DM>(c, yu, gu, alpha, u, dim);
            // the pulls of the nodes that chose u as their partner, each its own step
            if (move_u && mid_w > 0.0f && o.rev_indptr) {
                const int32_t rs = o.rev_indptr[u], re = o.rev_indptr[u + 1];
                float p = c.mid_rate * (float)(re - rs) * inv_n_mid;
                while (p > 0.0f && re > rs) {
                    if (r.uniform() < p) {
                        const int32_t x = o.rev_indices[rs + (int32_t)r.below((uint32_t)(re - rs))];
                        if (x != u) {
                            const float* yx = o.Yr + (int64_t)x * dim;
#pragma unroll
                            for (int d = 0; d < DM; ++d)
                                if (d < dim) gk[d] = -mid_w * (yu[d] - yx[d]);
                            owner_step<DM>(c, yu, gk, alpha, u, dim);
                        }
                    }
                    p -= 1.0f;
                }
            }
        }
    }
    if (move_u) {
#pragma unroll
        for (int d = 0; d < DM; ++d)
            if (d < dim) c.Y[u * dim + d] = yu[d];
    }
    return r.s;
}

// ---------------------------------------------------------------------------------------------- pipelined node pass
// Each head by a group of 1 to 8 lanes, with owner_node's arithmetic in its order, for the common case (2-d, power
// kernel, no per-node b, sgd, no mid-range pulls). What depends on no position runs ahead: the group's first lane lists
// the row's sampled edges in shared memory and makes their draws, as many edges as fit the head's kSlots positions (a
// round: the whole row, as a rule); then all positions of the round are copied into shared memory at once (cp.async),
// and the edges computed from there one after another, an edge's negatives by the group's lanes side by side, their
// terms added in the negatives' order by every lane. A head so waits for one L2 read per round; owner_node waits for
// one per negative, 37 us per epoch of a 48-row transform. Per epoch of the same transform other forms took 17 us (one
// lane per head: the negatives' divisions one after another) and 14 us (8 lanes, each repeating the whole stream's
// 64-bit steps to keep its own draw).
constexpr int kEpochThreads = 128;
constexpr int kRowList = 32;    // edges of a row listed at a time
constexpr int kSlots = 48;      // positions of a round

__device__ __forceinline__ float2 ld2(const float* Y, int64_t u) {
    return __ldcg(reinterpret_cast<const float2*>(Y) + u);   // rows other SMs wrote in the previous epoch
}

// what a step reads besides positions, kept in registers over a launch's epochs
struct OwnerCoef {
    float a, b, rep_a, rep_b, two_b, att;   // att = -1.5 * exaggeration * 2 a b, in the reference's order of products
    bool b_one, rep_b_one, norm_clip;
    __device__ __forceinline__ explicit OwnerCoef(const SgdDev& c)
        : a(c.a), b(c.b), rep_a(c.rep_a), rep_b(c.rep_b), two_b(c.two_b),
          att(-kOwnerAttraction * c.exaggeration * 2.0f * c.a * c.b), b_one(c.b_is_one), rep_b_one(c.rep_b_is_one),
          norm_clip(c.clip_mode == 1) {}
};

// one negative at yk; at distance 0 the reference draws jitter, which marks the chunk for the replay
__device__ __forceinline__ void add_negative(const OwnerCoef& c, float2 yu, float2 yk, float2& gu, bool& jitter) {
    const float dx = yu.x - yk.x, dy = yu.y - yk.y;
    const float dd = dx * dx + dy * dy;
    if (dd > 0.0f) {
        const float pw = c.rep_b_one ? dd : powf(dd, c.rep_b);
        const float coeff = c.two_b / ((0.001f + dd) * (c.rep_a * pw + 1.0f));
        gu.x += coeff * dx; gu.y += coeff * dy;
    } else {
        jitter = true;
    }
}

__device__ __forceinline__ void xorshift(uint64_t& s) { s ^= s >> 12; s ^= s << 25; s ^= s >> 27; }   // Rng::next() without its output
__device__ __forceinline__ int32_t below_state(uint64_t s, int64_t n) {
    return (int32_t)((((s * 0x2545F4914F6CDD1DULL) >> 32) * (uint64_t)(uint32_t)n) >> 32);
}

__device__ __forceinline__ void copy8(float2* dst, const float2* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct EpochShared {
    int2 edge[kRowList][kEpochThreads];       // (negatives, tail) of the listed edges
    int32_t index[kSlots][kEpochThreads];     // the round's rows: per edge its tail, then its negatives (-1: the head itself)
    float2 pos[kSlots][kEpochThreads];        // their positions
};

// the walk over a head's sampled edges, in the head's own column of the shared arrays (held by the group's first lane)
struct HeadWalk {
    int col;
    int64_t row1, w0;
    int have, taken;        // edges listed, edges taken by rounds so far
    int first, used;        // the round: its first edge in the list, its slots
    bool wide;              // the round is one edge of more negatives than the slots hold: drawn as it is computed
    uint64_t stream;
    Beat beat;

    __device__ __forceinline__ void fill(const int32_t* __restrict__ rec, const int32_t* __restrict__ tails, EpochShared& sh) {
        const int cnt = (int)(row1 - w0 < kRowList ? row1 - w0 : kRowList);
        beat.tick();
        have = 0; taken = 0;
        for (int t0 = 0; t0 < cnt; t0 += 8) {
            int nn[8], tt[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                nn[t] = t0 + t < cnt ? rec[w0 + t0 + t] : kNotSampled;
                tt[t] = t0 + t < cnt ? tails[w0 + t0 + t] : 0;
            }
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (nn[t] != kNotSampled) sh.edge[have++][col] = make_int2(nn[t], tt[t]);
        }
    }
    // the next round's edges and draws; false when the row has ended
    __device__ __forceinline__ bool round(const int32_t* __restrict__ rec, const int32_t* __restrict__ tails, int64_t u,
                                          int64_t n_nodes, EpochShared& sh) {
        while (taken == have && w0 + kRowList < row1) { w0 += kRowList; fill(rec, tails, sh); }
        first = taken; used = 0; wide = false;
        while (taken < have) {
            const int2 e = sh.edge[taken][col];
            const int nn = e.x > 0 ? e.x : 0;
            beat.tick();
            if (used + 1 + nn > kSlots) {
                if (used > 0) break;
                wide = true;
                sh.index[0][col] = e.y;
                used = 1;
                ++taken;
                break;
            }
            sh.index[used++][col] = e.y;
            for (int t = 0; t < nn; ++t) {
                xorshift(stream);
                const int32_t k = below_state(stream, n_nodes);
                sh.index[used++][col] = k != (int32_t)u ? k : -1;
            }
            ++taken;
        }
        return taken > first;
    }
};

// the heads of a warp's groups of G lanes (has: the group has one, u), walks started and first rounds made by the
// groups' first lanes (more: the round has edges); the groups step together. Returns whether this lane met a
// distance-0 negative.
__device__ __forceinline__ bool owner_heads(const OwnerCoef& c, const float* __restrict__ Yr, float* __restrict__ Yw,
                                            const int32_t* __restrict__ rec, const int32_t* __restrict__ tails,
                                            int64_t n, int64_t n_fixed, int64_t u, bool has, HeadWalk& walk, bool more,
                                            float alpha, EpochShared& sh, int G) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), lead = lane - gl, col = threadIdx.x / G;
    bool jitter = false;
    const bool move_u = has && u >= n_fixed;
    float2 yu = make_float2(0.0f, 0.0f);
    if (has) yu = ld2(Yr, u);
    const float cap = 4.0f * alpha;
    for (;;) {
        const bool go = __shfl_sync(kFull, (int)(has && more), lead) != 0;
        if (!__any_sync(kFull, go)) break;
        const int first = __shfl_sync(kFull, walk.first, lead);
        const int taken = __shfl_sync(kFull, walk.taken, lead);   // by the whole warp: `go` differs between its groups
        const int edges = go ? taken - first : 0;
        const int used = __shfl_sync(kFull, walk.used, lead);
        const bool wide = __shfl_sync(kFull, (int)walk.wide, lead) != 0;
        if (go)
            for (int q = gl; q < used; q += G) {
                const int32_t k = sh.index[q][col];
                if (k >= 0) copy8(&sh.pos[q][col], reinterpret_cast<const float2*>(Yr) + k);
            }
        copies_done();
        __syncwarp();
        int at = 0;
        for (int e = 0; __any_sync(kFull, e < edges); ++e) {
            const bool act = e < edges;
            float2 gu = make_float2(0.0f, 0.0f);
            int nn = 0;
            if (act) {
                nn = max(sh.edge[first + e][col].x, 0);
                const float2 yv = sh.pos[at++][col];
                if (!wide)
                    for (int t = gl; t < nn; t += G) {
                        if (sh.index[at + t][col] < 0) continue;
                        float2 term = make_float2(0.0f, 0.0f);
                        bool zero = false;
                        add_negative(c, yu, sh.pos[at + t][col], term, zero);
                        sh.pos[at + t][col] = term;
                        if (zero) { jitter = true; sh.index[at + t][col] = -1; }
                    }
                const float dx = yu.x - yv.x, dy = yu.y - yv.y;
                const float d2 = dx * dx + dy * dy;
                if (d2 > 0.0f) {
                    const float pw_v = c.b_one ? d2 : powf(d2, c.b);
                    const float coeff = c.att * pw_v / (d2 * (c.a * pw_v + 1.0f));
                    gu.x += coeff * dx; gu.y += coeff * dy;
                }
            }
            __syncwarp();
            if (act && !wide) {
#pragma unroll 4
                for (int t = 0; t < nn; ++t, ++at) {
                    const float2 term = sh.pos[at][col];
                    if (sh.index[at][col] >= 0) { gu.x += term.x; gu.y += term.y; }
                }
            }
            if (__any_sync(kFull, act && wide)) {
                if (act && wide && gl == 0)
                    for (int t = 0; t < nn; ++t) {
                        xorshift(walk.stream);
                        walk.beat.tick();
                        const int32_t k = below_state(walk.stream, n);
                        if (k != (int32_t)u) add_negative(c, yu, ld2(Yr, k), gu, jitter);
                    }
                gu.x = __shfl_sync(kFull, gu.x, wide ? lead : lane);
                gu.y = __shfl_sync(kFull, gu.y, wide ? lead : lane);
            }
            if (act && move_u) {
                // apply_step (src/layout.cpp:90-116), as owner_step
                float sx = alpha * gu.x, sy = alpha * gu.y;
                if (c.norm_clip) {
                    float n2 = 0.0f;
                    n2 += sx * sx; n2 += sy * sy;
                    if (n2 > cap * cap) { const float f = cap / sqrtf(n2); sx *= f; sy *= f; }
                } else {
                    sx = sx > cap ? cap : (sx < -cap ? -cap : sx);
                    sy = sy > cap ? cap : (sy < -cap ? -cap : sy);
                }
                yu.x += sx; yu.y += sy;
            }
        }
        __syncwarp();   // the round's columns are read no more
        if (has && more && gl == 0) more = walk.round(rec, tails, u, n, sh);
        __syncwarp();
    }
    if (move_u && gl == 0) reinterpret_cast<float2*>(Yw)[u] = yu;
    return jitter;
}

// ---------------------------------------------------------------------------------------------- set-up kernels
// first edge of every node (lower bound of u in the sorted heads), u in [0, n]
__global__ void owner_rows_kernel(const int32_t* __restrict__ head, int64_t E, int64_t n, int64_t* __restrict__ row) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u > n) return;
    int64_t lo = 0, hi = E;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((int64_t)head[mid] < u) lo = mid + 1; else hi = mid;
    }
    row[u] = lo;
}

// chunk boundaries (src/layout.cpp:448-462): own[t] = max(head[E t / nc], own[t - 1]), which is head[E t / nc]
// itself for sorted heads; eown[t] is the first edge of own[t]
__global__ void owner_chunks_kernel(const int32_t* __restrict__ head, int64_t E, int64_t n, int nc,
                                    const int64_t* __restrict__ row, int64_t* __restrict__ own,
                                    int64_t* __restrict__ eown) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > nc) return;
    const int64_t node = t == 0 ? 0 : (t == nc ? n : (int64_t)head[E * t / nc]);
    own[t] = node;
    eown[t] = t == nc ? E : row[node];
}

__global__ void owner_sorted_kernel(const int32_t* __restrict__ head, int64_t E, int* __restrict__ unsorted) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x + 1; i < E; i += (int64_t)gridDim.x * blockDim.x)
        if (head[i - 1] > head[i]) { atomicExch(unsorted, 1); return; }
}

// the heads (edges that start a row), in no order; for layouts whose fixed rows mostly have no edges
__global__ void owner_heads_kernel(const int32_t* __restrict__ head, int64_t E, int32_t* __restrict__ list,
                                   int* __restrict__ count) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < E; base += stride) {
        const int64_t i = base + lane;
        const bool first = i < E && (i == 0 || head[i] != head[i - 1]);
        const unsigned m = __ballot_sync(0xffffffffu, first);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (first) list[at + __popc(m & ((1u << lane) - 1u))] = head[i];
    }
}

// ---------------------------------------------------------------------------------------------- epoch kernels
// run_epochs' linear schedule inside a call (src/layout.cpp:284-289), as sgd_sched evaluates it on the host
struct OwnerSched {
    int e0, n_span;
    float alpha0, alpha1, mid_w0, mid_w1;
    bool use_mid;
    __device__ __forceinline__ float frac(int epoch) const { return (float)(epoch - e0) / (float)n_span; }
    __device__ __forceinline__ float alpha(int epoch) const { return alpha0 + (alpha1 - alpha0) * frac(epoch); }
    __device__ __forceinline__ float mid_w(int epoch) const {
        return use_mid ? mid_w0 + (mid_w1 - mid_w0) * frac(epoch) : 0.0f;
    }
};

// the schedule of epochs [b0, b0 + B), one thread per edge (coalesced): eons / eonns advanced as
// src/layout.cpp:135,160-163,184 advance them, and each epoch's negatives count recorded (kNotSampled when
// eons[i] > epoch)
__global__ void __launch_bounds__(256) owner_schedule_kernel(SgdDev c, int32_t* __restrict__ rec, int b0, int B) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < c.n_edges;
         i += (int64_t)gridDim.x * blockDim.x) {
        float eo = c.eons[i], en = c.eonns[i];
        const float ep = c.eps[i];
        const float epn = ep / c.negative_sample_rate;
        for (int k = 0; k < B; ++k) {
            const float fepoch = (float)(b0 + k);
            int n_neg = kNotSampled;
            if (!(eo > fepoch)) {
                eo = eo + ep;
                n_neg = (int)((fepoch - en) / epn);
                en = en + (float)n_neg * epn;
            }
            rec[(int64_t)k * c.n_edges + i] = n_neg;
        }
        c.eons[i] = eo;
        c.eonns[i] = en;
    }
}

// The chain pass. A head's state is recorded at its first sampled edge (edges that are not sampled draw nothing, and
// a head without sampled edges draws nothing in the node pass), so heads without edges, such as the fixed training
// rows of a transform, cost nothing. No position is read and nothing is stored but the heads' states.
// Two forms, by the edges per chunk:
//  * owner_chain_kernel, one thread per (chunk, epoch of the batch), consecutive threads on consecutive epochs of the
//    same chunk: they walk the same rows, so their draws between two heads come together. For the short chunks of a
//    transform (256 edges); a warp each, launched per epoch, took 25-28 us per epoch;
//  * owner_chain_warp_kernel, one warp per (chunk, epoch): the lanes read 32 edges' counts and heads at a time and
//    take the sampled ones in order from a ballot; every lane holds the same stream state. For the reference's chunks
//    of 4096 edges and more, of which a batch has too few for a thread each (0.46 ms per epoch of the 1M-point
//    graph, several ms with a thread each).
constexpr int kChainThreads = 64;
constexpr int kChainWarps = 4;                    // chunks per block of the warp form
constexpr int64_t kChainThreadMaxEdges = 1024;    // mean edges per chunk up to which the thread form runs

__global__ void __launch_bounds__(kChainThreads) owner_chain_kernel(SgdDev c, OwnerDev o, OwnerSched sc, int b0, int B) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)B * o.n_chunks) return;
    const int k = (int)(t / B), be = (int)(t - (int64_t)k * B);
    const int epoch = b0 + be;
    const float mid_w = sc.mid_w(epoch);
    Rng r(stream_seed(c.seed, epoch, (uint64_t)k));
    const float inv_n_mid = c.n_mid > 0 ? 1.0f / (float)c.n_mid : 0.0f;
    const int32_t* __restrict__ rec = o.n_neg + (int64_t)be * c.n_edges;
    uint64_t* __restrict__ state = o.state + (int64_t)be * c.n_edges;
    const int64_t e0 = o.eown[k], e1 = o.eown[k + 1];
    int64_t row_start = e0;
    int32_t u = -1, done = -1;   // the head walked, the head whose state is recorded
    int pend = 0;                // negatives' draws not made yet (made when the state is needed)
    float p0 = 0.0f;
    constexpr int kAhead = 8;
    int32_t nn[kAhead], hh[kAhead];
    auto fetch = [&](int64_t base) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            nn[q] = base + q < e1 ? __ldg(rec + base + q) : kNotSampled;
            hh[q] = base + q < e1 ? __ldg(c.head + base + q) : u;
        }
    };
    auto draw_pending = [&]() {
        for (; pend > 0; --pend) xorshift(r.s);
    };
    if (e0 < e1) fetch(e0);
    for (int64_t base = e0; base < e1; base += kAhead) {
        int32_t cn[kAhead], ch[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) { cn[q] = nn[q]; ch[q] = hh[q]; }
        if (base + kAhead < e1) fetch(base + kAhead);
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            if (base + q >= e1) break;
            if (ch[q] != u) { u = ch[q]; row_start = base + q; draw_pending(); }
            if (cn[q] == kNotSampled) continue;
            if (u != done) {
                done = u;
                state[row_start] = r.s;
                // the reverse-pull rounds of each of u's edges: the same p for every edge of u
                p0 = 0.0f;
                if (u >= c.n_fixed && mid_w > 0.0f && o.rev_indptr) {
                    const int32_t rs = o.rev_indptr[u], re = o.rev_indptr[u + 1];
                    if (re > rs) p0 = c.mid_rate * (float)(re - rs) * inv_n_mid;
                }
            }
            pend += cn[q] > 0 ? cn[q] : 0;
            if (mid_w > 0.0f) {
                draw_pending();
                if (r.uniform() < c.mid_rate) (void)mid_partner(c, r, u, c.tail[base + q]);
                for (float p = p0; p > 0.0f; p -= 1.0f)
                    if (r.uniform() < p) (void)r.next();
            }
        }
    }
}

__global__ void __launch_bounds__(32 * kChainWarps) owner_chain_warp_kernel(SgdDev c, OwnerDev o, OwnerSched sc, int b0, int B) {
    const int64_t t = (int64_t)blockIdx.x * kChainWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= (int64_t)B * o.n_chunks) return;
    const int be = (int)(t / o.n_chunks), k = (int)(t - (int64_t)be * o.n_chunks);
    const int epoch = b0 + be;
    const float mid_w = sc.mid_w(epoch);
    Rng r(stream_seed(c.seed, epoch, (uint64_t)k));
    const float inv_n_mid = c.n_mid > 0 ? 1.0f / (float)c.n_mid : 0.0f;
    const int32_t* __restrict__ rec = o.n_neg + (int64_t)be * c.n_edges;
    uint64_t* __restrict__ state = o.state + (int64_t)be * c.n_edges;
    const int64_t e0 = o.eown[k], e1 = o.eown[k + 1];
    int64_t u = -1;
    float p0 = 0.0f;
    for (int64_t base = e0; base < e1; base += 32) {
        const int64_t i = base + lane;
        const int mine = i < e1 ? __ldg(rec + i) : kNotSampled;
        const int32_t my_head = i < e1 ? c.head[i] : -1;
        unsigned todo = __ballot_sync(0xffffffffu, mine != kNotSampled);
        while (todo) {
            const int b = __ffs(todo) - 1;
            todo &= todo - 1;
            const int n_neg = __shfl_sync(0xffffffffu, mine, b);
            const int32_t h = __shfl_sync(0xffffffffu, my_head, b);
            if (h != u) {
                u = h;
                if (lane == 0) state[o.row[u]] = r.s;
                // the reverse-pull rounds of each of u's edges: the same p for every edge of u
                p0 = 0.0f;
                if (u >= c.n_fixed && mid_w > 0.0f && o.rev_indptr) {
                    const int32_t rs = o.rev_indptr[u], re = o.rev_indptr[u + 1];
                    if (re > rs) p0 = c.mid_rate * (float)(re - rs) * inv_n_mid;
                }
            }
            for (int p = 0; p < n_neg; ++p) xorshift(r.s);
            if (mid_w > 0.0f && r.uniform() < c.mid_rate) (void)mid_partner(c, r, u, c.tail[base + b]);
            for (float p = p0; p > 0.0f; p -= 1.0f)
                if (r.uniform() < p) (void)r.next();
        }
    }
}

// the chunk holding u: the last k with own[k] <= u (empty chunks share their bound with the next one)
__device__ __forceinline__ int chunk_of(const OwnerDev& o, int64_t u) {
    int lo = 0, hi = o.n_chunks;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (o.own[mid] <= u) lo = mid; else hi = mid;
    }
    return lo;
}

template <int D>
__global__ void __launch_bounds__(128) owner_node_kernel(SgdDev c, OwnerDev o, float alpha, float mid_w) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= c.n || o.row[u] == o.row[u + 1]) return;
    bool jitter = false;
    NoBeat none;
    owner_node<D>(c, o, u, o.state[o.row[u]], alpha, mid_w, jitter, none);
    if (jitter) atomicExch(&o.dirty[chunk_of(o, u)], 1);
}

// the marked chunk k replayed serially from its seed; rows without edges never move
template <int D, class B>
__device__ __noinline__ void owner_replay(const SgdDev& c, const OwnerDev& o, int k, int epoch, float alpha,
                                          float mid_w, B beat) {
    // the heads of the chunk's edges (a marked chunk has at least one)
    const int64_t u0 = c.head[o.eown[k]], u1 = (int64_t)c.head[o.eown[k + 1] - 1] + 1;
    const int dim = c.dim;
    for (int64_t j = u0 * dim; j < u1 * dim; ++j) {
        c.Y[j] = o.Yr[j];
        beat.tick();
    }
    if (c.optimizer == 1) {
        for (int64_t j = u0 * dim; j < u1 * dim; ++j) { c.adam_m[j] = o.snap_m[j]; c.adam_v[j] = o.snap_v[j]; }
        for (int64_t u = u0; u < u1; ++u) c.adam_t[u] = o.snap_t[u];
    }
    uint64_t state = Rng(stream_seed(c.seed, epoch, (uint64_t)k)).s;
    bool jitter = false;
    for (int64_t u = u0; u < u1; ++u) {
        beat.tick();
        state = owner_node<D>(c, o, u, state, alpha, mid_w, jitter, beat);
    }
}

template <int D>
__global__ void __launch_bounds__(32) owner_fallback_kernel(SgdDev c, OwnerDev o, int epoch, float alpha,
                                                            float mid_w) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= o.n_chunks || !o.dirty[k]) return;
    o.dirty[k] = 0;
    owner_replay<D>(c, o, k, epoch, alpha, mid_w, NoBeat());
}

template <int D>
void owner_epoch_launch(const SgdDev& c, const OwnerDev& o, int epoch, float alpha, float mid_w, cudaStream_t s) {
    owner_node_kernel<D><<<ceil_div(c.n, 128), 128, 0, s>>>(c, o, alpha, mid_w);
    MGB_LAUNCH_CHECK();
    owner_fallback_kernel<D><<<ceil_div(o.n_chunks, 32), 32, 0, s>>>(c, o, epoch, alpha, mid_w);
    MGB_LAUNCH_CHECK();
}

// Grid barrier of a cooperative launch, in two halves: every block arrives on a counter that only grows, then waits for
// all. What it waits for has no bound of its own (a marked chunk is replayed by one thread, and a chunk may hold every
// edge of the call; a row may draw any number of negatives), so the wait ends without the others only when kPolls polls
// (one to three seconds) pass in which neither a block arrived nor a working thread's beat moved: it then sets *err
// and lets the kernel end. While every block runs, the polls that see no beat stay far below that.
struct GridBarrier {
    unsigned* count;
    unsigned* beat;
    int* err;
    unsigned passed = 0;
    static constexpr int kPolls = 4000000;
    __device__ __forceinline__ void arrive() {
        ++passed;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(count, 1u);
        }
    }
    __device__ __forceinline__ bool wait() {
        __shared__ int ok;
        if (threadIdx.x == 0) {
            const unsigned want = passed * gridDim.x;
            unsigned arrived, seen_arrived = 0u, seen_beat = 0u;
            int tries = 0;
            int good = 1;
            while ((arrived = *reinterpret_cast<volatile unsigned*>(count)) < want) {
                if (*reinterpret_cast<volatile int*>(err)) { good = 0; break; }
                if (++tries < kPolls) continue;
                const unsigned now = *reinterpret_cast<volatile unsigned*>(beat);
                if (now == seen_beat && arrived == seen_arrived) { atomicExch(err, 1); good = 0; break; }
                seen_beat = now;
                seen_arrived = arrived;
                tries = 0;
            }
            __threadfence();
            ok = good;
        }
        __syncthreads();
        return ok != 0;
    }
};

// epoch `epoch`'s marked chunks, replayed by the grid's threads (its records at rec / state, layout Yr -> Yw)
__device__ __noinline__ void owner_replay_marked(const SgdDev& call, const OwnerDev& own, int epoch, float alpha,
                                                 const float* Yr, float* Yw, int32_t* rec, uint64_t* state,
                                                 unsigned* beat) {
    SgdDev c = call;
    OwnerDev o = own;
    c.Y = Yw;
    o.Yr = Yr; o.n_neg = rec; o.state = state;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < o.n_chunks; q += (int64_t)gridDim.x * blockDim.x)
        if (__ldcg(&o.dirty[q])) {
            o.dirty[q] = 0;
            owner_replay<2>(c, o, (int)q, epoch, alpha, 0.0f, Beat{beat});
        }
}

// Epochs [b0, b0 + B) of the pipelined node pass in one cooperative launch: epoch k reads buffer k & 1 and writes the
// other; a grid barrier separates the epochs, and a second one follows the fallback of an epoch that marked a chunk.
// Bound by the latency of one epoch (one L2 read, the steps of the longest row, the barrier).
// 14 us per epoch of a 48-row transform and 18 of a 4096-row one, where the five operations per epoch before it took
// 68 and 76 (200k fixed rows, 14 edges per row, 100 epochs).
// Few heads are spread thin, by groups of G lanes (G a power of two up to 8): as long as every scheduler has a warp.
__global__ void __launch_bounds__(kEpochThreads) owner_epochs_kernel(const __grid_constant__ SgdDev c,
                                                           const __grid_constant__ OwnerDev o, OwnerSched sc, int b0, int B,
                                                           int G, float* buf0, float* buf1,
                                                           const int32_t* __restrict__ heads,
                                                           const int* __restrict__ n_heads, int* __restrict__ any_dirty,
                                                           unsigned* bar, unsigned* beat, int* err) {
    extern __shared__ __align__(16) unsigned char epoch_smem[];
    EpochShared& sh = *reinterpret_cast<EpochShared*>(epoch_smem);
    const int gl = threadIdx.x & (G - 1);
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x / G);
    const int64_t work = heads ? *n_heads : c.n;
    const int64_t g0 = (int64_t)blockIdx.x * (blockDim.x / G) + threadIdx.x / G;
    const int64_t gw = (int64_t)blockIdx.x * (blockDim.x / G) + (threadIdx.x & ~31) / G;   // the warp's first group
    const OwnerCoef coef(c);
    const int64_t n = c.n, n_fixed = c.n_fixed, E = c.n_edges;
    const int32_t* const tail = c.tail;
    const int64_t* const row = o.row;
    GridBarrier barrier{bar, beat, err};
    // one head per group (every transform): its row bounds stay in registers, and the first round of an epoch is made
    // between the two halves of the barrier that ends the epoch before
    const bool single = work <= groups;
    int64_t u = -1, row0 = 0, row1 = 0;
    HeadWalk walk{};
    walk.col = threadIdx.x / G;
    walk.beat.at = beat;
    bool more = false, has = false;
    auto head_at = [&](int64_t h) {
        u = heads ? (int64_t)heads[h] : h;
        row0 = row[u];
        row1 = row[u + 1];
        has = row0 < row1;
    };
    auto begin = [&](int k) {
        const int32_t* rec = o.n_neg + (int64_t)k * E;
        walk.w0 = row0; walk.row1 = row1;
        walk.stream = o.state[(int64_t)k * E + row0];   // used when an edge of the row is sampled
        walk.fill(rec, tail, sh);
        more = walk.round(rec, tail, u, n, sh);
    };
    if (single && g0 < work) {
        head_at(g0);
        if (has && gl == 0) begin(0);
    }
    __syncwarp();
    for (int k = 0; k < B; ++k) {
        const int epoch = b0 + k;
        const float alpha = sc.alpha(epoch);
        const float* const Yr = (k & 1) ? buf1 : buf0;
        float* const Yw = (k & 1) ? buf0 : buf1;
        for (int64_t hw = gw; hw < work; hw += groups) {   // uniform in the warp
            if (!single) {
                const int64_t h = hw + (threadIdx.x & 31) / G;
                has = false;
                if (h < work) head_at(h);
                if (has && gl == 0) begin(k);
                __syncwarp();
            }
            if (owner_heads(coef, Yr, Yw, o.n_neg + (int64_t)k * E, tail, n, n_fixed, u, has, walk, more, alpha, sh, G)) {
                atomicExch(&o.dirty[chunk_of(o, u)], 1);
                atomicExch(&any_dirty[k], 1);
            }
        }
        barrier.arrive();
        if (single && has && gl == 0 && k + 1 < B) begin(k + 1);
        if (!barrier.wait()) return;
        if (__ldcg(&any_dirty[k])) {
            owner_replay_marked(c, o, epoch, alpha, Yr, Yw, o.n_neg + (int64_t)k * E, o.state + (int64_t)k * E, beat);
            barrier.arrive();
            if (!barrier.wait()) return;
        }
    }
}

// resident blocks of owner_epochs_kernel, asked once per thread and device
int owner_resident_blocks() {
    static thread_local int dev_known = -1, blocks = 0;
    int dev = 0;
    MGB_CUDA(cudaGetDevice(&dev));
    if (dev != dev_known) {
        int per_sm = 0;
        MGB_CUDA(cudaFuncSetAttribute((const void*)owner_epochs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(EpochShared)));
        MGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, owner_epochs_kernel, kEpochThreads,
                                                               sizeof(EpochShared)));
        blocks = std::max(1, per_sm) * kNumSMs;
        dev_known = dev;
    }
    return blocks;
}

// bytes of records (negatives counts and head states, 12 per edge and epoch) that a batch of epochs may hold
constexpr int64_t kOwnerAheadBytes = 96LL << 20;

}  // namespace

int owner_chunk_count(int64_t n_edges, int chunk_edges) {
    const int64_t per = chunk_edges > 0 ? chunk_edges : 4096;
    return (int)std::min<int64_t>(chunk_edges > 0 ? INT32_MAX / 2 : 4096, std::max<int64_t>(1, n_edges / per));
}

// the call's flags: [0] unsorted heads, [1] a grid barrier of an earlier call gave up
static int* owner_flags(SgdWork& w, cudaStream_t s) {
    const bool fresh = w.flag.p == nullptr;
    int* flag = static_cast<int*>(w.flag.ensure(2 * sizeof(int)));
    if (fresh || !w.flags_ready) MGB_CUDA(cudaMemsetAsync(flag, 0, 2 * sizeof(int), s));
    w.flags_ready = true;
    return flag;
}

static void owner_check_timeout(int gave_up, SgdWork& w, cudaStream_t s) {
    if (!gave_up) return;
    MGB_CUDA(cudaMemsetAsync(w.flag.as<int>() + 1, 0, sizeof(int), s));
    throw Error(MG_ERR_TIMEOUT, "owner mode: a grid barrier gave up; the layout of that call is not valid");
}

bool owner_heads_sorted(const int32_t* head_dev, int64_t n_edges, SgdWork& w, cudaStream_t s) {
    if (n_edges < 2) return true;
    int* flag = owner_flags(w, s);
    MGB_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));
    owner_sorted_kernel<<<std::min(ceil_div(n_edges, 256), 4 * kNumSMs), 256, 0, s>>>(head_dev, n_edges, flag);
    MGB_LAUNCH_CHECK();
    int h[2] = {0, 0};
    MGB_CUDA(cudaMemcpyAsync(h, flag, sizeof(h), cudaMemcpyDeviceToHost, s));
    MGB_CUDA(cudaStreamSynchronize(s));
    owner_check_timeout(h[1], w, s);
    return h[0] == 0;
}

void owner_finish(SgdWork& w, cudaStream_t s) {
    if (!w.unasked) {
        MGB_CUDA(cudaStreamSynchronize(s));
        return;
    }
    int gave_up = 0;
    MGB_CUDA(cudaMemcpyAsync(&gave_up, owner_flags(w, s) + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    MGB_CUDA(cudaStreamSynchronize(s));
    w.unasked = false;
    owner_check_timeout(gave_up, w, s);
}

void owner_run(SgdDev& c, SgdWork& w, const int32_t* rev_indptr, const int32_t* rev_indices, int chunk_edges,
               int e0, int e1, float alpha0, float alpha1, float mid_w0, float mid_w1, cudaStream_t s) {
    const int64_t n = c.n, E = c.n_edges;
    const int dim = c.dim;
    const int nc = owner_chunk_count(E, chunk_edges);
    const size_t y_bytes = sizeof(float) * (size_t)(n * dim);
    OwnerDev o{};
    int64_t* row = static_cast<int64_t*>(w.o_row.ensure(sizeof(int64_t) * (n + 1)));
    int64_t* own = static_cast<int64_t*>(w.o_own.ensure(sizeof(int64_t) * (nc + 1) * 2));
    int64_t* eown = own + (nc + 1);
    o.row = row; o.own = own; o.eown = eown; o.n_chunks = nc;
    o.rev_indptr = rev_indptr; o.rev_indices = rev_indices;
    // epochs whose schedule and draws are made together: as many as the records' bound allows
    const int64_t per_epoch = 12 * std::max<int64_t>(E, 1);
    const int ahead = (int)std::max<int64_t>(1, std::min<int64_t>(e1 - e0, kOwnerAheadBytes / per_epoch));
    // (sized a quarter above the call's edges: the next request of about the same rows keeps the buffers)
    const size_t room = (size_t)((E + E / 4 + 1) * ahead);
    int32_t* rec = static_cast<int32_t*>(w.o_neg.ensure(sizeof(int32_t) * room));
    uint64_t* state = static_cast<uint64_t*>(w.o_state.ensure(sizeof(uint64_t) * room));
    o.dirty = static_cast<int*>(w.o_dirty.ensure(sizeof(int) * nc));
    float* snap = static_cast<float*>(w.o_snap.ensure(std::max<size_t>(y_bytes, sizeof(float))));
    float* const Y = c.Y;
    const bool adam = c.optimizer == 1;
    float* snap_m = nullptr; float* snap_v = nullptr; int32_t* snap_t = nullptr;
    if (adam) {
        snap_m = static_cast<float*>(w.o_snap_m.ensure(std::max<size_t>(y_bytes, sizeof(float))));
        snap_v = static_cast<float*>(w.o_snap_v.ensure(std::max<size_t>(y_bytes, sizeof(float))));
        snap_t = static_cast<int32_t*>(w.o_snap_t.ensure(sizeof(int32_t) * std::max<int64_t>(n, 1)));
    }
    o.snap_m = snap_m; o.snap_v = snap_v; o.snap_t = snap_t;
    MGB_CUDA(cudaMemsetAsync(o.dirty, 0, sizeof(int) * nc, s));
    owner_rows_kernel<<<ceil_div(n + 1, 256), 256, 0, s>>>(c.head, E, n, row);
    MGB_LAUNCH_CHECK();
    owner_chunks_kernel<<<ceil_div(nc + 1, 256), 256, 0, s>>>(c.head, E, n, nc, row, own, eown);
    MGB_LAUNCH_CHECK();
    OwnerSched sc{e0, std::max(1, e1 - e0), alpha0, alpha1, mid_w0, mid_w1, c.use_mid};
    // the pipelined node pass: 8-byte aligned 2-d rows, the power kernel without per-node b, plain steps, and heads
    // that the device holds at once (more take turns in a block's few warps: 0.68 against 0.55 ms per epoch at 300k
    // rows of 24 edges, where 20k rows take 0.08 against 0.28)
    const int64_t rows = c.n_fixed > 0 ? std::min<int64_t>(E, n - c.n_fixed) : n;
    const bool pipelined = rows <= (int64_t)owner_resident_blocks() * kEpochThreads && dim == 2 && c.kernel == 0 && !c.node_b && !adam &&
                        (reinterpret_cast<uintptr_t>(Y) % sizeof(float2)) == 0;
    int32_t* heads = nullptr;
    int* sync_words = nullptr;   // [0] barrier, [1] beat, [2] head count, [3 + k] epoch k of the batch marked a chunk
    if (pipelined) {
        sync_words = static_cast<int*>(w.o_sync.ensure(sizeof(int) * (size_t)(3 + ahead)));
        MGB_CUDA(cudaMemsetAsync(sync_words, 0, sizeof(int) * 3, s));
        if (c.n_fixed > 0) {
            heads = static_cast<int32_t*>(w.o_heads.ensure(sizeof(int32_t) * (size_t)E));
            owner_heads_kernel<<<std::min(ceil_div(E, 256), 4 * kNumSMs), 256, 0, s>>>(c.head, E, heads, sync_words + 2);
            MGB_LAUNCH_CHECK();
        }
    }
    // the two buffers of the layout: cur is read next, the other written (Adam's epochs always read the copy)
    float* cur = Y;
    float* other = snap;
    if (!adam) MGB_CUDA(cudaMemcpyAsync(snap, Y, y_bytes, cudaMemcpyDeviceToDevice, s));
    for (int b0 = e0; b0 < e1; b0 += ahead) {
        const int B = std::min(ahead, e1 - b0);
        owner_schedule_kernel<<<std::min(ceil_div(E, 256), 8 * kNumSMs), 256, 0, s>>>(c, rec, b0, B);
        MGB_LAUNCH_CHECK();
        o.n_neg = rec; o.state = state;
        if (E <= kChainThreadMaxEdges * nc)
            owner_chain_kernel<<<ceil_div((int64_t)B * nc, kChainThreads), kChainThreads, 0, s>>>(c, o, sc, b0, B);
        else
            owner_chain_warp_kernel<<<ceil_div((int64_t)B * nc, kChainWarps), 32 * kChainWarps, 0, s>>>(c, o, sc, b0, B);
        MGB_LAUNCH_CHECK();
        for (int k = 0; k < B;) {
            float alpha, mid_w;
            sgd_sched(c, b0 + k, e0, e1, alpha0, alpha1, mid_w0, mid_w1, alpha, mid_w);
            int run = 0;   // epochs from k on without mid-range pulls
            while (pipelined && k + run < B) {
                float a, mw;
                sgd_sched(c, b0 + k + run, e0, e1, alpha0, alpha1, mid_w0, mid_w1, a, mw);
                if (mw > 0.0f) break;
                ++run;
            }
            o.n_neg = rec + (int64_t)k * E;
            o.state = state + (int64_t)k * E;
            SgdDev cc = c;
            if (run > 0) {
                MGB_CUDA(cudaMemsetAsync(sync_words, 0, sizeof(int), s));
                MGB_CUDA(cudaMemsetAsync(sync_words + 3, 0, sizeof(int) * (size_t)run, s));
                // lanes per head: 8 while the warps are at most one per scheduler
                int G = 8;
                while (G > 1 && rows * G > 4LL * kNumSMs * 32) G /= 2;
                int blocks = (int)std::min<int64_t>(owner_resident_blocks(), std::max(1, ceil_div(rows * G, kEpochThreads)));
                int b = b0 + k;
                const int* n_heads = sync_words + 2;
                int* any_dirty = sync_words + 3;
                unsigned* bar = reinterpret_cast<unsigned*>(sync_words);
                unsigned* beat = bar + 1;
                int* err = owner_flags(w, s) + 1;
                void* args[] = {&cc, &o, &sc, &b, &run, &G, &cur, &other, &heads, &n_heads, &any_dirty, &bar, &beat, &err};
                MGB_CUDA(cudaLaunchCooperativeKernel((const void*)owner_epochs_kernel, dim3(blocks), dim3(kEpochThreads), args, sizeof(EpochShared), s));
                MGB_LAUNCH_CHECK();
                w.unasked = true;
                if (run & 1) std::swap(cur, other);
                k += run;
                continue;
            }
            if (adam) {
                MGB_CUDA(cudaMemcpyAsync(snap, Y, y_bytes, cudaMemcpyDeviceToDevice, s));
                MGB_CUDA(cudaMemcpyAsync(snap_m, c.adam_m, y_bytes, cudaMemcpyDeviceToDevice, s));
                MGB_CUDA(cudaMemcpyAsync(snap_v, c.adam_v, y_bytes, cudaMemcpyDeviceToDevice, s));
                MGB_CUDA(cudaMemcpyAsync(snap_t, c.adam_t, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s));
                o.Yr = snap;
            } else {
                o.Yr = cur;
                cc.Y = other;
                std::swap(cur, other);
            }
            MGB_DIM_DISPATCH(dim, owner_epoch_launch, cc, o, b0 + k, alpha, mid_w, s);
            ++k;
        }
    }
    if (cur != Y) MGB_CUDA(cudaMemcpyAsync(Y, cur, y_bytes, cudaMemcpyDeviceToDevice, s));
}

}  // namespace mgb
