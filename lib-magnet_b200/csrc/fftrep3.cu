// The FFT repulsion's three transforms on the in-place engine (fft3.cuh): forward rows, columns with the kernel
// products, inverse rows (src/fftconv.cpp:124-199), and the FP64 Z of :226-229.
//
// The three real charge fields run as two transforms. x W and y W are packed as one complex field 2^j x W +
// i 2^k y W (set_field_scale): its column products with the real kernel spectrum give 2^j phi_2 + i 2^k phi_3, so nothing is ever
// separated and its spectrum stays in the order the stages leave (row position p of the transposed buffer holds frequency freq_of_pos(p)). The
// charge field W needs its own spectrum for Z; two of its rows share a transform, separated into half spectra after
// the forward rows and rebuilt before the inverse ones.
//
// Work items: rows by pairs (the complex field) or fours (W), columns by position (the complex field) or frequency (W),
// one per block at a time. The items of all layouts of a launch are one list, dealt over the resident blocks.
//
//   columns: the first forward stage reads the live rows (g < N) from global memory, the last inverse stage writes the
//   live rows, so a column costs 2 (S - 1) shared-memory passes per transform and no reordering pass.
// Output convention as the one-radix engine: PhT = unnormalised inverse (M x the circular convolution).
//
// Bound by the scattered 16 and 32 byte transposed accesses (rows) and by the latency of the stages at 4 to 6 warps per
// scheduler (columns). Packing the fields took a third of the transforms' work off the columns and the separation off
// the rows; M = 4320: forward rows 133 to 131 us, columns 255 to 231, inverse rows 166 to 153; M = 2400: 76 to 50, 96 to
// 87, 89 to 59.
#include "fftrep.cuh"
#include "fft3.cuh"
#include <vector>
#include <algorithm>

namespace mgb {

namespace {

constexpr int kColThreads = 192;
constexpr int kRowThreads = 256;
// Blocks per SM the registers are capped for (80 a thread in the columns, 128 in the rows). A loop's buffers are sized
// for its largest length (M = 6000: 50 KB a column, 100 KB a row block), so more row blocks would not fit beside each
// other; at M = 4320 3 x 256 and 4 x 128 threads took 142 and 147 us forward, 169 and 208 us inverse, against 127 and
// 157 us.
constexpr int kColBlocks = 4;
constexpr int kRowBlocks = 2;

// ---------------------------------------------------------------------------------------------- items
// the launch's items: layout l holds items [first[l], first[l + 1])
struct Items {
    int first[kMaxLoops + 1];
};

// items_of(N, M) per layout; called by the whole block
template <bool MANY, class F>
__device__ __forceinline__ void list_items(const LoopArgs& a, Items& it, F items_of) {
    if (!MANY) {
        if (threadIdx.x == 0) {
            it.first[0] = 0;
            it.first[1] = items_of(a.one.g->N, a.one.g->M);
        }
        __syncthreads();
        return;
    }
    for (int l = threadIdx.x; l < a.count; l += blockDim.x) {
        const GridDesc* g = a.many[l].g;
        it.first[l + 1] = items_of(g->N, g->M);
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // running sums: 32 runs of consecutive layouts
        const int per = (a.count + 31) / 32, b = threadIdx.x * per, e = min(a.count, b + per);
        int run = 0;
        for (int l = b; l < e; ++l) run += it.first[l + 1];
        int x = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)threadIdx.x >= o) x += y;
        }
        int acc = x - run;
        for (int l = b; l < e; ++l) { acc += it.first[l + 1]; it.first[l + 1] = acc; }
        if (threadIdx.x == 0) it.first[0] = 0;
    }
    __syncthreads();
}

// the layout of an item
__device__ __forceinline__ int layout_of(const Items& it, int count, int item) {
    int lo = 0, hi = count;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (it.first[mid] <= item) lo = mid; else hi = mid;
    }
    return lo;
}

// The descriptor of an item's layout: the launch's own (constant operands), or with several layouts a copy in shared
// memory (held in registers, its pointers were spilled around every stage).
template <bool MANY>
__device__ __forceinline__ const LoopDesc& desc_of(const LoopArgs& a, const Items& items, int at, int& item, int& have,
                                                   LoopDesc& held) {
    if constexpr (!MANY) {
        item = at;
        return a.one;
    } else {
        const int l = layout_of(items, a.count, at);
        item = at - items.first[l];
        if (l != have) {   // (a barrier has ended the item before)
            for (int w = threadIdx.x; w < (int)(sizeof(LoopDesc) / sizeof(int)); w += blockDim.x)
                reinterpret_cast<int*>(&held)[w] = reinterpret_cast<const int*>(a.many + l)[w];
            __syncthreads();
            have = l;
        }
        return held;
    }
}

// the block's copy of the plan of its item
__device__ __forceinline__ void load_plan(const fft3::Plan* plans, int M, fft3::Plan& p, int& have) {
    if (have != M) {
        for (int w = threadIdx.x; w < (int)(sizeof(fft3::Plan) / sizeof(int)); w += blockDim.x)
            reinterpret_cast<int*>(&p)[w] = reinterpret_cast<const int*>(plans + M)[w];
        __syncthreads();
        have = M;
    }
}

// ---------------------------------------------------------------------------------------------- columns
// element n of a column at a
struct ColLoad {
    const float2* a;
    __device__ __forceinline__ float2 operator()(int, int n) const { return a[n]; }
};
struct ColStore {
    float2* a;
    __device__ __forceinline__ void operator()(int, int n, float2 v) const { a[n] = v; }
};

// A real kernel spectrum along a column. Frequencies k2 past M / 2 read the half spectrum mirrored (kMirror,
// K(k1, k2) = K(-k1, -k2)); in the complex field's columns 0 and M / 2 the two halves are averaged (kMean), which is
// what dropping the imaginary parts of those columns does to a real field.
constexpr int kPlain = 0, kMirror = 1, kMean = 2;

// last forward stage, product with one real kernel spectrum, first inverse stage (in place)
template <int R>
__device__ __noinline__ void middle1(const fft3::Plan& p, const float* __restrict__ K, int mode) {
    float2* const A = fft3::buffers();
    const int pb = p.padR ? R + 1 : R;
    const int nb = p.M / R;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        const int base = b * pb;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = A[base + r];
        fft3::dft_fwd<R>(v);
        // frequency f of the column, or M - f (0 stays 0): a step from the first, and its end only where f is 0
        const int fb = fft3::base_freq(p, b);
        const int f0 = mode == kMirror ? p.M - fb : fb, step = mode == kMirror ? -nb : nb;
        float kv[R];
#pragma unroll
        for (int q = 0; q < R; ++q) kv[q] = __ldg(&K[q == 0 && f0 == p.M ? 0 : f0 + step * q]);
        if (mode == kMean)
            for (int q = 0; q < R; ++q) { const int f = fb + nb * q; kv[q] = 0.5f * (kv[q] + __ldg(&K[f ? p.M - f : 0])); }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = fft::cscale(v[q], kv[q]);
        fft3::dft_inv<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) A[base + r] = v[r];
    }
}

// the charge field: the last forward stage, this thread's share of sum K1 |X|^2 (for Z), the product with K2 and the
// first inverse stage (in place in A); returns the share
template <int R>
__device__ __noinline__ double middle2(const fft3::Plan& p, const float* __restrict__ K1, const float* __restrict__ K2) {
    float2* const A = fft3::buffers();
    const int pb = p.padR ? R + 1 : R;
    const int nb = p.M / R;
    double zs = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        const int base = b * pb;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = A[base + r];
        fft3::dft_fwd<R>(v);
        const int fb = fft3::base_freq(p, b);
        float zt = 0.f;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int f = fb + nb * q;
            zt += __ldg(&K1[f]) * (v[q].x * v[q].x + v[q].y * v[q].y);
            v[q] = fft::cscale(v[q], __ldg(&K2[f]));
        }
        zs += (double)zt;
        fft3::dft_inv<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) A[base + r] = v[r];
    }
    return zs;
}

__device__ __forceinline__ double middle2_dispatch(int R, const fft3::Plan& p, const float* K1, const float* K2) {
    switch (R) {
        case 2: return middle2<2>(p, K1, K2);
        case 3: return middle2<3>(p, K1, K2);
        case 4: return middle2<4>(p, K1, K2);
        case 5: return middle2<5>(p, K1, K2);
        case 6: return middle2<6>(p, K1, K2);
        case 8: return middle2<8>(p, K1, K2);
        case 9: return middle2<9>(p, K1, K2);
        case 10: return middle2<10>(p, K1, K2);
        case 12: return middle2<12>(p, K1, K2);
        case 15: return middle2<15>(p, K1, K2);
        case 16: return middle2<16>(p, K1, K2);
        case 18: return middle2<18>(p, K1, K2);
        default: return middle2<20>(p, K1, K2);
    }
}

// FP64 sum over the block (in its first thread)
__device__ __forceinline__ double block_sum(double x, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    return s;
}

template <bool MANY>
__global__ void __launch_bounds__(kColThreads, kColBlocks) col3_kernel(const __grid_constant__ LoopArgs a) {
    __shared__ Items items;
    __shared__ fft3::Plan p;
    __shared__ LoopDesc held;
    __shared__ double red[kColThreads / 32];
    __shared__ int last;
    // the charge field's columns first, so that the Z shares are ready early
    list_items<MANY>(a, items, [](int, int M) { return M / 2 + 1 + M; });
    int have = -1, have_l = -1;
    int N = MANY ? 0 : a.one.g->N, M = MANY ? 0 : a.one.g->M;
    const int total = items.first[MANY ? a.count : 1];
    for (int at = blockIdx.x; at < total; at += gridDim.x) {
        int item;
        const LoopDesc& L = desc_of<MANY>(a, items, at, item, have_l, held);
        if (MANY) { N = L.g->N; M = L.g->M; }
        const int Mh = M / 2 + 1;
        load_plan(L.plans, M, p, have);
        const int S = p.S, R0 = p.st[0].R, RS = p.st[S - 1].R;
        const bool charge = item < Mh;
        const int row = charge ? item : item - Mh;                     // row of the transposed buffers
        const int f2 = charge ? row : fft3::freq_of_pos(p, row);       // the column's frequency
        const int k = f2 < Mh ? f2 : M - f2;
        const int mode = charge ? kPlain : (f2 >= Mh ? kMirror : (k == 0 || 2 * k == M ? kMean : kPlain));
        const float2* src = L.WhT + ((size_t)(charge ? 0 : L.Mhmax) + row) * L.Npmax;
        float2* dst = L.PhT + ((size_t)(charge ? L.Mhmax : 2 * L.Mhmax) + row) * L.Npmax;
        const float* K2 = L.Kt + ((size_t)L.Mhmax + k) * L.Mmax;
        const float2* tw = L.tw;
        MGB_FFT3_RADIX_DISPATCH(R0, fft3::dif_first, p, 0, 0, 1, ColLoad{src}, N, tw);
        __syncthreads();
        for (int s = 1; s < S - 1; ++s) {
            MGB_FFT3_RADIX_DISPATCH(p.st[s].R, fft3::dif_mid, p, s, 0, 0, 1, tw);
            __syncthreads();
        }
        if (charge) {
            const double z = block_sum(middle2_dispatch(RS, p, L.Kt + (size_t)k * L.Mmax, K2), red);
            if (threadIdx.x == 0) {
                const bool single = (k == 0) || ((M & 1) == 0 && k == M / 2);
                L.zpart[k] = single ? z : 2.0 * z;
                __threadfence();
                last = atomicAdd(&L.g->counter, 1u) == (unsigned)(Mh - 1);
            }
            __syncthreads();
            if (last) {
                // the block that finishes the layout's last share: Z = sum of the shares / M^2 - n
                __threadfence();
                double x = 0.0;
                for (int q = threadIdx.x; q < Mh; q += blockDim.x) x += __ldcg(&L.zpart[q]);
                x = block_sum(x, red);
                if (threadIdx.x == 0) {
                    const double sumQ = x / ((double)M * (double)M) - (double)L.n;
                    L.g->sumQ = sumQ;
                    const float sf = (float)sumQ;
                    L.g->sumQ_f = sf;
                    L.g->inv_sumQ = (float)(1.0 / fmax((double)sf, 1e-12));
                    L.g->counter = 0u;
                }
            }
        } else {
            MGB_FFT3_RADIX_DISPATCH(RS, middle1, p, K2, mode);
            __syncthreads();
        }
        for (int s = S - 2; s >= 1; --s) {
            MGB_FFT3_RADIX_DISPATCH(p.st[s].R, fft3::dit_mid, p, s, 0, 0, 1, tw);
            __syncthreads();
        }
        MGB_FFT3_RADIX_DISPATCH(R0, fft3::dit_last, p, 0, 0, 1, ColStore{dst}, N, tw);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------- rows
// Two buffers per block. Items of a layout: the charge field's rows by fours (first, they are the longer ones), then the
// complex field's rows by pairs. The transposed spectra are read and written 16 (a pair of complex rows) or 32 (four
// rows' half spectra) contiguous bytes per frequency.

// rows g0 + 2t and g0 + 2t + 1 of the charges, packed as one complex row (rows at or past N read as zero)
struct ChargeLoad {
    const float4* W;
    int pitch, g0, N;
    __device__ __forceinline__ float2 operator()(int t, int n) const {
        const int ga = g0 + 2 * t, gb = ga + 1;
        const float x = ga < N ? W[(size_t)ga * pitch + n].x : 0.f;
        const float y = gb < N ? W[(size_t)gb * pitch + n].x : 0.f;
        return make_float2(x, y);
    }
};
// row g0 + t of the complex field
struct FieldLoad {
    const float4* W;
    int pitch, g0;
    __device__ __forceinline__ float2 operator()(int t, int n) const {
        const float4 v = W[(size_t)(g0 + t) * pitch + n];
        return make_float2(v.y, v.z);
    }
};

// potential 1 of rows g0 + 2t (Re) and g0 + 2t + 1 (Im), scaled by 1 / M^2
struct ChargeStore {
    float* phi;
    int pitch, g0, N;
    float scale;
    __device__ __forceinline__ void operator()(int t, int n, float2 v) const {
        const int ga = g0 + 2 * t, gb = ga + 1;
        if (ga < N) phi[(size_t)ga * pitch + n] = v.x * scale;
        if (gb < N) phi[(size_t)gb * pitch + n] = v.y * scale;
    }
};
// potentials 2 (Re, times 2^j) and 3 (Im, times 2^k) of row g0 + t
struct FieldStore {
    float* phi2;
    float* phi3;
    int pitch, g0;
    float scale2, scale3;   // 2^-j / M^2, 2^-k / M^2
    __device__ __forceinline__ void operator()(int t, int n, float2 v) const {
        const size_t at = (size_t)(g0 + t) * pitch + n;
        phi2[at] = v.x * scale2;
        phi3[at] = v.y * scale3;
    }
};

__device__ __forceinline__ int row_items(int N) { return (N + 3) / 4 + (N + 1) / 2; }

template <bool MANY>
__global__ void __launch_bounds__(kRowThreads, kRowBlocks) row_fwd3_kernel(const __grid_constant__ LoopArgs a) {
    __shared__ Items items;
    __shared__ fft3::Plan p;
    __shared__ LoopDesc held;
    list_items<MANY>(a, items, [](int N, int) { return row_items(N); });
    int have = -1, have_l = -1;
    int N = MANY ? 0 : a.one.g->N, M = MANY ? 0 : a.one.g->M;
    const int total = items.first[MANY ? a.count : 1];
    float2* const A = fft3::buffers();
    for (int at = blockIdx.x; at < total; at += gridDim.x) {
        int item;
        const LoopDesc& L = desc_of<MANY>(a, items, at, item, have_l, held);
        if (MANY) { N = L.g->N; M = L.g->M; }
        const int Mh = M / 2 + 1;
        load_plan(L.plans, M, p, have);
        float2* const B = A + p.Mp;
        const int fours = (N + 3) / 4;
        const bool charge = item < fours;
        const int g0 = charge ? 4 * item : 2 * (item - fours);
        const int nbuf = g0 + (charge ? 2 : 1) < N ? 2 : 1;
        const float2* tw = L.tw;
        if (charge) {
            MGB_FFT3_RADIX_DISPATCH(p.st[0].R, fft3::dif_first, p, 0, p.Mp, nbuf, ChargeLoad{L.W, L.Nmax, g0, N}, N, tw);
        } else {
            MGB_FFT3_RADIX_DISPATCH(p.st[0].R, fft3::dif_first, p, 0, p.Mp, nbuf, FieldLoad{L.W, L.Nmax, g0}, N, tw);
        }
        __syncthreads();
        for (int s = 1; s < p.S; ++s) {
            MGB_FFT3_RADIX_DISPATCH(p.st[s].R, fft3::dif_mid, p, s, 0, p.Mp, nbuf, tw);
            __syncthreads();
        }
        if (charge) {
            // rows a, b of a pair from Z_k and Z_{-k}: (Z_k + conj Z_{-k}) / 2 and (Z_k - conj Z_{-k}) / 2i; walked in
            // position order (consecutive threads read consecutive positions), frequencies past M/2 skipped
            for (int pos = threadIdx.x; pos < M; pos += blockDim.x) {
                const int k = fft3::freq_of_pos(p, pos);
                if (k >= Mh) continue;
                const int pk = p.padR ? pos + fft3::udiv(pos, p.mpad) : pos;
                const int pm = fft3::pos_of_freq(p, k == 0 ? 0 : M - k);
                float2* dst = L.WhT + (size_t)k * L.Npmax + g0;
                for (int q = 0; q < nbuf; ++q) {
                    const float2* buf = q ? B : A;
                    const float2 zk = buf[pk], zm = buf[pm];
                    reinterpret_cast<float4*>(dst)[q] = make_float4(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y),
                                                                    0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
                }
            }
        } else {
            float2* dst = L.WhT + (size_t)L.Mhmax * L.Npmax + g0;
#pragma unroll 4
            for (int pos = threadIdx.x; pos < M; pos += blockDim.x) {
                const int pk = p.padR ? pos + fft3::udiv(pos, p.mpad) : pos;
                const float2 va = A[pk], vb = nbuf > 1 ? B[pk] : make_float2(0.f, 0.f);
                *reinterpret_cast<float4*>(dst + (size_t)pos * L.Npmax) = make_float4(va.x, va.y, vb.x, vb.y);
            }
        }
        __syncthreads();
    }
}

// The inverse rows; the complex field's items also zero their rows of W for the next spread (every forward row has run).
template <bool MANY>
__global__ void __launch_bounds__(kRowThreads, kRowBlocks) row_inv3_kernel(const __grid_constant__ LoopArgs a) {
    __shared__ Items items;
    __shared__ fft3::Plan p;
    __shared__ LoopDesc held;
    list_items<MANY>(a, items, [](int N, int) { return row_items(N); });
    int have = -1, have_l = -1;
    int N = MANY ? 0 : a.one.g->N, M = MANY ? 0 : a.one.g->M;
    const int total = items.first[MANY ? a.count : 1];
    float2* const A = fft3::buffers();
    for (int at = blockIdx.x; at < total; at += gridDim.x) {
        int item;
        const LoopDesc& L = desc_of<MANY>(a, items, at, item, have_l, held);
        if (MANY) { N = L.g->N; M = L.g->M; }
        const int Mh = M / 2 + 1;
        load_plan(L.plans, M, p, have);
        float2* const B = A + p.Mp;
        const int fours = (N + 3) / 4;
        const bool charge = item < fours;
        const int g0 = charge ? 4 * item : 2 * (item - fours);
        const int nbuf = g0 + (charge ? 2 : 1) < N ? 2 : 1;
        const float2* tw = L.tw;
        const float scale = 1.f / ((float)M * (float)M);
        const size_t plane = (size_t)L.Nmax * L.Nmax;
        // the spectra enter in position order (consecutive threads write consecutive positions)
        if (charge) {
            // the position's frequency from the half spectra of the rows a, b of each pair: a + i b, past M / 2
            // conj a + i conj b of its mirror (Hermitian extension, DC and Nyquist imaginary parts dropped as a c2r does;
            // src/fftconv.cpp:176, 188-198)
            const bool even = (M & 1) == 0;
#pragma unroll 2
            for (int up = threadIdx.x; up < M; up += blockDim.x) {
                const int k = fft3::freq_of_pos(p, up);
                const int kk = k < Mh ? k : M - k;
                const float4* src = reinterpret_cast<const float4*>(L.PhT + ((size_t)L.Mhmax + kk) * L.Npmax + g0);
                const int pos = p.padR ? up + fft3::udiv(up, p.mpad) : up;
                for (int q = 0; q < nbuf; ++q) {
                    const float4 v = src[q];
                    float2 x = make_float2(v.x, v.y), y = make_float2(v.z, v.w);
                    if (g0 + 2 * q + 1 >= N) y = make_float2(0.f, 0.f);   // no row b: nothing was written there
                    if (kk == 0 || (even && kk == M / 2)) { x.y = 0.f; y.y = 0.f; }
                    if (k >= Mh) { x.y = -x.y; y.y = -y.y; }
                    (q ? B : A)[pos] = make_float2(x.x - y.y, x.y + y.x);
                }
            }
        } else {
            const float2* src = L.PhT + (size_t)2 * L.Mhmax * L.Npmax + g0;
#pragma unroll 4
            for (int up = threadIdx.x; up < M; up += blockDim.x) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(src + (size_t)up * L.Npmax));
                const int pos = p.padR ? up + fft3::udiv(up, p.mpad) : up;
                A[pos] = make_float2(v.x, v.y);
                if (nbuf > 1) B[pos] = make_float2(v.z, v.w);
            }
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int q = 0; q < nbuf; ++q)
                for (int n = threadIdx.x; n < N; n += blockDim.x) L.W[(size_t)(g0 + q) * L.Nmax + n] = zero;
        }
        __syncthreads();
        for (int s = p.S - 1; s >= 1; --s) {
            MGB_FFT3_RADIX_DISPATCH(p.st[s].R, fft3::dit_mid, p, s, 0, p.Mp, nbuf, tw);
            __syncthreads();
        }
        if (charge) {
            MGB_FFT3_RADIX_DISPATCH(p.st[0].R, fft3::dit_last, p, 0, p.Mp, nbuf,
                                    ChargeStore{L.phi + plane, L.Nmax, g0, N, scale}, N, tw);
        } else {
            MGB_FFT3_RADIX_DISPATCH(p.st[0].R, fft3::dit_last, p, 0, p.Mp, nbuf,
                                    FieldStore{L.phi + 2 * plane, L.phi + 3 * plane, L.Nmax, g0, scale * L.g->down.x, scale * L.g->down.y}, N, tw);
        }
        __syncthreads();
    }
}

}  // namespace

// Plans of every 5-smooth length up to Mmax (table indexed by M; S = 0 where there is none) and the largest
// padded length among them.
void fft3_build_plans(DevBuf& table, int Mmax, int& Mp_max) {
    std::vector<fft3::Plan> plans((size_t)Mmax + 1);
    Mp_max = 0;
    for (int M = 4; M <= Mmax; ++M) {
        if (!fft::is_5smooth(M)) continue;
        if (fft3::make_plan(M, plans[M])) Mp_max = std::max(Mp_max, plans[M].Mp);
    }
    table.ensure(plans.size() * sizeof(fft3::Plan));
    MGB_CUDA(cudaMemcpy(table.p, plans.data(), plans.size() * sizeof(fft3::Plan), cudaMemcpyHostToDevice));
}

namespace {
size_t col3_smem(int Mp) { return (size_t)Mp * sizeof(float2); }       // one transform per column block
size_t row3_smem(int Mp) { return (size_t)2 * Mp * sizeof(float2); }   // two per row block

// Threads per block by the largest length of the launch: short transforms have few butterflies per stage (12 of length
// 144), so a batch of small layouts runs more and smaller blocks.
int threads_for(int Mmax, int full) { return Mmax <= 1536 ? 64 : full; }

// resident blocks of a kernel for a buffer size and block size
int resident(const void* fn, int threads, size_t smem) {
    struct Known { const void* fn; int dev, threads, blocks; size_t smem; };
    static thread_local std::vector<Known> known;   // per thread: host threads may drive layouts side by side
    int dev = 0;
    MGB_CUDA(cudaGetDevice(&dev));
    for (const Known& k : known)
        if (k.fn == fn && k.dev == dev && k.threads == threads && k.smem == smem) return k.blocks;
    int per_sm = 0;
    MGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    if (known.size() >= 64) known.clear();
    known.push_back(Known{fn, dev, threads, std::max(1, per_sm) * kNumSMs, smem});
    return known.back().blocks;
}

template <class K>
void launch(K one, K many, const LoopArgs& a, int Mmax, int full, size_t smem, int64_t items, cudaStream_t s) {
    K fn = a.many ? many : one;
    const int threads = threads_for(Mmax, full);
    const int blocks = (int)std::min<int64_t>(resident((const void*)fn, threads, smem), std::max<int64_t>(1, a.count * items));
    fn<<<blocks, threads, smem, s>>>(a);
    MGB_LAUNCH_CHECK();
}
}  // namespace

// raises the kernels' shared-memory limits; called when buffers are sized, before any stream capture
void fft3_prepare(int Mp_max) {
    int dev = 0, optin = 0;
    MGB_CUDA(cudaGetDevice(&dev));
    static thread_local int done_dev = -1;   // per thread: host threads may drive layouts side by side
    MGB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes f;
    for (const void* fn : {(const void*)col3_kernel<false>, (const void*)row_fwd3_kernel<false>, (const void*)row_inv3_kernel<false>,
                           (const void*)col3_kernel<true>, (const void*)row_fwd3_kernel<true>, (const void*)row_inv3_kernel<true>}) {
        MGB_CUDA(cudaFuncGetAttributes(&f, fn));
        require(row3_smem(Mp_max) + f.sharedSizeBytes <= (size_t)optin, "FFT side too large for the row engine");
        if (done_dev != dev)
            MGB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)f.sharedSizeBytes));
    }
    done_dev = dev;
}

void rep_row_fwd3(const LoopArgs& a, const LoopSizes& z, cudaStream_t s) {
    launch(row_fwd3_kernel<false>, row_fwd3_kernel<true>, a, z.Mmax, kRowThreads, row3_smem(z.Mp), z.Nmax + 1, s);
}
void rep_row_inv3(const LoopArgs& a, const LoopSizes& z, cudaStream_t s) {
    launch(row_inv3_kernel<false>, row_inv3_kernel<true>, a, z.Mmax, kRowThreads, row3_smem(z.Mp), z.Nmax + 1, s);
}
void rep_col3(const LoopArgs& a, const LoopSizes& z, cudaStream_t s) {
    launch(col3_kernel<false>, col3_kernel<true>, a, z.Mmax, kColThreads, col3_smem(z.Mp), 2LL * z.Mmax, s);
}

}  // namespace mgb
