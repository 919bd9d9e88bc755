// FFT-interpolated repulsion on the device (the pass of src/fftconv.cpp:58-230 and magnet/tsne.py:30-90).
//
// HBM layout (N = live grid side = n_boxes * n_interp, M = padded FFT side, Mh = M/2 + 1, Np = N rounded up
// to even):
//   W    float4 [N][N]        spread charges (1, 2^j x, 2^k y, -) per node, interleaved; zeroed by the row passes
//   WhT  float2 [3][Mh][Np]   row spectra, transposed (node row index contiguous) for the column pass
//   PhT  float2 [4][Mh][Np]   products after the inverse column transforms, same layout
//        The in-place engine holds channel 0 in WhT[0] / PhT[1] by frequency, and 2^j x W + i 2^k y W, one complex
//        field, in the M rows from WhT[1] / PhT[2] on by position (the order its stages leave)
//   phi  float  [4][N][N]     potentials per channel (planar)
//   Kt   float  [2][Mh][M]    kernel spectra K1h, K2h transposed (k1 contiguous)
//   Rt   float2 [2][Mh][M/2+1] row spectra of the two kernels (spectrum generation only)
//   tw   float2 [M]           exp(-2 pi i m / M), FP64-rounded
// GridDesc is device-resident: the grid choice is made on the device each iteration, so a captured
// iteration needs no host round trip; every pass kernel reads the live sizes from it.
#pragma once
#include "common.cuh"

namespace mgb {

namespace fft3 { struct Plan; }

struct GridDesc {
    float xmin, ymin, width, inv_width;
    int n_boxes, N, M, Mh;
    int spec_dirty;           // kernel spectra must be recomputed before the convolution
    double spec_width;        // FP64 box width the spectra are computed for (magnet/tsne.py:57)
    int tw_M;                 // length of the current twiddle table (0 = none)
    int tw_dirty;             // the twiddle table must be recomputed (M changed)
    int key_nb; long long key_w;   // spectrum cache key: (n_boxes, round(width * 1e6)) as magnet/tsne.py:51
    double sumQ;              // FP64 sum of the kernel over all pairs (self terms removed)
    float sumQ_f, inv_sumQ;   // (float)sumQ, (float)(1 / max((double)sumQ_f, 1e-12)) as magnet/tsne.py:177
    float2 up, down;          // 2^j, 2^k and their inverses of the charges (1, 2^j x, 2^k y); 1 outside the in-place engine
    unsigned peak[2];         // bits of the largest |x| and |y| while they are taken, else 0
    float mean[2];            // pending recentring of the layout (t-SNE loop)
    int recentre;             // 1: subtract mean at the next bbox pass
    int iter;                 // iteration counter of the device loop
    unsigned counter;         // last-block counters (reset by the last block)
    unsigned counter2;
};

// The in-place engine packs x W and y W as one complex field, and a transform rounds on the scale of the larger of its
// two halves: the column of the smaller values is brought next to the other, within a factor of 1.42 of the largest |x|
// and |y| (by a power of two: exact, undone where the potentials are stored). Unscaled, a layout 10 times as wide as high
// had F_y 2.4 to 3 times further from 64 bits than with a transform per field, one 1000 off the origin in x 5 to 16
// times. A column of zeros has no potential.
__device__ __forceinline__ void set_field_scale(GridDesc* g, float ax, float ay) {
    const bool scaled = ax > 0.f && ay > 0.f && ax < INFINITY && ay < INFINITY;
    const int k = scaled ? max(-120, min(120, (int)rintf(log2f(ax) - log2f(ay)))) : 0;
    const float up = __int_as_float((127 + abs(k)) << 23), down = __int_as_float((127 - abs(k)) << 23);
    g->up = make_float2(k < 0 ? up : 1.f, k > 0 ? up : 1.f);
    g->down = make_float2(ax == 0.f ? 0.f : (k < 0 ? down : 1.f), ay == 0.f ? 0.f : (k > 0 ? down : 1.f));
}

struct RepBuffers {
    int Nmax = 0, Mmax = 0, Mhmax = 0, Npmax = 0, ni = 3;
    DevBuf W, WhT, PhT, phi, Kt, Rt, tw, zpart, fft_len_table;
    DevBuf plans3;            // in-place engine (fft3.cuh) plans, indexed by M
    int Mp3max = 0;           // its largest padded length up to Mmax
    bool use3 = false;        // the in-place column pass (fftrep3.cu) runs every length these buffers see
    void alloc(int Nmax_, int Mmax_, int ni_);
};

// What the in-place engine and the t-SNE loop's kernels read of one layout (device addresses, sizes, schedule)
struct TsneSched {
    int early_iter;
    float early_exag, exag, mom0, mom1, lr, inv_dof;
    double box_width;
    int min_boxes, max_boxes, ni;
};

struct LoopDesc {
    GridDesc* g;
    float4* W; float2* WhT; float2* PhT; float* phi; float* Kt; float2* Rt; float2* tw;
    const fft3::Plan* plans; double* zpart; const int* fft_len;
    int Nmax, Npmax, Mhmax, Mmax;
    int64_t n;
    // the loop only
    float2* Ycur; float2* Ynext; float2* U; float2* G;
    const int32_t* ip; const int32_t* ix; const float* P;
    float4* box_part; double2* mean_part;
    TsneSched sch;
    double dof;
};

// the layouts of one launch: `one`, or `count` of them in device memory (at most kMaxLoops)
constexpr int kMaxLoops = 1024;
struct LoopArgs {
    LoopDesc one;
    const LoopDesc* many;
    int count;
};

// the largest of a launch's layouts
struct LoopSizes {
    int64_t n;            // points
    int Nmax, Mmax, Mp;   // grid side, FFT side, padded FFT length
    int ni;
};

// host-side next_fast_len(target, real=True) of scipy: smallest 5-smooth integer >= target
int next_5smooth(int target);
// smallest 5-smooth length >= target that the in-place engine has a plan for
int next_fft_len(int target);

// kernel launches (all asynchronous on stream s; sizes read from the device GridDesc g)
// the grid of a call on n points (none: Y may be null); in_place: the in-place engine will run it
void rep_set_grid(GridDesc* g_dev, const float2* Y, int64_t n, float xmin, float ymin, float width, int n_boxes, int ni,
                  int M, bool in_place, cudaStream_t s);
void rep_spread(const float2* Y, int64_t n, GridDesc* g, RepBuffers& b, cudaStream_t s);
void rep_prepare_device_spectra(RepBuffers& b);   // before capture: scratch of the spectrum generation
void rep_convolve(GridDesc* g, RepBuffers& b, int64_t n, cudaStream_t s);
void rep_gather_forces(const float2* Y, int64_t n, GridDesc* g, RepBuffers& b, float2* F, cudaStream_t s);
void rep_set_spectra_from_host_layout(RepBuffers& b, const float* K1h_dev, const float* K2h_dev, int M,
                                      cudaStream_t s);
void rep_twiddles(GridDesc* g, RepBuffers& b, cudaStream_t s, bool force);   // recompute tw if g->tw_dirty

// allocation-free FFTConv2D.compute on a static scratch (noalloc.cu); device arrays only
int noalloc_max_fft_side();
void fftconv_compute_noalloc(const float* K1h, const float* K2h, int M, int n_interp, const float* Y, int64_t n,
                             float xmin, float ymin, float width, int n_boxes, float* sumQ, float* F);

// in-place engine (fftrep3.cu): the three transforms over every layout of the launch
void fft3_build_plans(DevBuf& table, int Mmax, int& Mp_max);
void fft3_prepare(int Mp_max);   // shared-memory limits, before any capture
void rep_row_fwd3(const LoopArgs& a, const LoopSizes& z, cudaStream_t s);
void rep_col3(const LoopArgs& a, const LoopSizes& z, cudaStream_t s);
void rep_row_inv3(const LoopArgs& a, const LoopSizes& z, cudaStream_t s);
// kernel spectra of the layouts whose grid changed
void rep_update_spectra(const LoopArgs& a, int Mmax, cudaStream_t s);
LoopDesc rep_desc(RepBuffers& b, GridDesc* g, int64_t n);   // the FFT fields

}  // namespace mgb
