// t-SNE pass on the device: the per-iteration kernels of src/fftrep.cpp (attraction, step, update, bbox) and
// the whole optimisation loop of magnet/tsne.py:132-214 (common path) kept on the device.
#pragma once
#include "fftrep.cuh"
#include <functional>
#include <string>

namespace mgb {

// standalone kernels (one call = one reference call)
void tsne_attraction_dev(const int32_t* ip, const int32_t* ix, const float* P, const float* Y, int64_t n, int dim,
                         float dof, float* out, cudaStream_t s);
void tsne_step_dev(float* Y, float* U, float* G, const float* A, const float* F, int64_t n, int dim, float rho,
                   float inv_sumQ, float lr, float momentum, DevBuf& scratch, cudaStream_t s);
void tsne_update_dev(float* Y, float* U, float* G, const float* grad, int64_t n, int dim, float lr, float momentum,
                     DevBuf& scratch, cudaStream_t s);
void bbox_dev(const float* Y, int64_t n, float* out4_dev, DevBuf& scratch, cudaStream_t s);
void mid_spring_dev(const float* Y, const int32_t* pairs, float* grad, int64_t n, int dim, int m, float w,
                    cudaStream_t s);
void center_scale_dev(float* Y, int64_t n, int dim, double target_std, DevBuf& scratch, cudaStream_t s);

// Device-resident state of one t-SNE layout: the layout double buffer, the optimiser state, the normalised
// affinities and the repulsion buffers. One instance per stream.
struct TsneDev {
    int64_t n = 0, nnz = 0;
    int ni = 3, tpr = 8;
    float dof = 1.f;
    TsneSched sch{};
    DevBuf Ycur, Ynext, U, G, ip, ix, P, gdesc, box_part, mean_part;
    RepBuffers rb;
    cudaGraphExec_t graph = nullptr;
    bool graph_stale = false;           // it was captured with another signature
    uint64_t graph_kernels = 0;         // kernel nodes of the captured iteration
    std::string graph_sig;              // sizes, schedule and buffer addresses the graph was captured with
    // spatial order of the points (the loop of a large layout): row r of every per-point array holds the caller's
    // point perm[r]; the affinity rows and their column indices are relabelled to match. Set by reorder(),
    // undone by set_layout / get_layout, so callers always see their own order.
    bool permuted = false;
    int reorder_every = 0;              // iterations between reorders (0: never)
    DevBuf perm, perm_t, okey, ocnt, ostart, osrc, onew, olen, oip, oscan, Yt, Ut, Gt, ipt, ixt, Pt;
    ~TsneDev();
    // sizes the buffers and copies the graph (device arrays); the caller then writes its affinities, normalised to sum 1
    // (magnet/tsne.py:149-150), to P
    void init(const int32_t* ip_d, const int32_t* ix_d, int64_t n, int64_t nnz, const TsneSched& s, float dof,
              int threads_per_row, cudaStream_t st);
    void set_layout(const float* Y, bool host_ptr, cudaStream_t st);   // also resets update = 0, gains = 1
    void get_layout(float* Y, bool host_ptr, cudaStream_t st);         // applies the pending recentring
    LoopDesc desc();   // what the loop's kernels read
    void run(int n_iter, bool use_graph, cudaStream_t st);
    // plain launches with per-stage event timing; stage_ms[0..7] += stage times, grid[4] = last grid
    void run_profiled(int n_iter, cudaStream_t st, double* stage_ms, int* grid);
    // sorts the points by grid box (Morton order of the boxes of the last iteration's grid), so that the rows a
    // warp handles touch nearby nodes of the grid and nearby positions; plain launches, outside any capture
    void reorder(cudaStream_t st);
    bool reorder_due(int i) const;
    std::string signature() const;
    GridDesc* g() { return gdesc.as<GridDesc>(); }
};

// The loop's launches over the layouts of `a` (all of one n_interp).
// the first grid of every layout, from its starting positions; the later ones come out of the iterations
void loop_start(const LoopArgs& a, const LoopSizes& z, cudaStream_t st);
// one iteration; layouts [from[q], from[q + 1]) take tprs[q] lanes per row (runs of equal lanes). `side` (or null)
// takes the kernel spectra off the iteration's path (a stream of the same capture); with ev (8 events) the stage
// boundaries are recorded: grid, spread, spectra, forward rows, columns, inverse rows, gather + step.
struct LaneRun {
    int first, count, tpr;
};
void loop_iterate(const LoopArgs& a, const LoopSizes& z, const LaneRun* runs, int n_runs, cudaStream_t st,
                  cudaStream_t side, cudaEvent_t fork, cudaEvent_t join, cudaEvent_t* ev);

// a captured iteration: body(stream, side stream, fork, join) launches it; exec is made or brought up to it
void capture_loop(const std::function<void(cudaStream_t, cudaStream_t, cudaEvent_t, cudaEvent_t)>& body,
                  cudaGraphExec_t& exec, uint64_t& kernels);

}  // namespace mgb
