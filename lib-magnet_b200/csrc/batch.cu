// Batched t-SNE layouts: many independent layouts of uneven size optimised together (the loop of
// magnet/tsne.py:132-214 for each of them, as a loop of optimize_tsne calls would run them one after another).
//
// Every layout keeps its own device state (TsneDev: positions, optimiser state, normalised affinities, a repulsion
// grid sized for it). Every kernel of the iteration runs over all layouts of a set at once (their descriptors in device
// memory; the transforms deal the layouts' rows and columns over the device as one list), so a set costs the spread, three
// transforms, a step launch for each number of lanes per row among its layouts, and two launches for the spectra beside
// the spread, however many layouts it holds; `branches` up to kMaxSets sets run as branches of one CUDA graph, which
// the host replays once per iteration. The schedule (exaggeration, momentum) follows each layout's device-side
// iteration counter. With a branch of nine launches per layout, the launches themselves took 1.7 us each whatever the
// branches: 24 layouts of 500-5000 points, 30 iterations, took 11.1 ms, with sets 6.2 ms.
//
// A layout's grid is allocated for at most max_boxes boxes per side (by default 64 + 2 ceil(sqrt(n)), rounded up to
// a multiple of 4 and at most the caller's limit, about twice the side a t-SNE layout of n points reaches); a
// layout that grows past it is clamped to that many boxes with wider boxes, where the reference would take more.
#include "tsne.cuh"
#include <vector>
#include <memory>
#include <cmath>
#include <algorithm>

namespace mgb {

void tsne_prepare(TsneDev& d, const int32_t* indptr, const int32_t* indices, const float* P, int64_t n, int64_t nnz,
                  const mg_tsne_params& p, double box_width_exact, cudaStream_t s);

int batch_default_max_boxes(int64_t n, int limit) {
    int b = 64 + 2 * (int)std::ceil(std::sqrt((double)std::max<int64_t>(n, 1)));
    b = (b + 3) & ~3;
    return std::max(1, std::min(b, limit));
}

constexpr int kMaxSets = 2;   // sets side by side: one's latencies under another's work

struct TsneBatch {
    std::vector<std::unique_ptr<TsneDev>> layouts;   // in the caller's order
    struct Set {
        DevBuf descs;
        LoopArgs args{};
        LoopSizes sizes{};
        std::vector<LaneRun> lanes;
        cudaStream_t stream = nullptr, side = nullptr;
        cudaEvent_t fork = nullptr, join = nullptr, done = nullptr;
        ~Set() {
            for (cudaEvent_t e : {fork, join, done})
                if (e) cudaEventDestroy(e);
            for (cudaStream_t s : {stream, side})
                if (s) cudaStreamDestroy(s);
        }
    };
    std::vector<std::unique_ptr<Set>> sets;
    cudaEvent_t begin = nullptr;
    cudaGraphExec_t graph = nullptr;
    uint64_t graph_kernels = 0;
    int n_iter = 0;

    ~TsneBatch() {
        if (graph) cudaGraphExecDestroy(graph);
        if (begin) cudaEventDestroy(begin);
    }

    // the layouts dealt over the sets by size (largest first, in turn), each set's ordered by lanes per row
    void make_sets(int branches) {
        const int count = (int)layouts.size();
        const int n_sets = std::max(std::min({branches, kMaxSets, count}), ceil_div(count, kMaxLoops));
        std::vector<int> order(count);
        for (int i = 0; i < count; ++i) order[i] = i;
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return layouts[x]->nnz > layouts[y]->nnz; });
        for (int q = 0; q < n_sets; ++q) {
            std::vector<int> mine;
            for (int i = q; i < count; i += n_sets) mine.push_back(order[i]);
            std::stable_sort(mine.begin(), mine.end(), [&](int x, int y) { return layouts[x]->tpr < layouts[y]->tpr; });
            std::unique_ptr<Set> s(new Set());
            std::vector<LoopDesc> d;
            for (int i : mine) {
                TsneDev& t = *layouts[i];
                if (s->lanes.empty() || s->lanes.back().tpr != t.tpr) s->lanes.push_back(LaneRun{(int)d.size(), 0, t.tpr});
                ++s->lanes.back().count;
                d.push_back(t.desc());
                s->sizes.n = std::max(s->sizes.n, t.n);
                s->sizes.Nmax = std::max(s->sizes.Nmax, t.rb.Nmax);
                s->sizes.Mmax = std::max(s->sizes.Mmax, t.rb.Mmax);
                s->sizes.Mp = std::max(s->sizes.Mp, t.rb.Mp3max);
                s->sizes.ni = t.ni;
            }
            s->descs.ensure(sizeof(LoopDesc) * d.size());
            MGB_CUDA(cudaMemcpy(s->descs.p, d.data(), sizeof(LoopDesc) * d.size(), cudaMemcpyHostToDevice));
            s->args = LoopArgs{d[0], s->descs.as<LoopDesc>(), (int)d.size()};
            MGB_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
            MGB_CUDA(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
            for (cudaEvent_t* e : {&s->fork, &s->join, &s->done}) MGB_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
            sets.push_back(std::move(s));
        }
        MGB_CUDA(cudaEventCreateWithFlags(&begin, cudaEventDisableTiming));
    }

    // one iteration of every layout as one graph: the sets are its branches
    void capture() {
        if (graph) return;   // (the executable may be launched on any stream)
        capture_loop([&](cudaStream_t cap, cudaStream_t, cudaEvent_t, cudaEvent_t) {
            MGB_CUDA(cudaEventRecord(begin, cap));
            for (auto& s : sets) {
                MGB_CUDA(cudaStreamWaitEvent(s->stream, begin, 0));
                loop_iterate(s->args, s->sizes, s->lanes.data(), (int)s->lanes.size(), s->stream, s->side, s->fork, s->join,
                             nullptr);
                MGB_CUDA(cudaEventRecord(s->done, s->stream));
                MGB_CUDA(cudaStreamWaitEvent(cap, s->done, 0));
            }
        }, graph, graph_kernels);
    }
};

}  // namespace mgb

struct mg_tsne_batch {
    mgb::TsneBatch b;
};

using namespace mgb;

extern "C" int mg_tsne_batch_create(int count, const int64_t* n, const int64_t* nnz, const int32_t* const* indptr,
                                    const int32_t* const* indices, const float* const* P, const mg_tsne_params* p,
                                    const int* max_boxes, int branches, mg_tsne_batch** out) {
    return guard_call([&] {
        require(out != nullptr, "out must not be NULL");
        *out = nullptr;
        require(count >= 1, "the batch needs at least one layout");
        require(n && nnz && indptr && indices && P, "n, nnz, indptr, indices and P must hold `count` entries");
        require(branches >= 1 && branches <= 1024, "branches must be between 1 and 1024");
        mg_tsne_params def;
        mg_tsne_params_default(&def);
        const mg_tsne_params& pp = p ? *p : def;
        std::unique_ptr<mg_tsne_batch> h(new mg_tsne_batch());
        cudaStream_t s = current_stream();
        for (int i = 0; i < count; ++i) {
            mg_tsne_params pi = pp;
            pi.max_boxes = max_boxes ? std::min(pp.max_boxes, max_boxes[i]) : batch_default_max_boxes(n[i], pp.max_boxes);
            require(pi.max_boxes >= pi.min_boxes, "max_boxes below min_boxes for layout " + std::to_string(i));
            h->b.layouts.emplace_back(new TsneDev());
            tsne_prepare(*h->b.layouts.back(), indptr[i], indices[i], P[i], n[i], nnz[i], pi, (double)pi.box_width, s);
        }
        h->b.n_iter = pp.n_iter;
        h->b.make_sets(branches);
        MGB_CUDA(cudaStreamSynchronize(s));
        *out = h.release();
    });
}

extern "C" int mg_tsne_batch_run(mg_tsne_batch* h, float* const* Y) {
    return guard_call([&] {
        require(h != nullptr && Y != nullptr, "batch and Y must not be NULL");
        auto& b = h->b;
        cudaStream_t s = current_stream();
        for (size_t i = 0; i < b.layouts.size(); ++i) {
            require(Y[i] != nullptr, "Y must hold one (n, 2) array per layout");
            b.layouts[i]->set_layout(Y[i], !is_device_ptr(Y[i]), s);
        }
        if (b.n_iter > 0) {
            b.capture();
            for (auto& q : b.sets) loop_start(q->args, q->sizes, s);
            for (int it = 0; it < b.n_iter; ++it) {
                MGB_CUDA(cudaGraphLaunch(b.graph, s));
                count_launch(b.graph_kernels);
            }
        }
        for (size_t i = 0; i < b.layouts.size(); ++i) b.layouts[i]->get_layout(Y[i], !is_device_ptr(Y[i]), s);
        MGB_CUDA(cudaStreamSynchronize(s));
    });
}

extern "C" int mg_tsne_batch_size(const mg_tsne_batch* h, int* count, uint64_t* kernels_per_iteration) {
    return guard_call([&] {
        require(h != nullptr, "batch must not be NULL");
        if (count) *count = (int)h->b.layouts.size();
        if (kernels_per_iteration) *kernels_per_iteration = h->b.graph_kernels;
    });
}

extern "C" void mg_tsne_batch_destroy(mg_tsne_batch* h) {
    delete h;
}
