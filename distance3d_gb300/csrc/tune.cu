// tune.cu -- autotuner of the batch kernels' launch parameters.
//
// d3d_autotune times d3d_collide (GJK distance, EPA on the intersecting
// pairs) on the caller's sample pairs for candidate tunings and keeps the
// fastest; d3d_autotune_batches times several batches side by side as a server
// of as many slots runs them, each a CUDA graph on a stream of its own (with
// the kernels launched one by one the host sets the pace, and every candidate
// with fewer kernels wins):
//
//   stage 1  GJK threads per block {64, 128, 256} x resident warps per SM
//            {all that fit, 16} x type sorting {as set, never}, with the EPA
//            setting unchanged
//   stage 2  mixed EPA's warps per block {2, 4, 8} with the stage-1 winner
//
// A candidate that launches what an earlier one launched (a parameter that
// the forms and sizes at hand do not read) is left out, and the setting that
// was there stays unless another one is kMargin faster: the result is process
// state (d3d_set_tuning) that later launches of other sizes read too, so it is
// not to change by the noise of a timing.
//
// Each candidate runs once untimed, then three timed samples of 1-16 runs
// (CUDA events on the caller's stream); the fastest sample counts.
#include <climits>
#include <cmath>
#include <vector>

#include "capi_util.h"
#include "epa_mixed.h"
#include "gjk_impl.h"
#include "scratch.h"

namespace {

// Runs of one setting differ by up to 1 %.
constexpr float kMargin = 0.02f;

struct Problem {
    const d3d_store* store;
    const int32_t *i1, *i2;
    int64_t n;
    const d3d_gjk_options* gjk;
    const d3d_epa_options* epa;
};

// One batch's device memory, and its stream and event where batches run side by side.
struct Batch {
    void* p[12] = {};
    cudaStream_t stream = nullptr;
    cudaEvent_t done = nullptr;
    cudaGraphExec_t graph = nullptr;
};

struct Bench {
    std::vector<Batch> batches;
    size_t scratch_bytes = 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ~Bench() {
        for (Batch& b : batches) {
            for (void* q : b.p) cudaFree(q);
            if (b.graph) cudaGraphExecDestroy(b.graph);
            if (b.stream) cudaStreamDestroy(b.stream);
            if (b.done) cudaEventDestroy(b.done);
        }
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
    }
};

cudaError_t prepare(const Problem& q, int32_t batches, Bench& b, cudaStream_t st) {
    const size_t bytes[11] = {8, 8, 24, 24, 96, 1, 1, 4, 24, 1, 4};
    b.batches.resize((size_t)batches);
    cudaError_t e = cudaEventCreate(&b.e0);
    if (e == cudaSuccess) e = cudaEventCreate(&b.e1);
    for (Batch& x : b.batches) {
        for (int k = 0; k < 11 && e == cudaSuccess; ++k) e = cudaMalloc(&x.p[k], bytes[k] * (k == 0 ? 1 : (size_t)q.n));
        if (e == cudaSuccess) e = cudaMalloc(&x.p[11], b.scratch_bytes);
        if (e == cudaSuccess) e = cudaMemcpyAsync(x.p[0], &q.n, sizeof(int64_t), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess && batches > 1) e = cudaStreamCreateWithFlags(&x.stream, cudaStreamNonBlocking);
        if (e == cudaSuccess && batches > 1) e = cudaEventCreateWithFlags(&x.done, cudaEventDisableTiming);
    }
    return e;
}

int launch(const Problem& q, const Bench& b, size_t k, cudaStream_t st) {
    void* const* p = b.batches[k].p;
    return d3d_collide(q.store, q.i1 + (int64_t)k * q.n, q.i2 + (int64_t)k * q.n, q.n, static_cast<int64_t*>(p[0]),
                       q.gjk, q.epa, (double*)p[1], (double*)p[2], (double*)p[3], (double*)p[4], (int8_t*)p[5],
                       (int8_t*)p[6], (int32_t*)p[7], (double*)p[8], (int8_t*)p[9], (int32_t*)p[10], p[11],
                       b.scratch_bytes, st);
}

// The batches' graphs under the current tuning.
int capture(const Problem& q, Bench& b) {
    for (size_t k = 0; k < b.batches.size(); ++k) {
        Batch& x = b.batches[k];
        if (x.graph) cudaGraphExecDestroy(x.graph);
        x.graph = nullptr;
        int rc = k == 0 ? launch(q, b, k, x.stream) : D3D_SUCCESS;  // first use of the kernels
        if (rc) return rc;
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(x.stream, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            rc = launch(q, b, k, x.stream);
            e = cudaStreamEndCapture(x.stream, &g);
        }
        if (e == cudaSuccess && !rc) e = cudaGraphInstantiate(&x.graph, g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            d3d::set_error("d3d_autotune: %s", cudaGetErrorString(e));
            return D3D_ERR_CUDA;
        }
        if (rc) return rc;
    }
    return D3D_SUCCESS;
}

int run(const Problem& q, Bench& b, cudaStream_t st) {
    if (b.batches.size() == 1) return launch(q, b, 0, st);
    for (Batch& x : b.batches) {
        const cudaError_t e = cudaGraphLaunch(x.graph, x.stream);
        if (e != cudaSuccess) {
            d3d::set_error("d3d_autotune: %s", cudaGetErrorString(e));
            return D3D_ERR_CUDA;
        }
    }
    return D3D_SUCCESS;
}

// milliseconds per run (the fastest of three timed samples, each sample
// repeating the run until it spans about 2 ms, so that small batches are not
// timed at the events' resolution)
float time_tuning(const d3d_tuning& t, const Problem& q, Bench& b, cudaStream_t st, int* rc) {
    *rc = d3d_set_tuning(&t);
    if (!*rc && b.batches.size() > 1) *rc = capture(q, b);
    if (*rc) return -1.f;
    int reps = 1;
    float best = -1.f;
    for (int k = 0; k < 4 && !*rc; ++k) {  // sample 0: warm-up and estimate
        cudaEventRecord(b.e0, st);
        for (Batch& x : b.batches)
            if (x.stream) cudaStreamWaitEvent(x.stream, b.e0, 0);
        for (int r = 0; r < reps && !*rc; ++r) *rc = run(q, b, st);
        for (Batch& x : b.batches)
            if (x.stream) {
                cudaEventRecord(x.done, x.stream);
                cudaStreamWaitEvent(st, x.done, 0);
            }
        cudaEventRecord(b.e1, st);
        if (cudaEventSynchronize(b.e1) != cudaSuccess) {
            *rc = D3D_ERR_CUDA;
            break;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, b.e0, b.e1);
        if (k == 0) {
            reps = ms > 0.f ? (int)ceilf(2.f / ms) : 16;
            reps = reps < 1 ? 1 : (reps > 16 ? 16 : reps);
            continue;
        }
        ms /= (float)reps;
        if (best < 0.f || ms < best) best = ms;
    }
    return best;
}

// What a batch launches under tuning t.
struct Launch {
    d3d::GjkLaunch gjk;
    int epa_warps, epa64_warps;
    bool operator==(const Launch& o) const {
        return gjk == o.gjk && epa_warps == o.epa_warps && epa64_warps == o.epa64_warps;
    }
};

Launch launch_of(const d3d_tuning& t, const Problem& q) {
    const bool warp = q.epa->precision == D3D_PRECISION_MIXED && d3d::epa_warp_supported(*q.epa);
    return {q.gjk->precision == D3D_PRECISION_MIXED ? d3d::gjk_mixed_launch(*q.store, t, q.n)
                                                    : d3d::gjk_f64_launch(t, q.n),
            warp ? d3d::epa_warp_count(t, *q.epa, false) : 0,
            warp && d3d::epa_warp_supported(*q.epa, true) ? d3d::epa_warp_count(t, *q.epa, true) : 0};
}

}  // namespace

extern "C" int d3d_autotune_batches(const d3d_store* store, const int32_t* i1, const int32_t* i2, int64_t n,
                                    int32_t batches, const d3d_gjk_options* gjk, const d3d_epa_options* epa,
                                    d3d_tuning* out, void* stream) {
    int rc = d3d::check_store(store, "d3d_autotune");
    if (rc) return rc;
    D3D_REQUIRE(gjk && epa && out && i1 && i2 && n > 0 && n <= INT32_MAX, "d3d_autotune: invalid argument");
    D3D_REQUIRE(batches > 0 && batches <= 1024, "d3d_autotune: %d batches", batches);
    cudaStream_t st = d3d::as_stream(stream);
    const Problem q{store, i1, i2, n, gjk, epa};
    Bench b;
    b.scratch_bytes = d3d_collide_scratch_bytes(n, gjk, epa);
    D3D_REQUIRE(b.scratch_bytes > 0, "d3d_autotune: invalid options");
    const cudaError_t e = prepare(q, batches, b, st);
    if (e != cudaSuccess) {
        d3d::set_error("d3d_autotune: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    const d3d::SharedGpu shared((size_t)batches > d3d::kAloneBatches);
    const d3d_tuning start = d3d::tuning();
    d3d_tuning best = start;
    float start_ms = time_tuning(start, q, b, st, &rc);
    float best_ms = start_ms;
    std::vector<Launch> seen;
    if (!rc) seen.push_back(launch_of(start, q));  // after a run: the kernels' attributes are set
    auto candidate = [&](const d3d_tuning& t) {
        if (rc) return;
        const Launch l = launch_of(t, q);
        for (const Launch& x : seen)
            if (x == l) return;
        seen.push_back(l);
        const float ms = time_tuning(t, q, b, st, &rc);
        if (rc || ms >= best_ms) return;
        best_ms = ms;
        best = t;
    };
    // stage 1: the GJK kernels
    for (int bl : {start.gjk_block, 64, 128, 256})
        for (int w : {start.gjk_warps_per_sm, 0, 16})
            for (int so : {start.sort_min, INT_MAX}) {
                d3d_tuning t = start;
                t.gjk_block = bl;
                t.gjk_warps_per_sm = w;
                t.sort_min = so;
                candidate(t);
            }
    // stage 2: the mixed EPA
    for (int w : {2, 4, 8}) {
        d3d_tuning t = best;
        t.epa_warps = w;
        candidate(t);
    }
    if (!rc) start_ms = fminf(start_ms, time_tuning(start, q, b, st, &rc));
    if (!rc && best_ms > (1.f - kMargin) * start_ms) best = start;
    if (rc) {
        d3d_set_tuning(&start);
        return rc;
    }
    d3d_set_tuning(&best);
    *out = best;
    return D3D_SUCCESS;
}

extern "C" int d3d_autotune(const d3d_store* store, const int32_t* i1, const int32_t* i2, int64_t n,
                            const d3d_gjk_options* gjk, const d3d_epa_options* epa, d3d_tuning* out, void* stream) {
    return d3d_autotune_batches(store, i1, i2, n, 1, gjk, epa, out, stream);
}
