// gjk.cu -- the plain FP64 GJK drop-in: batched distance and intersection, a
// pool of pairs per block (gjk_pool.cuh), and the distance with MeshGraph vertex
// caching, one thread per pair.  Compiled with -fmad=false so that the arithmetic is
// the reference's rounding sequence (see d3d_device.cuh); the results are the
// reference's bit for bit.
#include "capi_util.h"
#include "gjk_impl.h"
#include "gjk_out.cuh"
#include "gjk_pool.cuh"
#include "persist.cuh"
#include "scratch.h"
#include "jolt.cuh"

namespace {

using namespace d3d;

// The reference's loop, one lane per pair, with its MeshGraph vertex caching: the mesh
// supports of pair k start from mesh_cache[2k] (collider i1[k]) and
// mesh_cache[2k+1] (collider i2[k]), -1 meaning the mesh's start vertex, and
// leave there the vertex their last call returned, as the reference's support
// object keeps it (mesh.py:84-85).  One thread per pair, in input order;
// entries of non-mesh colliders pass through unchanged.
__global__ void __launch_bounds__(128) k_gjk_distance_f64_cached(d3d_store s, const int32_t* __restrict__ i1,
                                                                 const int32_t* __restrict__ i2, int64_t n,
                                                                 d3d_gjk_options opt, DistanceOut o,
                                                                 int32_t* __restrict__ mesh_cache) {
    __shared__ double rows[24 * 128];
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int a = i1[k], b = i2[k];
    if (!pair_ok(s, a, b)) {
        store_bad_index(o, k);
        return;
    }
    const JoltEps<double> E = reference_eps<double>();
    GjkLoop<double, SmemRows<double, 128>> g;
    g.S.R.base = rows + threadIdx.x;
    simplex_clear(g.S);
    const d3 dir = mk(1.0, 0.0, 0.0);
    gjk_begin(g, dir, dot(dir, dir), DBL_MAX);
    int cache[2] = {mesh_cache[2 * k], mesh_cache[2 * k + 1]};
    const double tol_sq = opt.tolerance * opt.tolerance;
    while (!gjk_step<double>(g, s, a, b, tol_sq, opt.max_distance_squared, opt.max_iterations, E, cache)) {
    }
    GjkResult<double> r;
    gjk_end(g, opt.sanity_check, E, r);
    store_result(o, k, r, g.S);
    mesh_cache[2 * k] = cache[0];
    mesh_cache[2 * k + 1] = cache[1];
}

// Pairs (and threads) per block of the pool kernel.
constexpr int kPool = 256;

template <int PQ>
int pool_blocks(const d3d_tuning& t, int64_t n) {
    // a block per pair for the smallest batches: their pairs run side by side
    return persistent_blocks((const void*)pool::k_gjk_pool<kPool, PQ>, kPool, launch_items(n * kPool, n),
                             blocks_per_sm(t, kPool), (int)sizeof(pool::Mem<kPool, PQ>));
}

template <int PQ>
int launch_pool(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* order, int64_t n,
                const unsigned long long* n_dev, unsigned long long* cursor, const d3d_gjk_options& opt,
                const DistanceOut& o, int8_t* hits, cudaStream_t stream) {
    const void* fn = (const void*)pool::k_gjk_pool<kPool, PQ>;
    const int smem = (int)sizeof(pool::Mem<kPool, PQ>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) {
        set_error("FP64 GJK: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    pool::k_gjk_pool<kPool, PQ><<<pool_blocks<PQ>(tuning(), n), kPool, smem, stream>>>(store, i1, i2, order, n, n_dev, cursor, opt, o, hits);
    return check_launch(PQ == 4 ? "d3d_gjk_distance" : "d3d_gjk_intersection");
}

}  // namespace

extern "C" int d3d_gjk_distance(const d3d_store* store, const int32_t* i1, const int32_t* i2, int64_t n,
                                const d3d_gjk_options* options, double* dist, double* cp1, double* cp2,
                                double* simplex, int8_t* n_simplex, int8_t* status, int32_t* iterations,
                                void* stream) {
    int rc = d3d::check_store(store, "d3d_gjk_distance");
    if (rc) return rc;
    D3D_REQUIRE(options, "d3d_gjk_distance: null options");
    D3D_REQUIRE(n >= 0, "d3d_gjk_distance: n < 0");
    D3D_REQUIRE(options->max_iterations >= 1, "d3d_gjk_distance: max_iterations < 1");
    D3D_REQUIRE(options->precision == D3D_PRECISION_FP64 || options->precision == D3D_PRECISION_MIXED,
                "d3d_gjk_distance: unknown precision %d", options->precision);
    if (n == 0) return D3D_SUCCESS;
    D3D_REQUIRE(i1 && i2 && dist && cp1 && cp2 && simplex && n_simplex && status,
                "d3d_gjk_distance: null pointer");
    if (options->precision == D3D_PRECISION_MIXED)
        return d3d::gjk_distance_mixed(*store, i1, i2, n, *options, dist, cp1, cp2, simplex, n_simplex, status,
                                       iterations, d3d::as_stream(stream));
    cudaStream_t st = d3d::as_stream(stream);
    void* block = nullptr;
    rc = d3d::scratch_alloc(&block, d3d::gjk_f64_scratch_bytes(n), st);
    if (rc) return rc;
    DistanceOut o{dist, cp1, cp2, simplex, n_simplex, status, iterations};
    rc = d3d::gjk_f64_run(*store, i1, i2, n, nullptr, *options, o, block, st);
    d3d::scratch_free(block, st);
    return rc;
}

namespace d3d {

GjkLaunch gjk_f64_launch(const d3d_tuning& t, int64_t n) { return {0, 0, pool_blocks<4>(t, n), n >= t.sort_min}; }

size_t gjk_f64_scratch_bytes(int64_t capacity) {
    return 256 + ((sizeof(int32_t) * (size_t)capacity + 255) & ~size_t(255)) + pair_order_temp_bytes(capacity);
}

int gjk_f64_run(const d3d_store& store, const int32_t* i1, const int32_t* i2, int64_t n, const int64_t* n_dev,
                const d3d_gjk_options& opt, const DistanceOut& o, void* scratch, cudaStream_t stream) {
    const bool sched = n >= tuning().sort_min;
    unsigned long long* cursor = static_cast<unsigned long long*>(scratch);
    int32_t* order = sched ? reinterpret_cast<int32_t*>(static_cast<char*>(scratch) + 256) : nullptr;
    const size_t order_bytes = (sizeof(int32_t) * (size_t)n + 255) & ~size_t(255);
    cudaError_t e = cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), stream);
    if (e != cudaSuccess) {
        set_error("d3d_gjk_distance: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    int rc = D3D_SUCCESS;
    if (sched)
        rc = pair_order(store, i1, i2, n, order, static_cast<char*>(scratch) + 256 + order_bytes,
                        pair_order_temp_bytes(n), stream, n_dev);
    if (!rc)
        rc = launch_gjk_f64(store, i1, i2, order, n, reinterpret_cast<const unsigned long long*>(n_dev), cursor,
                            opt, o, stream);
    return rc;
}

int launch_gjk_f64(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* order, int64_t n,
                   const unsigned long long* n_dev, unsigned long long* cursor, const d3d_gjk_options& opt,
                   const DistanceOut& o, cudaStream_t stream) {
    return launch_pool<4>(store, i1, i2, order, n, n_dev, cursor, opt, o, nullptr, stream);
}

}  // namespace d3d

extern "C" int d3d_gjk_distance_cached(const d3d_store* store, const int32_t* i1, const int32_t* i2, int64_t n,
                                       const d3d_gjk_options* options, int32_t* mesh_cache, double* dist,
                                       double* cp1, double* cp2, double* simplex, int8_t* n_simplex, int8_t* status,
                                       int32_t* iterations, void* stream) {
    int rc = d3d::check_store(store, "d3d_gjk_distance_cached");
    if (rc) return rc;
    D3D_REQUIRE(options, "d3d_gjk_distance_cached: null options");
    D3D_REQUIRE(n >= 0, "d3d_gjk_distance_cached: n < 0");
    D3D_REQUIRE(options->max_iterations >= 1, "d3d_gjk_distance_cached: max_iterations < 1");
    D3D_REQUIRE(options->precision == D3D_PRECISION_FP64,
                "d3d_gjk_distance_cached: the vertex cache is the reference's; only the FP64 form takes it");
    if (n == 0) return D3D_SUCCESS;
    D3D_REQUIRE(i1 && i2 && mesh_cache && dist && cp1 && cp2 && simplex && n_simplex && status,
                "d3d_gjk_distance_cached: null pointer");
    DistanceOut o{dist, cp1, cp2, simplex, n_simplex, status, iterations};
    k_gjk_distance_f64_cached<<<d3d::grid_for(n, 128), 128, 0, d3d::as_stream(stream)>>>(*store, i1, i2, n,
                                                                                          *options, o, mesh_cache);
    return d3d::check_launch("d3d_gjk_distance_cached");
}

extern "C" int d3d_gjk_intersection(const d3d_store* store, const int32_t* i1, const int32_t* i2, int64_t n,
                                    double tolerance, int32_t max_iterations, int8_t* hit, int8_t* status,
                                    void* stream) {
    int rc = d3d::check_store(store, "d3d_gjk_intersection");
    if (rc) return rc;
    D3D_REQUIRE(n >= 0, "d3d_gjk_intersection: n < 0");
    D3D_REQUIRE(max_iterations >= 1, "d3d_gjk_intersection: max_iterations < 1");
    if (n == 0) return D3D_SUCCESS;
    D3D_REQUIRE(i1 && i2 && hit && status, "d3d_gjk_intersection: null pointer");
    // In input order and without memory: a pool lists its supports by type itself, and these searches
    // are short.  Sorted by type from a full grid (77,824 pairs) on and claimed from a counter in
    // allocated memory -> dealt, us: six types 1,000 pairs 107 -> 97, 65,536 249 -> 248, 100,003 444 ->
    // 295, 1,048,576 2,080 -> 1,915; ten types 120 -> 112, 360 -> 366, 539 -> 419, 2,130 -> 2,260.
    const d3d_gjk_options opt{tolerance, 0.0, 0.0, max_iterations, D3D_PRECISION_FP64};
    // the kernel counts pairs in 31 bits
    constexpr int64_t kPart = int64_t(1) << 30;
    for (int64_t lo = 0; lo < n && !rc; lo += kPart) {
        DistanceOut o{};
        o.status = status + lo;
        rc = launch_pool<1>(*store, i1 + lo, i2 + lo, nullptr, n - lo < kPart ? n - lo : kPart, nullptr, nullptr, opt, o,
                            hit + lo, d3d::as_stream(stream));
    }
    return rc;
}
