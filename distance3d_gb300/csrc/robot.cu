// robot.cu -- forward kinematics of serial chains on the device, for batched
// self-collision checks (the caller of the path in distance3d's
// self_collision.detect, self_collision.py:5-64, with the URDF chain it gets
// from urdf.py, here given directly).
//
// Link 0 is the base (identity).  Joint j (revolute) sits at the fixed
// transform origin_j of link j and turns link j+1 about its unit axis:
//   T_{j+1} = T_j * origin_j * Rot(axis_j, q_j)
// and body b, fixed to link link_b at origin_b, has the pose
//   T_{link_b} * origin_b.
// Compiled with -fmad=false; sin/cos are CUDA's.
#include "capi_util.h"

namespace {

// 3x4 transforms: R row-major (9) then t (3), the store's pose layout
__device__ __forceinline__ void compose(const double* A, const double* B, double* C) {
    double R[9], t[3];
    for (int i = 0; i < 3; ++i) {
        for (int j = 0; j < 3; ++j)
            R[3 * i + j] = A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
        t[i] = A[3 * i] * B[9] + A[3 * i + 1] * B[10] + A[3 * i + 2] * B[11] + A[9 + i];
    }
    for (int k = 0; k < 9; ++k) C[k] = R[k];
    for (int k = 0; k < 3; ++k) C[9 + k] = t[k];
}

// rotation by angle q about unit axis a (Rodrigues), no translation
__device__ __forceinline__ void axis_angle(const double* a, double q, double* T) {
    double s, c;
    sincos(q, &s, &c);
    const double C = 1.0 - c;
    const double x = a[0], y = a[1], z = a[2];
    T[0] = c + x * x * C;
    T[1] = x * y * C - z * s;
    T[2] = x * z * C + y * s;
    T[3] = y * x * C + z * s;
    T[4] = c + y * y * C;
    T[5] = y * z * C - x * s;
    T[6] = z * x * C - y * s;
    T[7] = z * y * C + x * s;
    T[8] = c + z * z * C;
    T[9] = T[10] = T[11] = 0.0;
}

// Row i, element e of compose(A, B) from A's row and B, in compose's order.
__device__ __forceinline__ double compose_at(const double* A, const double* B, int e) {
    if (e < 9) {
        const int i = e / 3, j = e - 3 * i;
        return A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
    }
    const int i = e - 9;
    return A[3 * i] * B[9] + A[3 * i + 1] * B[10] + A[3 * i + 2] * B[11] + A[9 + i];
}

// Bound by the FP64 pipe: a (configuration, body) per thread walked its whole
// chain, sines and cosines included, 97.6 us for 1,024 configurations of 7
// joints and 30 bodies.  Here a block takes kConfigs configurations: the joint
// rotations one per thread, the links of a configuration by the twelve
// elements of their transforms on a half warp, then the bodies one element per
// thread (coalesced): 21 us.  Every element is computed in compose's order.
constexpr int kConfigs = 8;
constexpr int kFkBlock = 16 * kConfigs;
constexpr int kMaxJoints = 30;  // the joint rotations and links of kConfigs configurations: 46.5 KB

__global__ void __launch_bounds__(kFkBlock) k_chain_fk(d3d_chain ch, const double* __restrict__ q, int64_t n_configs,
                                                       double* __restrict__ poses) {
    extern __shared__ double fk_smem[];
    const int J = ch.n_joints;
    double* const rot = fk_smem;                      // [config][joint][12]
    double* const link = rot + kConfigs * J * 12;     // [config][link][12]
    double* const half = link + kConfigs * (J + 1) * 12;  // [config][12]: T_j * origin_j
    const int64_t c0 = (int64_t)blockIdx.x * kConfigs;
    const int nc = (int)(n_configs - c0 < kConfigs ? n_configs - c0 : kConfigs);
    for (int x = threadIdx.x; x < nc * J; x += kFkBlock) {
        const int j = x % J;
        axis_angle(ch.joint_axis + 3 * j, q[c0 * J + x], rot + 12 * x);
    }
    const int c = threadIdx.x >> 4, e = threadIdx.x & 15;
    double* const T = link + c * (J + 1) * 12;
    if (e < 12) T[e] = e == 0 || e == 4 || e == 8 ? 1.0 : 0.0;
    __syncthreads();
    for (int j = 0; j < J; ++j) {
        if (c < nc && e < 12) half[12 * c + e] = compose_at(T + 12 * j, ch.joint_origin + 12 * j, e);
        __syncwarp();
        if (c < nc && e < 12) T[12 * (j + 1) + e] = compose_at(half + 12 * c, rot + 12 * (c * J + j), e);
        __syncwarp();
    }
    __syncthreads();
    const int per = 12 * ch.n_bodies;
    for (int x = threadIdx.x; x < nc * per; x += kFkBlock) {
        const int cc = x / per, y = x - cc * per, b = y / 12;
        const int l = min(max(ch.body_link[b], 0), J);
        poses[c0 * per + x] = compose_at(link + (cc * (J + 1) + l) * 12, ch.body_origin + 12 * b, y - 12 * b);
    }
}

// Longer chains: one thread per (configuration, body) walks the chain.
__global__ void k_chain_fk_long(d3d_chain ch, const double* __restrict__ q, int64_t n_configs,
                                double* __restrict__ poses) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_configs * ch.n_bodies) return;
    const int64_t c = k / ch.n_bodies;
    const int b = (int)(k - c * ch.n_bodies);
    const int link = ch.body_link[b];
    double T[12] = {1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0};
    for (int j = 0; j < link && j < ch.n_joints; ++j) {
        double O[12], R[12];
        compose(T, ch.joint_origin + 12 * j, O);
        axis_angle(ch.joint_axis + 3 * j, q[c * ch.n_joints + j], R);
        compose(O, R, T);
    }
    compose(T, ch.body_origin + 12 * b, poses + 12 * k);
}

// contacts[c][b] = 1 for both bodies of every pair at distance 0 (contacts
// cleared before; equal values may be stored by several threads).
__global__ void k_chain_contacts(const double* __restrict__ dist, int64_t n, const int32_t* __restrict__ pairs,
                                 int64_t n_pairs, int n_bodies, uint8_t* __restrict__ contacts) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || (__double_as_longlong(dist[k]) << 1) != 0) return;  // dist == 0, -0 included
    const int64_t c = k / n_pairs, p = k - c * n_pairs;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int b = pairs[2 * p + j];
        if (b >= 0 && b < n_bodies) contacts[c * n_bodies + b] = 1;
    }
}

}  // namespace

extern "C" int d3d_chain_fk(const d3d_chain* chain, const double* q, int64_t n_configs, double* poses,
                            void* stream) {
    D3D_REQUIRE(chain && n_configs >= 0, "d3d_chain_fk: invalid argument");
    D3D_REQUIRE(chain->n_joints >= 0 && chain->n_bodies >= 0, "d3d_chain_fk: negative sizes");
    const int64_t n = n_configs * chain->n_bodies;
    if (n == 0) return D3D_SUCCESS;
    D3D_REQUIRE(q && poses && chain->body_link && chain->body_origin &&
                    (chain->n_joints == 0 || (chain->joint_axis && chain->joint_origin)),
                "d3d_chain_fk: null pointer");
    cudaStream_t st = d3d::as_stream(stream);
    if (chain->n_joints <= kMaxJoints && chain->n_bodies <= INT32_MAX / (12 * kConfigs)) {
        const size_t smem = sizeof(double) * 12 * kConfigs * (size_t)(2 * chain->n_joints + 2);
        k_chain_fk<<<d3d::grid_for(n_configs, kConfigs), kFkBlock, smem, st>>>(*chain, q, n_configs, poses);
    } else {
        k_chain_fk_long<<<d3d::grid_for(n, 128), 128, 0, st>>>(*chain, q, n_configs, poses);
    }
    return d3d::check_launch("d3d_chain_fk");
}

extern "C" int d3d_chain_contacts(const double* dist, int64_t n_configs, const int32_t* pairs, int64_t n_pairs,
                                  int32_t n_bodies, uint8_t* contacts, void* stream) {
    D3D_REQUIRE(n_configs >= 0 && n_pairs >= 0 && n_bodies >= 0, "d3d_chain_contacts: negative size");
    if (n_configs == 0 || n_bodies == 0) return D3D_SUCCESS;
    D3D_REQUIRE(contacts && (n_pairs == 0 || (dist && pairs)), "d3d_chain_contacts: null pointer");
    cudaStream_t st = d3d::as_stream(stream);
    const cudaError_t e = cudaMemsetAsync(contacts, 0, (size_t)n_configs * (size_t)n_bodies, st);
    if (e != cudaSuccess) {
        d3d::set_error("d3d_chain_contacts: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    const int64_t n = n_configs * n_pairs;
    if (n > 0)
        k_chain_contacts<<<d3d::grid_for(n, 256), 256, 0, st>>>(dist, n, pairs, n_pairs, n_bodies, contacts);
    return d3d::check_launch("d3d_chain_contacts");
}
