// Stand-alone (non-fused) encoding and activation kernels.
// They replace EncodingForwardKernel / EncodingAdjointKernel (src_cpp/include/qmlp/kernels/encoding_kernels.cuh:26-62,
// launched by src_cpp/src/iencoding.cpp:12-196) and ActivationForwardKernel / ActivationAdjointKernel
// (src_cpp/include/qmlp/kernels/activation_kernels.cuh:28-62, launched by src_cpp/src/activation.cpp:64-150).
#pragma once
#include "fused_network.cuh"
#include "fused_forward_tc.cuh"
#include "fused_train_tc.cuh"
#include "fused_forward_ts.cuh"

namespace qmlp {
namespace kernel {

struct FloatRowWriter {
    float* row; long long s1;
    __device__ __forceinline__ void operator()(int c, float v) const { row[c * s1] = v; }
};
struct FloatRowReader {
    const float* row; long long s1;
    __device__ __forceinline__ float operator()(int c) const { return __ldg(row + c * s1); }
};

// EncSpec: NUM_ENCODINGS == 1 and Enc<0>
template <class EncSpec>
__global__ void __launch_bounds__(256) encoding_forward_kernel(const __grid_constant__ LaunchArgs p)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < p.numel;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        RowReader in{p.input + i * p.inS0, p.inS1};
        encode_point<EncSpec, 0>(p, in, FloatRowWriter{p.output + i * p.outS0, p.outS1});
    }
}

template <class EncSpec, bool INPUT_GRAD, bool PARAM_GRAD>
__global__ void __launch_bounds__(256) encoding_adjoint_kernel(const __grid_constant__ LaunchArgs p)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < p.numel;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        RowReader in{p.input + i * p.inS0, p.inS1};
        float* adjInRow = INPUT_GRAD ? p.adjInput + i * p.aiS0 : nullptr;
        encode_adjoint_point<EncSpec, 0, INPUT_GRAD, PARAM_GRAD>(
            p, in, FloatRowReader{p.adjOutput + i * p.aoS0, p.aoS1}, adjInRow, p.aiS1);
    }
}

// ---- plain grids: warp tiles and lane pairs ----------------------------------------------------------------------------
// A warp works on 32 points. Feature rows pass through a shared-memory tile, so that global memory sees whole contiguous
// rows however many features a point has, and the lanes work in pairs (see grid.cuh). Both lanes of a pair take the even
// lane's point first, then the odd lane's; every level is the same for the whole warp.
// Against one lane per point with strided rows, 10^6 points through a 2-D pyramid of five levels of four fp32 features:
// forward 104 -> 61 us (L1 wavefronts of the gathers, 87 % busy), table gradients 384 -> 295 us, and 295 -> 100 us with
// copies of the coarse levels' gradients (GradReplicas: before, 15 M reductions queued up on a few hundred lines).
template <class Enc>
struct EncodingTile {
    static constexpr int C = Enc::NUM_OUT, F = Enc::F;
    // rows of whole 16-byte pieces move as such; an odd number of pieces (or an odd row length) per row keeps the lanes'
    // rows in different banks
    static constexpr bool VEC = C % 4 == 0 && F % 2 == 0;
    static constexpr int STRIDE = VEC ? (C / 4 % 2 == 1 ? C : C + 4) : C + (C % 2 == 0 ? 1 : 0);
    static constexpr int WARPS = STRIDE <= 47 ? 8 : (STRIDE <= 95 ? 4 : 2);
    static constexpr int BYTES = WARPS * 32 * STRIDE * 4;
    static constexpr bool USED = BYTES <= 48 * 1024;   // up to 188 features; more take the kernels above
    // tile <-> rows [row0, row0 + 32) of an (n, C) tensor, rows past n are left alone
    template <bool STORE, class T>
    static __device__ __forceinline__ void copy(float* tile, T* base, long long s0, long long s1, long long row0, long long n, int lane)
    {
        const long long left = n - row0;
        const int rows = left < 32 ? static_cast<int>(left) : 32;
        if constexpr (VEC) {
            if (s1 == 1 && s0 == C && (reinterpret_cast<uintptr_t>(base) & 15) == 0) {
                constexpr int Q = C / 4;
#pragma unroll 4
                for (int i = lane; i < rows * Q; i += 32) {
                    float4* t = reinterpret_cast<float4*>(tile + i / Q * STRIDE + i % Q * 4);
                    T* at = base + row0 * C + i * 4;
                    if constexpr (STORE) *reinterpret_cast<float4*>(at) = *t;
                    else *t = __ldg(reinterpret_cast<const float4*>(at));
                }
                return;
            }
        }
        for (int i = lane; i < rows * C; i += 32) {
            const int r = i / C, c = i % C;
            T* at = base + (row0 + r) * s0 + c * s1;
            if constexpr (STORE) *at = tile[r * STRIDE + c];
            else tile[r * STRIDE + c] = __ldg(at);
        }
    }
    // the F features starting at channel c of a tile row
    static __device__ __forceinline__ void put(float* row, int c, const float (&v)[F])
    {
        if constexpr (VEC && F % 4 == 0) {
#pragma unroll
            for (int i = 0; i < F; i += 4) *reinterpret_cast<float4*>(row + c + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        } else if constexpr (VEC) {
#pragma unroll
            for (int i = 0; i < F; i += 2) *reinterpret_cast<float2*>(row + c + i) = make_float2(v[i], v[i + 1]);
        } else {
#pragma unroll
            for (int i = 0; i < F; ++i) row[c + i] = v[i];
        }
    }
    static __device__ __forceinline__ void get(const float* row, int c, float (&v)[F])
    {
        if constexpr (VEC && F % 4 == 0) {
#pragma unroll
            for (int i = 0; i < F; i += 4) {
                const float4 x = *reinterpret_cast<const float4*>(row + c + i);
                v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
            }
        } else if constexpr (VEC) {
#pragma unroll
            for (int i = 0; i < F; i += 2) {
                const float2 x = *reinterpret_cast<const float2*>(row + c + i);
                v[i] = x.x; v[i + 1] = x.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < F; ++i) v[i] = row[c + i];
        }
    }
};

template <class Enc>
__global__ void __launch_bounds__(EncodingTile<Enc>::WARPS * 32) grid_encoding_forward_kernel(const __grid_constant__ LaunchArgs p)
{
    using T = EncodingTile<Enc>;
    constexpr int D = Enc::D, F = Enc::F;
    __shared__ __align__(16) float tiles[T::WARPS][32 * T::STRIDE];
    const int lane = threadIdx.x & 31, side = lane & 1;
    float* tile = tiles[threadIdx.x >> 5];
    const GridP& g = p.grids[0];
    const long long last = p.numel - 1;
    for (long long row0 = (blockIdx.x * static_cast<long long>(T::WARPS) + (threadIdx.x >> 5)) * 32; row0 < p.numel;
         row0 += static_cast<long long>(gridDim.x) * T::WARPS * 32) {
        const long long i0 = row0 + (lane & ~1), i1 = i0 + 1;
        float pos0[D], pos1[D];
        grid_position<D, Enc::START>(g, RowReader{p.input + (i0 < last ? i0 : last) * p.inS0, p.inS1}, pos0);
        grid_position<D, Enc::START>(g, RowReader{p.input + (i1 < last ? i1 : last) * p.inS0, p.inS1}, pos1);
        float sum[F];
#pragma unroll
        for (int i = 0; i < F; ++i) sum[i] = 0.f;
        for (int l = 0; l < Enc::L; ++l) {
            const GridLevelP& lv = g.levels[l];
            float feat[F];
            grid_pair_forward<D, F, Enc::HALF_TABLE, false>(g, lv, grid_cells(p.level->cells, l), pos0, pos1, side, feat);
#pragma unroll
            for (int i = 0; i < F; ++i) sum[i] = Enc::CONCAT ? feat[i] : sum[i] + feat[i];
            if constexpr (Enc::CONCAT) T::put(tile + lane * T::STRIDE, l * F, sum);
        }
        if constexpr (!Enc::CONCAT) T::put(tile + lane * T::STRIDE, 0, sum);
        __syncwarp();
        T::template copy<true>(tile, p.output, p.outS0, p.outS1, row0, p.numel, lane);
        __syncwarp();
    }
}

template <class Enc, bool INPUT_GRAD, bool PARAM_GRAD>
__global__ void __launch_bounds__(EncodingTile<Enc>::WARPS * 32) grid_encoding_adjoint_kernel(const __grid_constant__ LaunchArgs p)
{
    using T = EncodingTile<Enc>;
    constexpr int D = Enc::D, F = Enc::F;
    __shared__ __align__(16) float tiles[T::WARPS][32 * T::STRIDE];
    const int lane = threadIdx.x & 31, side = lane & 1;
    float* tile = tiles[threadIdx.x >> 5];
    const GridP& g = p.grids[0];
    const long long last = p.numel - 1;
    for (long long row0 = (blockIdx.x * static_cast<long long>(T::WARPS) + (threadIdx.x >> 5)) * 32; row0 < p.numel;
         row0 += static_cast<long long>(gridDim.x) * T::WARPS * 32) {
        T::template copy<false>(tile, p.adjOutput, p.aoS0, p.aoS1, row0, p.numel, lane);
        const long long i0 = row0 + (lane & ~1);
        float pos[2][D], adjPos[2][D];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            grid_position<D, Enc::START>(g, RowReader{p.input + (i0 + s < last ? i0 + s : last) * p.inS0, p.inS1}, pos[s]);
#pragma unroll
            for (int k = 0; k < D; ++k) adjPos[s][k] = 0.f;
        }
        __syncwarp();
        for (int l = 0; l < Enc::L; ++l) {
            const GridLevelP& lv = g.levels[l];
            float* grad = g.grad;
            float* records = nullptr;
            if constexpr (PARAM_GRAD) {
                grad = grid_grad_of_cta(g, p.level->replicas, l, l, Enc::L);
                records = grid_records_of_cta<D, F>(g, p.level->replicas, l, l);
            }
            if constexpr (PARAM_GRAD && GridCellUnits<D, F>::USED) {
                if (records != nullptr) {
                    constexpr int C = Enc::CONCAT ? F : 0;
                    float own[D];
#pragma unroll
                    for (int k = 0; k < D; ++k) own[k] = side ? pos[1][k] : pos[0][k];
                    const bool done = grid_cells_scatter<D, F>(records, p.level->replicas.base + p.level->replicas.capacity, g.status, lv, own, row0 + lane <= last, [&](int r, float (&a)[F]) {
                        T::get(tile + (lane / GridCellUnits<D, F>::LANES * GridCellUnits<D, F>::LANES + r) * T::STRIDE, l * C, a);
                    });
                    if (!done) {
                        float a[F], none[D];
                        T::get(tile + lane * T::STRIDE, l * C, a);
                        grid_level_adjoint<D, F, Enc::HALF_TABLE, true, false>(g, lv, own, a, none);
                    }
                    if constexpr (!INPUT_GRAD) continue;
                }
            }
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (i0 + s > last) continue;
                float adjF[F];
                T::get(tile + ((lane & ~1) + s) * T::STRIDE, Enc::CONCAT ? l * F : 0, adjF);
                if constexpr (PARAM_GRAD && INPUT_GRAD && GridCellUnits<D, F>::USED) {
                    if (records != nullptr) {   // (the table's gradient is done)
                        if (lv.hashed) grid_half_adjoint<D, F, Enc::HALF_TABLE, false, true, 0>(g, grad, lv, pos[s], side, adjF, adjPos[s]);
                        else grid_half_adjoint<D, F, Enc::HALF_TABLE, false, true, D - 1>(g, grad, lv, pos[s], side, adjF, adjPos[s]);
                        continue;
                    }
                }
                if (lv.hashed) grid_half_adjoint<D, F, Enc::HALF_TABLE, PARAM_GRAD, INPUT_GRAD, 0>(g, grad, lv, pos[s], side, adjF, adjPos[s]);
                else grid_half_adjoint<D, F, Enc::HALF_TABLE, PARAM_GRAD, INPUT_GRAD, D - 1>(g, grad, lv, pos[s], side, adjF, adjPos[s]);
            }
        }
        if constexpr (INPUT_GRAD) {
            const long long i = row0 + lane;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const float own = side ? adjPos[1][k] : adjPos[0][k], other = side ? adjPos[0][k] : adjPos[1][k];
                const float v = own + __shfl_xor_sync(0xffffffffu, other, 1);
                if (i <= last) p.adjInput[i * p.aiS0 + (k + Enc::START) * p.aiS1] += v * g.boxInvSize[k];
            }
        }
        __syncwarp();
    }
}

// sums of the copies -> gradient table (blockIdx.y = level)
template <class Enc>
__global__ void __launch_bounds__(256) sum_replicas_kernel(const __grid_constant__ LaunchArgs p)
{
    grid_sum_copies<Enc::D, Enc::F>(p.grids[0], p.level->replicas, blockIdx.y, blockIdx.y, Enc::L);
}

template <class EncSpec>
struct EncodingLaunchers {
    using Enc = typename EncSpec::template Enc<0>;
    // one CTA per tile of points: the hardware refills an SM as soon as a CTA retires
    static unsigned blocksFor(const LaunchArgs& a, int points)
    {
        long long blocks = (a.numel + points - 1) / points;
        const long long cap = 1ll << 30;
        if (blocks > cap) blocks = cap;
        return static_cast<unsigned>(blocks < 1 ? 1 : blocks);
    }
    static cudaError_t forward(const LaunchArgs& a, cudaStream_t s, int& count)
    {
        if constexpr (Enc::IS_GRID) {
            if constexpr (EncodingTile<Enc>::USED) {
                const cudaError_t e = fill_cells<EncSpec>(a, s, &count);
                if (e != cudaSuccess) return e;
                constexpr int threads = EncodingTile<Enc>::WARPS * 32;
                grid_encoding_forward_kernel<Enc><<<blocksFor(a, threads), threads, 0, s>>>(a);
                return cudaGetLastError();
            }
        }
        encoding_forward_kernel<EncSpec><<<blocksFor(a, 256), 256, 0, s>>>(a);
        return cudaGetLastError();
    }
    template <bool INPUT_GRAD, bool PARAM_GRAD>
    static cudaError_t adjoint(const LaunchArgs& a, cudaStream_t s, int& count)
    {
        if constexpr (Enc::IS_GRID) {
            if constexpr (EncodingTile<Enc>::USED) {
                constexpr int threads = EncodingTile<Enc>::WARPS * 32;
                const bool copies = PARAM_GRAD && a.level->replicas.total > 0;
                if (copies) {
                    const cudaError_t e = cudaMemsetAsync(a.level->replicas.base, 0, a.level->replicas.total * sizeof(float), s);
                    if (e != cudaSuccess) return e;
                }
                grid_encoding_adjoint_kernel<Enc, INPUT_GRAD, PARAM_GRAD><<<blocksFor(a, threads), threads, 0, s>>>(a);
                if (copies) {
                    unsigned int blocks = 32;
                    for (int l = 0; l < Enc::L; ++l) {
                        const unsigned int n = grid_sum_blocks<Enc::D, Enc::F>(a.grids[0], a.level->replicas, l, l);
                        blocks = n > blocks ? n : blocks;
                    }
                    sum_replicas_kernel<Enc><<<dim3(blocks, Enc::L), 256, 0, s>>>(a);
                }
                count = copies ? 2 : 1;
                return cudaGetLastError();
            }
        }
        encoding_adjoint_kernel<EncSpec, INPUT_GRAD, PARAM_GRAD><<<blocksFor(a, 256), 256, 0, s>>>(a);
        return cudaGetLastError();
    }
    static int launch(int kernel, const void* args, cudaStream_t s, int* launches)
    {
        const LaunchArgs& a = *static_cast<const LaunchArgs*>(args);
        cudaError_t e = cudaErrorInvalidValue;
        int count = 1;
        if (kernel == KERNEL_ENCODING_FORWARD) {
            e = forward(a, s, count);
        } else if (kernel == KERNEL_ENCODING_ADJOINT) {
            const bool ig = (a.flags & 1) != 0, pg = (a.flags & 2) != 0;
            if (ig && pg) e = adjoint<true, true>(a, s, count);
            else if (ig) e = adjoint<true, false>(a, s, count);
            else if (pg) e = adjoint<false, true>(a, s, count);
            else { e = cudaSuccess; count = 0; }
        }
        if (launches) *launches = e == cudaSuccess ? count : 0;
        return static_cast<int>(e);
    }
};

// element-wise half activation over an (N, C) tensor with arbitrary strides
template <class Act, bool ADJOINT>
__global__ void __launch_bounds__(256) activation_kernel(const __grid_constant__ ActivationArgs p)
{
    const long long total = p.rows * p.cols;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long r = i / p.cols, c = i % p.cols;
        const half x = p.input[r * p.inS0 + c * p.inS1];
        if constexpr (ADJOINT) {
            const half g = p.adjOutput[r * p.aoS0 + c * p.aoS1];
            p.output[r * p.outS0 + c * p.outS1] = Act::adjoint(x, g);
        } else {
            p.output[r * p.outS0 + c * p.outS1] = Act::forward(x);
        }
    }
}

// contiguous fast path: half2 vectorised
template <class Act, bool ADJOINT>
__global__ void __launch_bounds__(256) activation_kernel_vec(const __grid_constant__ ActivationArgs p)
{
    const long long total2 = p.rows * p.cols / 2;
    const __half2* in = reinterpret_cast<const __half2*>(p.input);
    const __half2* go = reinterpret_cast<const __half2*>(p.adjOutput);
    __half2* out = reinterpret_cast<__half2*>(p.output);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total2;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        if constexpr (ADJOINT) out[i] = Act::adjoint2(in[i], go[i]);
        else out[i] = Act::forward2(in[i]);
    }
}

template <class Act>
struct ActivationLaunchers {
    static int launch(int kernel, const void* args, cudaStream_t s, int* launches)
    {
        const ActivationArgs& a = *static_cast<const ActivationArgs*>(args);
        const long long total = a.rows * a.cols;
        if (total == 0) { if (launches) *launches = 0; return 0; }
        const bool adj = kernel == KERNEL_ACTIVATION_ADJOINT;
        auto contiguous = [&](long long s0, long long s1) { return s1 == 1 && s0 == a.cols; };
        auto aligned4 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 3) == 0; };
        bool vec = (total % 2 == 0) && contiguous(a.inS0, a.inS1) && contiguous(a.outS0, a.outS1) && aligned4(a.input) && aligned4(a.output);
        if (adj) vec = vec && contiguous(a.aoS0, a.aoS1) && aligned4(a.adjOutput);
        const long long work = vec ? total / 2 : total;
        long long blocks = (work + 255) / 256;
        if (blocks > 148 * 16) blocks = 148 * 16;
        const unsigned g = static_cast<unsigned>(blocks);
        if (kernel == KERNEL_ACTIVATION_FORWARD) {
            if (vec) activation_kernel_vec<Act, false><<<g, 256, 0, s>>>(a);
            else activation_kernel<Act, false><<<g, 256, 0, s>>>(a);
        } else if (adj) {
            if (vec) activation_kernel_vec<Act, true><<<g, 256, 0, s>>>(a);
            else activation_kernel<Act, true><<<g, 256, 0, s>>>(a);
        } else {
            if (launches) *launches = 0;
            return static_cast<int>(cudaErrorInvalidValue);
        }
        cudaError_t e = cudaGetLastError();
        if (launches) *launches = e == cudaSuccess ? 1 : 0;
        return static_cast<int>(e);
    }
};

} // namespace kernel
} // namespace qmlp
