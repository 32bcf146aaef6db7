// Level-major encoding pass, and the scatter of table gradients from planes.
//
// When the gather runs inside the fused kernel, every warp walks through all levels of its own points, so at any moment
// the SMs touch all tables at once: with tables far larger than the 126 MB L2 (a 4-D grid of 16 levels of which 12 are hashed
// tables of 2^22 rows) nearly every corner fetch is a random 32-byte DRAM sector. This pass reorders the work instead
// of the data: the encodings of a chunk of points are computed one level at a time by the whole GPU (blockIdx.y =
// level, the slow grid dimension), so the table of the level being processed (32 MB in fp16) stays resident in L2 and
// corner fetches hit it there. The features go to level-major planes ([level][point][F] halfs, coalesced 4/8/16-byte
// stores); the layer kernel then reads its layer-0 operand from the planes (coalesced) instead of gathering. Inference takes
// the pass where that pays (planeChunk, capi.cpp) in chunks of up to 512 MB of planes; a training step always does, because
// its layer kernel reads features from, and leaves their adjoints in, the planes.
//
// Same arithmetic as the fused gather (grid.cuh; reference: src_cpp/include/qmlp/kernels/encoding_hashgrid.cuh:267-336).
#pragma once
#include "fused_network.cuh"

namespace qmlp {
namespace kernel {

// "groups": one per level of a concatenating grid, one for an adding grid, one for an identity encoding
template <class Spec, int E>
struct PlaneGroups {
    using Enc = typename Spec::template Enc<E>;
    __host__ __device__ static constexpr int own()
    {
        if constexpr (Enc::IS_GRID) return Enc::CONCAT ? Enc::L : 1;
        else return 1;
    }
    __host__ __device__ static constexpr int before()
    {
        if constexpr (E == 0) return 0;
        else return PlaneGroups<Spec, E - 1>::before() + PlaneGroups<Spec, E - 1>::own();
    }
};
template <class Spec>
__host__ __device__ constexpr int plane_group_count()
{
    return PlaneGroups<Spec, Spec::NUM_ENCODINGS - 1>::before() + PlaneGroups<Spec, Spec::NUM_ENCODINGS - 1>::own();
}

// levels of the plain grids, counted over all encodings
template <class Spec, int E>
struct ScatterGroups {
    using Enc = typename Spec::template Enc<E>;
    __host__ __device__ static constexpr int own()
    {
        if constexpr (Enc::IS_GRID) return Enc::L;
        else return 0;
    }
    __host__ __device__ static constexpr int before()
    {
        if constexpr (E == 0) return 0;
        else return ScatterGroups<Spec, E - 1>::before() + ScatterGroups<Spec, E - 1>::own();
    }
};
template <class Spec>
__host__ __device__ constexpr int scatter_group_count()
{
    return ScatterGroups<Spec, Spec::NUM_ENCODINGS - 1>::before() + ScatterGroups<Spec, Spec::NUM_ENCODINGS - 1>::own();
}

template <int W>
__device__ __forceinline__ void store_halfs(const LaunchArgs& p, __half* dst, const float (&v)[W])
{
    if (!scratch_ok(p, dst - p.planes, W, p.planeHalfs, STATUS_PLANES)) return;
    if constexpr (W == 2) {
        *reinterpret_cast<__half2*>(dst) = __floats2half2_rn(v[0], v[1]);
    } else if constexpr (W == 4) {
        uint2 u;
        u.x = h2_as_u32(__floats2half2_rn(v[0], v[1]));
        u.y = h2_as_u32(__floats2half2_rn(v[2], v[3]));
        *reinterpret_cast<uint2*>(dst) = u;
    } else if constexpr (W == 8) {
        uint4 u;
        u.x = h2_as_u32(__floats2half2_rn(v[0], v[1]));
        u.y = h2_as_u32(__floats2half2_rn(v[2], v[3]));
        u.z = h2_as_u32(__floats2half2_rn(v[4], v[5]));
        u.w = h2_as_u32(__floats2half2_rn(v[6], v[7]));
        *reinterpret_cast<uint4*>(dst) = u;
    } else {
#pragma unroll
        for (int i = 0; i < W; ++i) dst[i] = __float2half(v[i]);
    }
}

// Features of group `g` (relative to all groups) for the points `i` of a warp -> their planes. Lanes work in pairs (see
// grid.cuh): both lanes gather half of the corners of the even lane's point, then of the odd lane's, and each ends up
// with the sum for its own point. `in0` / `in1`: input rows of the pair's two points; all lanes of the warp take part.
template <class Spec, int E, bool EXACT>
__device__ __forceinline__ void encode_group(const LaunchArgs& p, int g, const RowReader& in0, const RowReader& in1, long long local, bool valid)
{
    if constexpr (E < Spec::NUM_ENCODINGS) {
        using Enc = typename Spec::template Enc<E>;
        using PG = PlaneGroups<Spec, E>;
        if (g >= PG::before() + PG::own()) {
            encode_group<Spec, E + 1, EXACT>(p, g, in0, in1, local, valid);
            return;
        }
        const int side = threadIdx.x & 1;
        if constexpr (!Enc::IS_GRID) {
            const RowReader& in = side ? in1 : in0;
            float v[Enc::N];
#pragma unroll
            for (int i = 0; i < Enc::N; ++i) v[i] = in(i + Enc::START);
            if (valid) store_halfs<Enc::N>(p, p.planes + p.planeStride * Enc::OUT_OFF + local * Enc::N, v);
        } else {
            constexpr int D = Enc::D, F = Enc::F;
            const GridP& grid = p.grids[Enc::SLOT];
            float pos0[D], pos1[D];
            grid_position<D, Enc::START>(grid, in0, pos0);
            grid_position<D, Enc::START>(grid, in1, pos1);
            float feat[F];
#pragma unroll
            for (int i = 0; i < F; ++i) feat[i] = 0.f;
            const int first = Enc::CONCAT ? g - PG::before() : 0, end = Enc::CONCAT ? first + 1 : Enc::L;
            for (int l = first; l < end; ++l) {
                const GridLevelP& lv = grid.levels[l];
                float f[F];
                grid_pair_forward<D, F, Enc::HALF_TABLE, EXACT>(grid, lv, grid_cells(p.level->cells, ScatterGroups<Spec, E>::before() + l), pos0, pos1, side, f);
#pragma unroll
                for (int i = 0; i < F; ++i) feat[i] += f[i];
            }
            if (valid) store_halfs<F>(p, p.planes + p.planeStride * (Enc::OUT_OFF + (Enc::CONCAT ? first * F : 0)) + local * F, feat);
        }
    }
}

// registers that hold one level's corner rows while its gathers are in flight; decides how many CTAs share an SM
template <class Spec, int E = 0>
__host__ __device__ constexpr int plane_row_registers()
{
    if constexpr (E >= Spec::NUM_ENCODINGS) {
        return 0;
    } else {
        using Enc = typename Spec::template Enc<E>;
        int own = 0;
        if constexpr (Enc::IS_GRID) own = (1 << Enc::D) * ((Enc::HALF_TABLE && Enc::F % 2 == 0) ? Enc::F / 2 : Enc::F);
        const int rest = plane_row_registers<Spec, E + 1>();
        return own > rest ? own : rest;
    }
}
template <class Spec>
__host__ __device__ constexpr int plane_min_blocks()
{
#ifdef QMLP_PLANE_MIN_BLOCKS
    return QMLP_PLANE_MIN_BLOCKS;
#else
    return plane_row_registers<Spec>() <= 32 ? 4 : (plane_row_registers<Spec>() <= 48 ? 3 : 2);
#endif
}

// EXACT: see grid_pair_forward
template <class Spec, bool EXACT>
__global__ void __launch_bounds__(256, plane_min_blocks<Spec>()) encode_planes_kernel(const __grid_constant__ LaunchArgs p)
{
    const int g = blockIdx.y;
    // whole warps stay together (the lanes of a pair exchange sums): lanes past the end repeat the last point
    for (long long base = blockIdx.x * static_cast<long long>(blockDim.x) + (threadIdx.x & ~31); base < p.numel;
         base += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long i = base + (threadIdx.x & 31), last = p.numel - 1;
        const long long i0 = i & ~1ll;
        const RowReader in0{p.input + (i0 < last ? i0 : last) * p.inS0, p.inS1}, in1{p.input + (i0 + 1 < last ? i0 + 1 : last) * p.inS0, p.inS1};
        encode_group<Spec, 0, EXACT>(p, g, in0, in1, i, i < p.numel);
    }
}

// ---- copies by cell (CellTables) --------------------------------------------------------------------------------------
// visit(encoding index constant, level of the grid, level over all grids) for every level that has a copy
template <class Spec, int E = 0, class Visit>
__host__ __device__ __forceinline__ void each_cell_level(const LaunchArgs& p, const Visit& visit)
{
    if constexpr (E < Spec::NUM_ENCODINGS) {
        using Enc = typename Spec::template Enc<E>;
        if constexpr (Enc::IS_GRID) {
            if constexpr (GridCellRows<Enc::D, Enc::F, Enc::HALF_TABLE>::USED) {
                for (int l = 0; l < Enc::L; ++l) {
                    const int group = ScatterGroups<Spec, E>::before() + l;
                    if (group < MAX_GRID_LEVELS && p.level->cells.offset[group] != 0) visit(Enc{}, l, group);
                }
            }
        }
        each_cell_level<Spec, E + 1>(p, visit);
    }
}
// one block after the other for every level that has a copy
template <class Spec>
__global__ void __launch_bounds__(FILL_THREADS) fill_cells_kernel(const __grid_constant__ LaunchArgs p)
{
    unsigned int block = blockIdx.x;
    each_cell_level<Spec>(p, [&](auto enc, int l, int group) {
        using Enc = decltype(enc);
        const GridP& grid = p.grids[Enc::SLOT];
        const unsigned int n = grid_fill_blocks<Enc::D, Enc::F, Enc::HALF_TABLE>(grid.levels[l].resolution);
        if (block < n)
            grid_fill_cells<Enc::D, Enc::F, Enc::HALF_TABLE>(grid, grid.levels[l], p.level->cells.base + static_cast<size_t>(p.level->cells.offset[group] - 1) * 256,
                                                                   p.level->cells.base + p.level->cells.bytes, block);
        block -= n;   // (wraps: the levels after this block's own are past its number)
    });
}
template <class Spec>
inline cudaError_t fill_cells(const LaunchArgs& a, cudaStream_t s, int* launches)
{
    if (a.level->cells.base == nullptr || !(a.flags & FLAG_FILL_CELLS)) return cudaSuccess;
    unsigned int blocks = 0;
    each_cell_level<Spec>(a, [&](auto enc, int l, int) {
        using Enc = decltype(enc);
        blocks += grid_fill_blocks<Enc::D, Enc::F, Enc::HALF_TABLE>(a.grids[Enc::SLOT].levels[l].resolution);
    });
    if (blocks == 0) return cudaSuccess;
    fill_cells_kernel<Spec><<<blocks, FILL_THREADS, 0, s>>>(a);
    if (launches) ++*launches;
    return cudaGetLastError();
}

// ---- level-major scatter of the table gradients --------------------------------------------------------------------
// Counterpart of the encoding pass for the backward direction: the backward kernel leaves the adjoint of every grid
// feature in the planes (write_adjoint_planes), and this kernel turns them into table gradients: light threads, many
// CTAs per SM, nothing but coalesced plane reads and reductions (the backward kernel itself runs 16 warps per SM at 128
// registers and alternates between MMA and scatter phases). A "group" is one level of one grid.
// lanes in pairs: both lanes of a pair scatter half of the corners of the even lane's point, then of the odd lane's
template <class Spec, int E>
__device__ __forceinline__ void scatter_group(const LaunchArgs& p, int g, const RowReader& in0, const RowReader& in1, long long point, bool valid)
{
    if constexpr (E < Spec::NUM_ENCODINGS) {
        using Enc = typename Spec::template Enc<E>;
        using SG = ScatterGroups<Spec, E>;
        if (g >= SG::before() + SG::own()) {
            scatter_group<Spec, E + 1>(p, g, in0, in1, point, valid);
            return;
        }
        if constexpr (Enc::IS_GRID) {
            const GridP& grid = p.grids[Enc::SLOT];
            if (grid.grad == nullptr) return;
            constexpr int D = Enc::D, F = Enc::F;
            const int side = threadIdx.x & 1;
            const int l = g - SG::before();
            const int c0 = Enc::OUT_OFF + (Enc::CONCAT ? l * F : 0);
            const __half* src = p.planes + p.planeStride * c0 + point * F;
            if (!scratch_ok(p, src - p.planes, F, p.planeHalfs, STATUS_PLANES)) valid = false;
            uint32_t own[(F + 1) / 2];
#pragma unroll
            for (int i = 0; i < (F + 1) / 2; ++i) own[i] = 0u;
            if (valid) {
                if constexpr (F == 2) {
                    own[0] = *reinterpret_cast<const uint32_t*>(src);
                } else if constexpr (F == 4) {
                    const uint2 u = *reinterpret_cast<const uint2*>(src);
                    own[0] = u.x; own[1] = u.y;
                } else {
#pragma unroll
                    for (int i = 0; i < F; ++i) own[i / 2] |= static_cast<uint32_t>(__half_as_ushort(src[i])) << (16 * (i & 1));
                }
            }
            const GridLevelP& lv = grid.levels[l];
            if (float* records = grid_records_of_cta<D, F>(grid, p.level->replicas, g, l)) {
                if constexpr (GridCellUnits<D, F>::USED) {
                    float pos[D];
                    grid_position<D, Enc::START>(grid, side ? in1 : in0, pos);
                    const auto unpack = [&](const uint32_t (&w)[(F + 1) / 2], float (&a)[F]) {
#pragma unroll
                        for (int i = 0; i < F / 2; ++i) {
                            const float2 x = __half22float2(u32_as_h2(w[i]));
                            a[2 * i] = x.x;
                            a[2 * i + 1] = x.y;
                        }
                    };
                    const bool done = grid_cells_scatter<D, F>(records, p.level->replicas.base + p.level->replicas.capacity, grid.status, lv, pos, valid, [&](int r, float (&a)[F]) {
                        uint32_t w[(F + 1) / 2];
#pragma unroll
                        for (int i = 0; i < (F + 1) / 2; ++i) w[i] = __shfl_sync(0xffffffffu, own[i], r, GridCellUnits<D, F>::LANES);
                        unpack(w, a);
                    });
                    if (!done) {
                        float a[F], none[D];
                        unpack(own, a);
                        grid_level_adjoint<D, F, false, true, false>(grid, lv, pos, a, none);
                    }
                }
                return;
            }
            float* grad = grid_grad_of_cta(grid, p.level->replicas, g, l, Enc::L);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                float pos[D], adjF[F];
                grid_position<D, Enc::START>(grid, s == 0 ? in0 : in1, pos);
                const bool ok = __shfl_sync(0xffffffffu, valid ? 1 : 0, (threadIdx.x & 30) + s) != 0;
#pragma unroll
                for (int i = 0; i < (F + 1) / 2; ++i) {
                    const float2 x = __half22float2(u32_as_h2(__shfl_sync(0xffffffffu, own[i], (threadIdx.x & 30) + s)));
                    adjF[2 * i] = x.x;
                    if (2 * i + 1 < F) adjF[2 * i + 1] = x.y;
                }
                if (!ok) continue;
                if (lv.hashed) grid_half_scatter<D, F, 0>(grid, grad, lv, pos, side, adjF);
                else grid_half_scatter<D, F, D - 1>(grid, grad, lv, pos, side, adjF);
            }
        }
    }
}

constexpr int SCATTER_THREADS = 128;

template <class Spec>
__global__ void __launch_bounds__(SCATTER_THREADS, 1024 / SCATTER_THREADS) scatter_planes_kernel(const __grid_constant__ LaunchArgs p)
{
    constexpr int groups = scatter_group_count<Spec>();
    const long long tiles = (p.numel + SCATTER_THREADS - 1) / SCATTER_THREADS;
    // levels of this launch (a data-parallel step scatters the levels in a few launches, so that the all-reduce of the
    // levels that are finished runs under the scatter of the next ones)
    const int begin = p.scatterLevelEnd > 0 ? p.scatterLevelBegin : 0;
    const int count = (p.scatterLevelEnd > 0 ? (p.scatterLevelEnd < groups ? p.scatterLevelEnd : groups) : groups) - begin;
    if (count <= 0) return;
    // A CTA takes its points through all levels, starting at a level that depends on the CTA: at any moment the CTAs of
    // the GPU are spread over all levels, so the reductions in flight go to many different rows and L2 slices (with all
    // CTAs on one small level, reductions to the same row queue up behind each other).
    const int first = static_cast<int>(blockIdx.x % count);
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        const long long i = t * SCATTER_THREADS + threadIdx.x, i0 = i & ~1ll, last = p.numel - 1;
        if ((i & ~31ll) >= p.numel) continue;   // whole warps stay together
        const RowReader in0{p.input + (i0 < last ? i0 : last) * p.inS0, p.inS1}, in1{p.input + (i0 + 1 < last ? i0 + 1 : last) * p.inS0, p.inS1};
        for (int gi = 0; gi < count; ++gi) {
            int g = first + gi;
            if (g >= count) g -= count;
            scatter_group<Spec, 0>(p, begin + g, in0, in1, i, i < p.numel);
        }
    }
}

// copies of group g's gradient (GradReplicas) -> table gradient
template <class Spec, int E>
__device__ __forceinline__ void sum_group(const LaunchArgs& p, int g)
{
    if constexpr (E < Spec::NUM_ENCODINGS) {
        using Enc = typename Spec::template Enc<E>;
        using SG = ScatterGroups<Spec, E>;
        if (g >= SG::before() + SG::own()) {
            sum_group<Spec, E + 1>(p, g);
        } else if constexpr (Enc::IS_GRID) {
            grid_sum_copies<Enc::D, Enc::F>(p.grids[Enc::SLOT], p.level->replicas, g, g - SG::before(), Enc::L);
        }
    }
}
template <class Spec, int E>
inline unsigned int sum_blocks(const LaunchArgs& a, int g)
{
    if constexpr (E < Spec::NUM_ENCODINGS) {
        using Enc = typename Spec::template Enc<E>;
        using SG = ScatterGroups<Spec, E>;
        if (g >= SG::before() + SG::own()) return sum_blocks<Spec, E + 1>(a, g);
        if constexpr (Enc::IS_GRID) return grid_sum_blocks<Enc::D, Enc::F>(a.grids[Enc::SLOT], a.level->replicas, g, g - SG::before());
    }
    return 0;
}
template <class Spec>
__global__ void __launch_bounds__(256) sum_copies_kernel(const __grid_constant__ LaunchArgs p)
{
    sum_group<Spec, 0>(p, blockIdx.y + (p.scatterLevelEnd > 0 ? p.scatterLevelBegin : 0));
}

template <class Spec>
struct PlaneLaunchers {
    static cudaError_t scatter(const LaunchArgs& a, cudaStream_t s, int* launches)
    {
        constexpr int groups = scatter_group_count<Spec>();
        if constexpr (groups == 0) {
            return cudaSuccess;
        } else {
            // one CTA per SCATTER_THREADS points: the hardware scheduler refills an SM as soon as a CTA retires, so the SMs drain
            // together at the end (with fewer, looping CTAs some took one tile more than others)
            long long bx = (a.numel + SCATTER_THREADS - 1) / SCATTER_THREADS;
            const long long cap = 1ll << 30;
            if (bx > cap) bx = cap;
            if (bx < 1) bx = 1;
            // The copies of the hot levels among the ones of this launch. Only these are cleared: the copies lie level by level, and
            // launches of other ranges may run at the same time.
            const int begin = a.scatterLevelEnd > 0 ? a.scatterLevelBegin : 0, end = a.scatterLevelEnd > 0 ? a.scatterLevelEnd : groups;
            int sums = 0;   // the levels up to the last one that has copies
            long long from = a.level->replicas.total, to = a.level->replicas.total;
            for (int g = 0; g < groups && g < MAX_GRID_LEVELS; ++g) {
                if (a.level->replicas.log2Copies[g] == 0 && a.level->replicas.byCell[g] == 0) continue;
                if (g >= begin && g < end) {
                    if (sums == 0) from = a.level->replicas.offset[g];
                    sums = g - begin + 1;
                } else if (g >= end) {
                    to = a.level->replicas.offset[g];
                    break;
                }
            }
            if (sums > 0) {
                const cudaError_t e = cudaMemsetAsync(a.level->replicas.base + from, 0, (to - from) * sizeof(float), s);
                if (e != cudaSuccess) return e;
            }
            scatter_planes_kernel<Spec><<<static_cast<unsigned>(bx), SCATTER_THREADS, 0, s>>>(a);
            if (sums > 0) {
                unsigned int blocks = 32;
                for (int g = begin; g < begin + sums; ++g) {
                    const unsigned int n = sum_blocks<Spec, 0>(a, g);
                    blocks = n > blocks ? n : blocks;
                }
                sum_copies_kernel<Spec><<<dim3(blocks, sums), 256, 0, s>>>(a);
                if (launches) *launches = 2;
            }
            return cudaGetLastError();
        }
    }
};

} // namespace kernel
} // namespace qmlp

#include "sorted_scatter.cuh"
