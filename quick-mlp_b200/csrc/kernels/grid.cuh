// Multi-resolution dense / hashed grid: cell lookup, N-linear gather, gradient scatter, input gradient.
//
// Integer path (cell coordinates, dense and hashed row index) follows the reference bit for bit:
// src_cpp/include/qmlp/kernels/encoding_hashgrid.cuh:18-24 (primes), :36-46 (dense: last coordinate fastest; hash:
// xor of coordinate*prime in uint32), :71-84 (mod table size, times F, plus level offset), :277-284 (cell).
// What differs is the memory side: all F features of a corner move as one vector load / one vector reduction,
// tables may be fp16, and the level table arrives as a kernel parameter.
#pragma once
#include "launch_args.h"
#include "mma.cuh"

namespace qmlp {
namespace kernel {

__device__ __forceinline__ constexpr unsigned int hash_prime(int d)
{
    return d == 0 ? 1u : d == 1 ? 43857811u : d == 2 ? 83857661u : d == 3 ? 73856093u : d == 4 ? 19349663u : 834927u;
}

template <int D>
struct GridCell {
    unsigned int lo[D], hi[D]; // corner coordinates
    float f[D];                // fractions
};

// encoding_hashgrid.cuh:277-284
template <int D>
__device__ __forceinline__ void grid_cell(const float (&pos)[D], int resolution, GridCell<D>& c)
{
    const int rm1 = resolution - 1;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        float p = pos[i] * (resolution - 1);
        int ip = static_cast<int>(p);
        int l = max(0, min(rm1, ip));
        int h = max(0, min(rm1, ip + 1));
        c.lo[i] = static_cast<unsigned int>(l);
        c.hi[i] = static_cast<unsigned int>(h);
        c.f[i] = p - static_cast<float>(l);
    }
}

// Element index (row*F + level offset) of the grid vertex with integer coordinates `v`.
template <int D, int F>
__device__ __forceinline__ unsigned int grid_vertex_index(const unsigned int (&v)[D], const GridLevelP& lv)
{
    unsigned int idx;
    if (lv.hashed) {
        idx = v[0] * hash_prime(0);
#pragma unroll
        for (int k = 1; k < D; ++k) idx = (v[k] * hash_prime(k)) ^ idx;
        idx = idx & (lv.hashGridSize - 1u); // == idx % hashGridSize: the table size is always 1 << log2_hashmap_size
    } else {
        idx = v[0];
#pragma unroll
        for (int k = 1; k < D; ++k) idx = v[k] + idx * static_cast<unsigned int>(lv.resolution);
    }
    return idx * F + lv.offset;
}

// Every table access of every kernel passes its element index through here (records and copies by cell: grid_cell_inside), so this is
// where a QMLP_BOUNDS_CHECK build tests it: a row that does not lie inside its level is reported through the status word and replaced by the level's first row
// (which the copies of a level's gradient hold too), and the kernel carries on.
template <int D, int F>
__device__ __forceinline__ unsigned int grid_checked_index(const GridP& g, const GridLevelP& lv, unsigned int e)
{
    if constexpr (BOUNDS_CHECK) {
        unsigned long long rows = lv.hashGridSize;
        if (!lv.hashed) {
            rows = 1;
#pragma unroll
            for (int k = 0; k < D; ++k) rows *= static_cast<unsigned long long>(lv.resolution);
        }
        const unsigned long long last = lv.offset + rows * F, end = last < g.tableCount ? last : g.tableCount;
        if (e < lv.offset || static_cast<unsigned long long>(e) + F > end) {
            if (g.status != nullptr) atomicOr(g.status, STATUS_TABLE_ROW);
            return lv.offset;
        }
    }
    (void)g; (void)lv;
    return e;
}

// QMLP_BOUNDS_CHECK builds: is `cell` a cell of the level, and does what is read or written for it end where the scratch memory does? If
// not, the status word says so and the caller does without. Compiles to `true` in regular builds.
template <int D>
__device__ __forceinline__ bool grid_cell_inside(const GridLevelP& lv, unsigned int cell, const void* upTo, const void* end, int* status)
{
    if constexpr (BOUNDS_CHECK) {
        unsigned long long cells = 1;
#pragma unroll
        for (int k = 0; k < D; ++k) cells *= static_cast<unsigned long long>(lv.resolution);
        if (cell >= cells || static_cast<const char*>(upTo) > static_cast<const char*>(end)) {
            if (status != nullptr) atomicOr(status, STATUS_CELL);
            return false;
        }
    }
    (void)lv; (void)cell; (void)upTo; (void)end; (void)status;
    return true;
}

// element index of corner `bits` of a cell (bit k set -> high corner in dimension k)
template <int D, int F>
__device__ __forceinline__ unsigned int grid_corner_index(const GridP& g, const GridCell<D>& c, const GridLevelP& lv, int bits)
{
    unsigned int v[D];
#pragma unroll
    for (int k = 0; k < D; ++k) v[k] = ((bits >> k) & 1) ? c.hi[k] : c.lo[k];
    return grid_checked_index<D, F>(g, lv, grid_vertex_index<D, F>(v, lv));
}

// encoding_hashgrid.cuh:177-185,209-215: product taken from dimension D-1 down to 0
template <int D>
__device__ __forceinline__ float grid_corner_weight(const GridCell<D>& c, int bits)
{
    float w = 1.f;
#pragma unroll
    for (int k = D - 1; k >= 0; --k) w *= ((bits >> k) & 1) ? c.f[k] : (1.f - c.f[k]);
    return w;
}

template <int F, bool HALF>
__device__ __forceinline__ void grid_load_row(const void* table, unsigned int e, bool vec, float (&v)[F])
{
    if constexpr (HALF) {
        const __half* t = static_cast<const __half*>(table) + e;
        if constexpr (F == 2) {
            if (vec) { __half2 h = u32_as_h2(ldg_nc_u32(t)); float2 x = __half22float2(h); v[0] = x.x; v[1] = x.y; return; }
        } else if constexpr (F == 4) {
            if (vec) {
                uint2 u = ldg_nc_u64(t);
                float2 a = __half22float2(u32_as_h2(u.x)), b = __half22float2(u32_as_h2(u.y));
                v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; return;
            }
        } else if constexpr (F == 8) {
            if (vec) {
                uint4 u = ldg_nc_u128(t);
                float2 a = __half22float2(u32_as_h2(u.x)), b = __half22float2(u32_as_h2(u.y));
                float2 c = __half22float2(u32_as_h2(u.z)), d = __half22float2(u32_as_h2(u.w));
                v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y; return;
            }
        }
#pragma unroll
        for (int i = 0; i < F; ++i) v[i] = __half2float(__ldg(t + i));
    } else {
        const float* t = static_cast<const float*>(table) + e;
        if constexpr (F == 2) {
            if (vec) { uint2 u = ldg_nc_u64(t); v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); return; }
        } else if constexpr (F == 4) {
            if (vec) {
                uint4 u = ldg_nc_u128(t);
                v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
                return;
            }
        } else if constexpr (F == 8) {
            if (vec) {
                uint4 u = ldg_nc_u128(t), w = ldg_nc_u128(t + 4);
                v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
                v[4] = __uint_as_float(w.x); v[5] = __uint_as_float(w.y); v[6] = __uint_as_float(w.z); v[7] = __uint_as_float(w.w);
                return;
            }
        }
#pragma unroll
        for (int i = 0; i < F; ++i) v[i] = __ldg(t + i);
    }
}

template <int F>
__device__ __forceinline__ void grid_scatter_row(float* grad, unsigned int e, bool vec, float w, const float (&a)[F])
{
    float* g = grad + e;
    if constexpr (F == 2) {
        if (vec) { red_add_v2_f32(g, w * a[0], w * a[1]); return; }
    } else if constexpr (F % 4 == 0) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < F; i += 4) red_add_v4_f32(g + i, w * a[i], w * a[i + 1], w * a[i + 2], w * a[i + 3]);
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < F; ++i) red_add_f32(g + i, w * a[i]);
}

// one fp16 row as packed words (vector-aligned tables)
template <int F>
__device__ __forceinline__ void grid_load_packed(const __half* t, uint32_t (&r)[F / 2])
{
    static_assert(F == 2 || F == 4 || F == 8);
    if constexpr (F == 2) {
        r[0] = ldg_nc_u32(t);
    } else if constexpr (F == 4) {
        const uint2 u = ldg_nc_u64(t);
        r[0] = u.x; r[1] = u.y;
    } else {
        const uint4 u = ldg_nc_u128(t);
        r[0] = u.x; r[1] = u.y; r[2] = u.z; r[3] = u.w;
    }
}

// position in the unit cube, encoding_hashgrid.cuh:316-320
template <int D, int START, class In>
__device__ __forceinline__ void grid_position(const GridP& g, const In& input, float (&pos)[D])
{
#pragma unroll
    for (int i = 0; i < D; ++i) pos[i] = (input(i + START) - g.boxMin[i]) * g.boxInvSize[i];
}

// Interpolated features of one level (fp32 blend), encoding_hashgrid.cuh:267-293.
template <int D, int F, bool HALF>
__device__ __forceinline__ void grid_level_forward(const GridP& g, const GridLevelP& lv, const float (&pos)[D], float (&feat)[F])
{
    GridCell<D> c;
    grid_cell<D>(pos, lv.resolution, c);
    const bool vec = g.vecOk != 0;
    if constexpr (HALF && (F == 2 || F == 4 || F == 8)) {
        // fp16 rows stay packed while the loads are in flight (half the registers of the unpacked rows, so more warps
        // fit on the SM to hide the gather latency); same blend order as below
        if (vec) {
            uint32_t raw[1 << D][F / 2];
#pragma unroll
            for (int b = 0; b < (1 << D); ++b)
                grid_load_packed<F>(static_cast<const __half*>(g.table) + grid_corner_index<D, F>(g, c, lv, b), raw[b]);
#pragma unroll
            for (int i = 0; i < F; ++i) feat[i] = 0.f;
#pragma unroll
            for (int b = 0; b < (1 << D); ++b) {
                const float w = grid_corner_weight<D>(c, b);
#pragma unroll
                for (int i = 0; i < F / 2; ++i) {
                    const float2 x = __half22float2(u32_as_h2(raw[b][i]));
                    feat[2 * i] += w * x.x;
                    feat[2 * i + 1] += w * x.y;
                }
            }
            return;
        }
    }
    float rows[1 << D][F];
    // issue every corner load before the blend so they are all in flight together
#pragma unroll
    for (int b = 0; b < (1 << D); ++b) grid_load_row<F, HALF>(g.table, grid_corner_index<D, F>(g, c, lv, b), vec, rows[b]);
#pragma unroll
    for (int i = 0; i < F; ++i) feat[i] = 0.f;
#pragma unroll
    for (int b = 0; b < (1 << D); ++b) {
        const float w = grid_corner_weight<D>(c, b);
#pragma unroll
        for (int i = 0; i < F; ++i) feat[i] += w * rows[b][i];
    }
}

// Adjoint of one level: scatter w*adjF to the corners (encoding_hashgrid.cuh:130-140) and, when requested,
// the gradient with respect to the unit-cube position. The position gradient carries the factor
// (resolution-1) of p = pos*(resolution-1), which the reference leaves out (encoding_hashgrid.cuh:224-239).
template <int D, int F, bool HALF, bool PARAM_GRAD, bool INPUT_GRAD>
__device__ __forceinline__ void grid_level_adjoint(const GridP& g, const GridLevelP& lv, const float (&pos)[D],
                                                   const float (&adjF)[F], float (&adjPos)[D])
{
    GridCell<D> c;
    grid_cell<D>(pos, lv.resolution, c);
    const bool vec = g.vecOk != 0;
    float lvl[D];
#pragma unroll
    for (int k = 0; k < D; ++k) lvl[k] = 0.f;
#pragma unroll
    for (int b = 0; b < (1 << D); ++b) {
        const unsigned int e = grid_corner_index<D, F>(g, c, lv, b);
        if constexpr (PARAM_GRAD) grid_scatter_row<F>(g.grad, e, vec, grid_corner_weight<D>(c, b), adjF);
        if constexpr (INPUT_GRAD) {
            float row[F];
            grid_load_row<F, HALF>(g.table, e, vec, row);
            float dot = 0.f;
#pragma unroll
            for (int i = 0; i < F; ++i) dot += adjF[i] * row[i];
#pragma unroll
            for (int k = 0; k < D; ++k) {
                float wk = 1.f;
#pragma unroll
                for (int j = D - 1; j >= 0; --j)
                    if (j != k) wk *= ((b >> j) & 1) ? c.f[j] : (1.f - c.f[j]);
                lvl[k] += (((b >> k) & 1) ? wk : -wk) * dot;
            }
        }
    }
    if constexpr (INPUT_GRAD) {
#pragma unroll
        for (int k = 0; k < D; ++k) adjPos[k] += lvl[k] * static_cast<float>(lv.resolution - 1);
    }
}

// Table gradient of one level with corner pairs merged (same sums as grid_level_adjoint<.., true, false>).
// The two corners that differ in the pairing dimension are neighbouring rows whenever the cell coordinate in that
// dimension is even: the hash multiplies dimension 0 by 1, so its low bit survives the xor (hashed levels: dimension
// 0); dense levels store the last coordinate fastest (dimension D-1). Two neighbouring rows of two fp32 features are
// one aligned 16-byte vector, i.e. one L2 reduction instead of two; at the upper border both corners are the same row
// and their weights are added first.
template <int D, int F>
__device__ __forceinline__ void grid_level_scatter_paired(const GridP& g, const GridLevelP& lv, const float (&pos)[D],
                                                          const float (&adjF)[F])
{
    GridCell<D> c;
    grid_cell<D>(pos, lv.resolution, c);
    const bool vec = g.vecOk != 0;
    if constexpr (F == 2) {
        if (vec) {
            const int pd = lv.hashed ? 0 : D - 1;
#pragma unroll
            for (int h = 0; h < (1 << (D - 1)); ++h) {
                const int b0 = pd == 0 ? (h << 1) : h;
                const int b1 = b0 | (1 << pd);
                const unsigned int eA = grid_corner_index<D, F>(g, c, lv, b0), eB = grid_corner_index<D, F>(g, c, lv, b1);
                const float wA = grid_corner_weight<D>(c, b0), wB = grid_corner_weight<D>(c, b1);
                float* pa = g.grad + eA;
                float* pb = g.grad + eB;
                if (eA == eB) {
                    red_add_v2_f32(pa, (wA + wB) * adjF[0], (wA + wB) * adjF[1]);
                } else if (eB == eA + 2 && (reinterpret_cast<uintptr_t>(pa) & 15) == 0) {
                    red_add_v4_f32(pa, wA * adjF[0], wA * adjF[1], wB * adjF[0], wB * adjF[1]);
                } else if (eA == eB + 2 && (reinterpret_cast<uintptr_t>(pb) & 15) == 0) {
                    red_add_v4_f32(pb, wB * adjF[0], wB * adjF[1], wA * adjF[0], wA * adjF[1]);
                } else {
                    red_add_v2_f32(pa, wA * adjF[0], wA * adjF[1]);
                    red_add_v2_f32(pb, wB * adjF[0], wB * adjF[1]);
                }
            }
            return;
        }
    }
#pragma unroll
    for (int b = 0; b < (1 << D); ++b)
        grid_scatter_row<F>(g.grad, grid_corner_index<D, F>(g, c, lv, b), vec, grid_corner_weight<D>(c, b), adjF);
}

// ---- lane pairs ----------------------------------------------------------------------------------------------------
// Two neighbouring lanes share a point: the even lane takes the low corner of the pairing dimension, the odd lane the high
// one, and both walk through the 2^(D-1) corners of the other dimensions. The pairing dimension is the one along which
// neighbouring vertices are neighbouring rows (hashed levels: dimension 0, whose hash factor is 1; dense levels: the last
// coordinate), so the two rows of an access usually lie in one 128-byte line and leave the SM as one request, where two
// accesses of one lane leave as two. Gathers are bound by the rate of these requests (one per clock and SM), reductions
// by the L2 tag lookups they cost. Measured against one lane per point: gather of 2^22 points through a 4-D grid (16
// levels of four fp16 features, 2^22 rows) 2.83 -> 2.21 ms; 3-D grid (16 levels of two fp16 features, 2^19 rows), 2^20
// points: gather 282 -> 243 us (59 M requests, port 85 % busy), table gradients 525 -> 472 us (101 M -> 73 M requests,
// 84 M sectors).
// Coordinates and weights of the lane's half cell: dimension PD reduced to one side.
template <int D, int PD>
struct GridHalfCell {
    GridCell<D> c;
    unsigned int vp;   // this lane's coordinate in the pairing dimension
    float wp;          // and its weight
    __device__ __forceinline__ GridHalfCell(const float (&pos)[D], int resolution, int side)
    {
        grid_cell<D>(pos, resolution, c);
        take(side);
    }
    __device__ __forceinline__ GridHalfCell(const GridCell<D>& cell, int side) : c(cell) { take(side); }
    __device__ __forceinline__ void take(int side)
    {
        vp = side ? c.hi[PD] : c.lo[PD];
        wp = side ? c.f[PD] : 1.f - c.f[PD];
    }
    // h: one bit per dimension other than PD, in ascending order
    template <int F>
    __device__ __forceinline__ unsigned int index(const GridP& g, const GridLevelP& lv, int h) const
    {
        unsigned int v[D];
#pragma unroll
        for (int k = 0, b = 0; k < D; ++k) {
            if (k == PD) { v[k] = vp; continue; }
            v[k] = ((h >> b) & 1) ? c.hi[k] : c.lo[k];
            ++b;
        }
        unsigned int idx;
        if constexpr (PD == 0) {   // hashed (D == 1: hashed and dense pair along the same dimension)
            if (D > 1 || lv.hashed) {
                idx = v[0] * hash_prime(0);
#pragma unroll
                for (int k = 1; k < D; ++k) idx = (v[k] * hash_prime(k)) ^ idx;
                idx &= lv.hashGridSize - 1u;
            } else {
                idx = v[0];
            }
        } else {
            idx = v[0];
#pragma unroll
            for (int k = 1; k < D; ++k) idx = v[k] + idx * static_cast<unsigned int>(lv.resolution);
        }
        return grid_checked_index<D, F>(g, lv, idx * F + lv.offset);
    }
    __device__ __forceinline__ float weight(int h) const
    {
        float w = 1.f;
#pragma unroll
        for (int k = D - 1, b = D - 2; k >= 0; --k) {
            if (k == PD) { w *= wp; continue; }
            w *= ((h >> b) & 1) ? c.f[k] : (1.f - c.f[k]);
            --b;
        }
        return w;
    }
};

// this lane's share of the features of one level: the sum over its half of the corners
template <int D, int F, bool HALF, int PD>
__device__ __forceinline__ void grid_half_forward(const GridP& g, const GridLevelP& lv, const float (&pos)[D], int side, float (&feat)[F])
{
    const GridHalfCell<D, PD> c(pos, lv.resolution, side);
    const bool vec = g.vecOk != 0;
    constexpr int H = 1 << (D - 1);
#pragma unroll
    for (int i = 0; i < F; ++i) feat[i] = 0.f;
    if constexpr (HALF && (F == 2 || F == 4 || F == 8)) {
        if (vec) {
            uint32_t raw[H][F / 2];
#pragma unroll
            for (int h = 0; h < H; ++h)
                grid_load_packed<F>(static_cast<const __half*>(g.table) + c.template index<F>(g, lv, h), raw[h]);
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const float w = c.weight(h);
#pragma unroll
                for (int i = 0; i < F / 2; ++i) {
                    const float2 x = __half22float2(u32_as_h2(raw[h][i]));
                    feat[2 * i] += w * x.x;
                    feat[2 * i + 1] += w * x.y;
                }
            }
            return;
        }
    }
    float rows[H][F];
#pragma unroll
    for (int h = 0; h < H; ++h) grid_load_row<F, HALF>(g.table, c.template index<F>(g, lv, h), vec, rows[h]);
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const float w = c.weight(h);
#pragma unroll
        for (int i = 0; i < F; ++i) feat[i] += w * rows[h][i];
    }
}

// Both lanes' rows of one level, exchanged before the blend: `raw0` / `raw1` are this lane's rows of the pair's points, and
// each lane sums all 2^D corners of its own point in the order of grid_level_forward.
template <int D, int F, int PD, int W, class Add>
__device__ __forceinline__ void grid_pair_blend(const GridCell<D>& c, int side, const uint32_t (&raw0)[1 << (D - 1)][W],
                                                const uint32_t (&raw1)[1 << (D - 1)][W], float (&feat)[F], const Add& add)
{
    constexpr int H = 1 << (D - 1);
    uint32_t low[H][W], high[H][W];
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const uint32_t own = side ? raw1[h][i] : raw0[h][i];
            const uint32_t other = __shfl_xor_sync(0xffffffffu, side ? raw0[h][i] : raw1[h][i], 1);
            low[h][i] = side ? other : own;
            high[h][i] = side ? own : other;
        }
#pragma unroll
    for (int b = 0; b < (1 << D); ++b) {
        const float w = grid_corner_weight<D>(c, b);
        const int h = PD == 0 ? b >> 1 : b & (H - 1);   // bits of the other dimensions
        if (((b >> PD) & 1) == 0) add(w, low[h], feat);
        else add(w, high[h], feat);
    }
}

// Features of one level for this lane's own point, with the gathers of grid_half_forward for the points of both lanes and the
// sums of grid_level_forward, bit for bit.
template <int D, int F, bool HALF, int PD>
__device__ __forceinline__ void grid_pair_exchange(const GridP& g, const GridLevelP& lv, const float (&pos0)[D], const float (&pos1)[D], int side,
                                                   float (&feat)[F])
{
    const GridHalfCell<D, PD> c0(pos0, lv.resolution, side), c1(pos1, lv.resolution, side);
    GridCell<D> own;
#pragma unroll
    for (int i = 0; i < D; ++i) own.f[i] = side ? c1.c.f[i] : c0.c.f[i];
    const bool vec = g.vecOk != 0;
    constexpr int H = 1 << (D - 1);
#pragma unroll
    for (int i = 0; i < F; ++i) feat[i] = 0.f;
    if constexpr (HALF && (F == 2 || F == 4 || F == 8)) {
        if (vec) {
            uint32_t raw0[H][F / 2], raw1[H][F / 2];
#pragma unroll
            for (int h = 0; h < H; ++h) {
                grid_load_packed<F>(static_cast<const __half*>(g.table) + c0.template index<F>(g, lv, h), raw0[h]);
                grid_load_packed<F>(static_cast<const __half*>(g.table) + c1.template index<F>(g, lv, h), raw1[h]);
            }
            grid_pair_blend<D, F, PD, F / 2>(own, side, raw0, raw1, feat, [](float w, const uint32_t (&r)[F / 2], float (&f)[F]) {
#pragma unroll
                for (int i = 0; i < F / 2; ++i) {
                    const float2 x = __half22float2(u32_as_h2(r[i]));
                    f[2 * i] += w * x.x;
                    f[2 * i + 1] += w * x.y;
                }
            });
            return;
        }
    }
    uint32_t raw0[H][F], raw1[H][F];
#pragma unroll
    for (int h = 0; h < H; ++h) {
        float r0[F], r1[F];
        grid_load_row<F, HALF>(g.table, c0.template index<F>(g, lv, h), vec, r0);
        grid_load_row<F, HALF>(g.table, c1.template index<F>(g, lv, h), vec, r1);
#pragma unroll
        for (int i = 0; i < F; ++i) {
            raw0[h][i] = __float_as_uint(r0[i]);
            raw1[h][i] = __float_as_uint(r1[i]);
        }
    }
    grid_pair_blend<D, F, PD, F>(own, side, raw0, raw1, feat, [](float w, const uint32_t (&r)[F], float (&f)[F]) {
#pragma unroll
        for (int i = 0; i < F; ++i) f[i] += w * __uint_as_float(r[i]);
    });
}

template <int D, int F, bool HALF, int PD>
__device__ __forceinline__ void grid_pair_sums(const GridP& g, const GridLevelP& lv, const float (&pos0)[D], const float (&pos1)[D], int side,
                                               float (&feat)[F])
{
    float f0[F], f1[F];
    grid_half_forward<D, F, HALF, PD>(g, lv, pos0, side, f0);
    grid_half_forward<D, F, HALF, PD>(g, lv, pos1, side, f1);
#pragma unroll
    for (int i = 0; i < F; ++i) feat[i] = (side ? f1[i] : f0[i]) + __shfl_xor_sync(0xffffffffu, side ? f0[i] : f1[i], 1);
}

// ---- copies by cell (CellTables) ------------------------------------------------------------------------------------
// A level with few cells, compared with the points of a batch, is copied so that the 2^D rows of a cell lie side by side: the lanes
// of a pair then read one contiguous piece of memory, one request, where the rows of the table take 2^(D-1) (the request
// rate bounds the gathers, see above). The rows of a cell stand as the lanes of a pair fetch them, in accesses of up to
// 32 bytes: low side of the pairing dimension, high side, low side, ...; within a side by the bits of the other dimensions. The
// terms and their order are those of the table's rows.
template <int D, int F, bool HALF>
struct GridCellRows {
    static constexpr int H = 1 << (D - 1), ROW = F * (HALF ? 2 : 4), WORDS = ROW / 4;   // rows per side; bytes and words of a row
    static constexpr int BYTES = 2 * H * ROW;
    static constexpr bool USED = D >= 2 && (F == 4 || F == 8) && BYTES >= 64 && BYTES <= 256;   // (the host's rule: EncodingHashGrid::planCells)
    static constexpr int ACCESS = H * ROW < 32 ? H * ROW : 32, PER_ACCESS = ACCESS / ROW, ACCESSES = H / PER_ACCESS;
};

// Cells are numbered by their low corner, neighbours along the dimension whose vertices are neighbouring rows first (the copy is
// filled with coalesced reads).
template <int D>
__device__ __forceinline__ unsigned int grid_cell_number(const GridCell<D>& c, const GridLevelP& lv)
{
    unsigned int n;
    if (lv.hashed) {
        n = c.lo[D - 1];
#pragma unroll
        for (int k = D - 2; k >= 0; --k) n = c.lo[k] + n * static_cast<unsigned int>(lv.resolution);
    } else {
        n = c.lo[0];
#pragma unroll
        for (int k = 1; k < D; ++k) n = c.lo[k] + n * static_cast<unsigned int>(lv.resolution);
    }
    return n;
}
// The copy holds the cells of points inside the box: high corner = low corner + 1, or the border. A point below the box has
// other corners.
template <int D>
__device__ __forceinline__ bool grid_cell_regular(const GridCell<D>& c, const GridLevelP& lv)
{
    bool ok = true;
#pragma unroll
    for (int k = 0; k < D; ++k) ok = ok && c.hi[k] == min(c.lo[k] + 1u, static_cast<unsigned int>(lv.resolution - 1));
    return ok;
}

// a level's copy (at null: none) and the end of the memory that holds it
struct CellCopy {
    const unsigned char* at;
    const unsigned char* end;
};

// this lane's rows (one side of the pairing dimension) of a cell
template <int D, int F, bool HALF>
__device__ __forceinline__ void grid_cell_load(const unsigned char* cells, unsigned int cell, int side,
                                               uint32_t (&raw)[1 << (D - 1)][GridCellRows<D, F, HALF>::WORDS])
{
    using C = GridCellRows<D, F, HALF>;
    const unsigned char* at = cells + static_cast<size_t>(cell) * C::BYTES + side * C::ACCESS;
#pragma unroll
    for (int u = 0; u < C::ACCESSES; ++u) {
        uint32_t v[8];
        static_assert(C::ACCESS == 32);
        ldg_nc_u256(at + u * 2 * C::ACCESS, v);
#pragma unroll
        for (int r = 0; r < C::PER_ACCESS; ++r)
#pragma unroll
            for (int i = 0; i < C::WORDS; ++i) raw[u * C::PER_ACCESS + r][i] = v[r * C::WORDS + i];
    }
}

// feat += w * row
template <int F, bool HALF>
__device__ __forceinline__ void grid_add_row(float w, const uint32_t (&r)[F * (HALF ? 2 : 4) / 4], float (&feat)[F])
{
    if constexpr (HALF) {
#pragma unroll
        for (int i = 0; i < F / 2; ++i) {
            const float2 x = __half22float2(u32_as_h2(r[i]));
            feat[2 * i] += w * x.x;
            feat[2 * i + 1] += w * x.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < F; ++i) feat[i] += w * __uint_as_float(r[i]);
    }
}

// grid_pair_forward from the copy. False, for the whole warp, if one of its points has other corners than the copy holds.
template <int D, int F, bool HALF, bool EXCHANGE, int PD>
__device__ __forceinline__ bool grid_pair_from_cells(const CellCopy& copy, const GridLevelP& lv, int* status, const float (&pos0)[D], const float (&pos1)[D],
                                                     int side, float (&feat)[F])
{
    using C = GridCellRows<D, F, HALF>;
    GridCell<D> c0, c1;
    grid_cell<D>(pos0, lv.resolution, c0);
    grid_cell<D>(pos1, lv.resolution, c1);
#pragma unroll
    for (int k = 0; k < D; ++k) asm volatile("" : "+f"(c0.f[k]), "+f"(c1.f[k]));   // (computed here, beside the product they come from, as in the other path)
    if (!__all_sync(0xffffffffu, grid_cell_regular<D>(c0, lv) && grid_cell_regular<D>(c1, lv))) return false;
    const unsigned int n0 = grid_cell_number<D>(c0, lv), n1 = grid_cell_number<D>(c1, lv);
    if constexpr (BOUNDS_CHECK) {
        const unsigned char *up0 = copy.at + (static_cast<size_t>(n0) + 1) * C::BYTES, *up1 = copy.at + (static_cast<size_t>(n1) + 1) * C::BYTES;
        const bool inside = grid_cell_inside<D>(lv, n0, up0, copy.end, status) && grid_cell_inside<D>(lv, n1, up1, copy.end, status);
        if (!__all_sync(0xffffffffu, inside)) return false;
    }
    uint32_t raw0[C::H][C::WORDS], raw1[C::H][C::WORDS];
    grid_cell_load<D, F, HALF>(copy.at, n0, side, raw0);
    grid_cell_load<D, F, HALF>(copy.at, n1, side, raw1);
    if constexpr (EXCHANGE) {
        GridCell<D> own;
#pragma unroll
        for (int i = 0; i < D; ++i) own.f[i] = side ? c1.f[i] : c0.f[i];
#pragma unroll
        for (int i = 0; i < F; ++i) feat[i] = 0.f;
        grid_pair_blend<D, F, PD, C::WORDS>(own, side, raw0, raw1, feat,
                                           [](float w, const uint32_t (&r)[C::WORDS], float (&f)[F]) { grid_add_row<F, HALF>(w, r, f); });
    } else {
        const GridHalfCell<D, PD> h0(c0, side), h1(c1, side);
        float f0[F], f1[F];
#pragma unroll
        for (int i = 0; i < F; ++i) f0[i] = f1[i] = 0.f;
#pragma unroll
        for (int h = 0; h < C::H; ++h) {
            grid_add_row<F, HALF>(h0.weight(h), raw0[h], f0);
            grid_add_row<F, HALF>(h1.weight(h), raw1[h], f1);
        }
#pragma unroll
        for (int i = 0; i < F; ++i) feat[i] = (side ? f1[i] : f0[i]) + __shfl_xor_sync(0xffffffffu, side ? f0[i] : f1[i], 1);
    }
    return true;
}

// copy of level `group` (counted over all grids)
__device__ __forceinline__ CellCopy grid_cells(const CellTables& t, int group)
{
    if (t.base == nullptr || group >= MAX_GRID_LEVELS || t.offset[group] == 0) return {nullptr, nullptr};
    return {t.base + static_cast<size_t>(t.offset[group] - 1) * 256, t.base + t.bytes};
}

constexpr int FILL_THREADS = 256;
// blocks that fill the copy of a level: a thread writes one access
template <int D, int F, bool HALF>
__host__ __device__ inline unsigned int grid_fill_blocks(int resolution)
{
    unsigned int n = 1;
    for (int k = 0; k < D; ++k) n *= static_cast<unsigned int>(resolution);
    return (n * (2 * GridCellRows<D, F, HALF>::ACCESSES) + FILL_THREADS - 1) / FILL_THREADS;
}
template <int D, int F, bool HALF>
__device__ __forceinline__ void grid_fill_cells(const GridP& g, const GridLevelP& lv, unsigned char* cells, const unsigned char* end, unsigned int block)
{
    using C = GridCellRows<D, F, HALF>;
    const unsigned int t = block * FILL_THREADS + threadIdx.x, side = t & 1u, u = (t >> 1) % C::ACCESSES, res = static_cast<unsigned int>(lv.resolution);
    unsigned int n = (t >> 1) / C::ACCESSES, lo[D];
    // (the dimension that varies first: grid_cell_number)
#pragma unroll
    for (int j = 0; j < D; ++j) {
        const unsigned int q = n / res, r = n - q * res;
        if (lv.hashed) lo[j] = r;
        else lo[D - 1 - j] = r;
        n = q;
    }
    if (n != 0) return;   // past the last cell
    GridCell<D> c;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        c.lo[k] = lo[k];
        c.hi[k] = min(lo[k] + 1u, res - 1u);
    }
    uint32_t v[8];
#pragma unroll
    for (int r = 0; r < C::PER_ACCESS; ++r) {
        const unsigned int h = u * C::PER_ACCESS + r;
        const int b = static_cast<int>(lv.hashed ? (h << 1 | side) : (h | side << (D - 1)));
        const unsigned int e = grid_corner_index<D, F>(g, c, lv, b);
        float row[F];
        grid_load_row<F, HALF>(g.table, e, g.vecOk != 0, row);
#pragma unroll
        for (int i = 0; i < C::WORDS; ++i) {
            if constexpr (HALF) v[r * C::WORDS + i] = h2_as_u32(__floats2half2_rn(row[2 * i], row[2 * i + 1]));
            else v[r * C::WORDS + i] = __float_as_uint(row[i]);
        }
    }
    unsigned char* at = cells + static_cast<size_t>(t) * C::ACCESS;   // (accesses in the order of the threads)
    if (!grid_cell_inside<D>(lv, 0, at + C::ACCESS, end, g.status)) return;
    stg_u256(at, v);
}

// Features of one level for this lane's own point; all lanes of the warp take part. The lanes exchange rows or, unless EXACT,
// half sums. With half sums a feature next to the middle of two fp16 numbers can be rounded to the other one, which moves a
// ReLU input across zero now and then and with it the gradients behind it (3-D grid of 16 levels, 25 843 points: one
// entry of the table gradient off by 1.8 times the rms), so every pass that gradients follow is EXACT. Inference takes
// what is quicker: up to four words per lane and point the exchange (3-D grid of two fp16 features, 2^20 points: 275 against
// 280 us in all), above that the half sums (two fp32 features, 100 000 points: 41.0 against 42.8 us; 4-D grid of four fp16
// features, 2^24 points: 10.5 against 11.7 ms).
template <int D, int F, bool HALF, bool EXACT>
__device__ __forceinline__ void grid_pair_forward(const GridP& g, const GridLevelP& lv, const CellCopy& copy, const float (&pos0)[D], const float (&pos1)[D],
                                                  int side, float (&feat)[F])
{
    constexpr int WORDS = (1 << (D - 1)) * ((HALF && F % 2 == 0) ? F / 2 : F);
    if constexpr (GridCellRows<D, F, HALF>::USED) {
        if (copy.at != nullptr) {
            if (lv.hashed ? grid_pair_from_cells<D, F, HALF, EXACT || WORDS <= 4, 0>(copy, lv, g.status, pos0, pos1, side, feat)
                          : grid_pair_from_cells<D, F, HALF, EXACT || WORDS <= 4, D - 1>(copy, lv, g.status, pos0, pos1, side, feat)) return;
        }
    }
    if constexpr (EXACT || WORDS <= 4) {
        if (lv.hashed) grid_pair_exchange<D, F, HALF, 0>(g, lv, pos0, pos1, side, feat);
        else grid_pair_exchange<D, F, HALF, D - 1>(g, lv, pos0, pos1, side, feat);
    } else {
        if (lv.hashed) grid_pair_sums<D, F, HALF, 0>(g, lv, pos0, pos1, side, feat);
        else grid_pair_sums<D, F, HALF, D - 1>(g, lv, pos0, pos1, side, feat);
    }
}

// table gradient (into `grad`) and, when requested, the gradient with respect to the unit-cube position (see
// grid_level_adjoint) from this lane's half of the corners; adjPos receives this lane's share of the sum
template <int D, int F, bool HALF, bool PARAM_GRAD, bool INPUT_GRAD, int PD>
__device__ __forceinline__ void grid_half_adjoint(const GridP& g, float* grad, const GridLevelP& lv, const float (&pos)[D], int side,
                                                  const float (&adjF)[F], float (&adjPos)[D])
{
    const GridHalfCell<D, PD> c(pos, lv.resolution, side);
    const bool vec = g.vecOk != 0;
    float lvl[D];
#pragma unroll
    for (int k = 0; k < D; ++k) lvl[k] = 0.f;
#pragma unroll
    for (int h = 0; h < (1 << (D - 1)); ++h) {
        const unsigned int e = c.template index<F>(g, lv, h);
        if constexpr (PARAM_GRAD) grid_scatter_row<F>(grad, e, vec, c.weight(h), adjF);
        if constexpr (INPUT_GRAD) {
            float row[F];
            grid_load_row<F, HALF>(g.table, e, vec, row);
            float dot = 0.f;
#pragma unroll
            for (int i = 0; i < F; ++i) dot += adjF[i] * row[i];
#pragma unroll
            for (int k = 0; k < D; ++k) {
                float wk = 1.f;   // weight without dimension k
#pragma unroll
                for (int j = D - 1, b = D - 2; j >= 0; --j) {
                    const int bit = j == PD ? 0 : b--;
                    if (j == k) continue;
                    wk *= j == PD ? c.wp : ((h >> bit) & 1) ? c.c.f[j] : (1.f - c.c.f[j]);
                }
                // bit of dimension k: its position among the dimensions other than PD
                const bool high = k == PD ? side != 0 : ((h >> (k > PD ? k - 1 : k)) & 1) != 0;
                lvl[k] += (high ? wk : -wk) * dot;
            }
        }
    }
    if constexpr (INPUT_GRAD) {
#pragma unroll
        for (int k = 0; k < D; ++k) adjPos[k] += lvl[k] * static_cast<float>(lv.resolution - 1);
    }
}

template <int D, int F, int PD>
__device__ __forceinline__ void grid_half_scatter(const GridP& g, float* grad, const GridLevelP& lv, const float (&pos)[D], int side, const float (&adjF)[F])
{
    float none[D];
    grid_half_adjoint<D, F, false, true, false, PD>(g, grad, lv, pos, side, adjF, none);
}

// ---- gradients by cell (GradReplicas::byCell) -----------------------------------------------------------------------
// A level with few cells, compared with the points of a batch, adds its gradient up by cell first: a record of the 2^D corners' rows
// per cell, so that a point's contributions are one contiguous piece of memory which several lanes send in one request. The records are then
// added up at the vertices. 2^20 random points, two features, 3-D: 64 bytes by four lanes 12 us, the four pairs of rows of the
// table 25 us (a level of 16^3 to 121^3 vertices; launches not counted).
template <int D, int F>
struct GridCellUnits {
    static constexpr int ROWS = 1 << D, ELEMENTS = ROWS * F;
    static constexpr bool USED = D >= 2 && D <= 4 && (F == 2 || F == 4 || F == 8) && ELEMENTS <= 64;
    static constexpr int UNITS = ELEMENTS / 4;                  // of 16 bytes
    static constexpr int LANES = UNITS < 8 ? UNITS : 8;         // that share a point
};
// The lanes of a group take the group's points in turn. `pos`: this lane's own point; adjoint(r, a): the adjoint of the features of the
// group's r-th point (all lanes of the warp take part). False if this lane's point lies in no cell that has a record.
template <int D, int F, class Adjoint>
__device__ __forceinline__ bool grid_cells_scatter(float* records, const float* end, int* status, const GridLevelP& lv, const float (&pos)[D], bool valid,
                                                   const Adjoint& adjoint)
{
    using C = GridCellUnits<D, F>;
    GridCell<D> c;
    grid_cell<D>(pos, lv.resolution, c);
    unsigned int own = c.lo[0];
#pragma unroll
    for (int k = 1; k < D; ++k) own = c.lo[k] + own * static_cast<unsigned int>(lv.resolution);
    if (!valid || !grid_cell_regular<D>(c, lv)) own = 0xffffffffu;
    const int lane = threadIdx.x % C::LANES;
#pragma unroll
    for (int r = 0; r < C::LANES; ++r) {
        const unsigned int cell = __shfl_sync(0xffffffffu, own, r, C::LANES);
        float f[D], a[F];
#pragma unroll
        for (int k = 0; k < D; ++k) f[k] = __shfl_sync(0xffffffffu, c.f[k], r, C::LANES);
        adjoint(r, a);
        if (cell == 0xffffffffu) continue;
        if (!grid_cell_inside<D>(lv, cell, records + (static_cast<size_t>(cell) + 1) * C::ELEMENTS, end, status)) continue;
        float* at = records + static_cast<size_t>(cell) * C::ELEMENTS + lane * 4;
#pragma unroll
        for (int u = 0; u < C::UNITS; u += C::LANES) {
            const int unit = u + lane;
            if constexpr (F == 2) {   // two rows, neighbours in dimension 0 (weights: the product of grid_corner_weight)
                float w = 1.f;
#pragma unroll
                for (int k = D - 1; k >= 1; --k) w *= ((unit >> (k - 1)) & 1) ? f[k] : (1.f - f[k]);
                const float w0 = w * (1.f - f[0]), w1 = w * f[0];
                red_add_v4_f32(at + u * 4, w0 * a[0], w0 * a[1], w1 * a[0], w1 * a[1]);
            } else {
                const int corner = unit / (F / 4);
                float w = 1.f;
#pragma unroll
                for (int k = D - 1; k >= 0; --k) w *= ((corner >> k) & 1) ? f[k] : (1.f - f[k]);
                if constexpr (F == 4) {
                    red_add_v4_f32(at + u * 4, w * a[0], w * a[1], w * a[2], w * a[3]);
                } else {
                    const bool upper = (unit & 1) != 0;
                    red_add_v4_f32(at + u * 4, w * (upper ? a[4] : a[0]), w * (upper ? a[5] : a[1]), w * (upper ? a[6] : a[2]), w * (upper ? a[7] : a[3]));
                }
            }
        }
    }
    return own != 0xffffffffu || !valid;
}
template <int D>
__host__ __device__ inline unsigned int grid_cell_count(int resolution)
{
    unsigned int n = 1;
    for (int k = 0; k < D; ++k) n *= static_cast<unsigned int>(resolution);
    return n;
}
// records of a level -> its gradient: the cells around a vertex (grid-stride over blockIdx.x, 256 threads)
template <int D, int F>
__device__ __forceinline__ void grid_sum_cells(const GridP& g, const GradReplicas& r, int group, int l)
{
    using C = GridCellUnits<D, F>;
    const GridLevelP& lv = g.levels[l];
    const unsigned int n = grid_cell_count<D>(lv.resolution), res = static_cast<unsigned int>(lv.resolution);
    const int copies = 1 << (r.byCell[group] - 1);
    const float* base = r.base + r.offset[group];
    if (!grid_cell_inside<D>(lv, 0, base + static_cast<size_t>(copies) * n * C::ELEMENTS, r.base + r.capacity, g.status)) return;
    for (unsigned int i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        unsigned int v[D], rest = i;
#pragma unroll
        for (int k = D - 1; k >= 0; --k) {
            const unsigned int q = rest / res;
            v[k] = rest - q * res;
            rest = q;
        }
        double sum[F];   // (2^D cells, 3^D at the upper border, of up to 64 copies each: added in fp32 the terms would cost more than the reductions did)
#pragma unroll
        for (int e = 0; e < F; ++e) sum[e] = 0.0;
        // In every dimension the vertex is the low corner of its own cell, the high corner of the one before, and at the border
        // also the high corner of its own.
        bool border = false;
#pragma unroll
        for (int k = 0; k < D; ++k) border = border || v[k] == res - 1;
        int combinations = 1;
        for (int k = 0; k < D; ++k) combinations *= border ? 3 : 2;
        for (int t = 0; t < combinations; ++t) {
            unsigned int cell = 0, corner = 0;
            bool there = true;
            int digits = t;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int what = border ? digits % 3 : digits & 1;
                digits = border ? digits / 3 : digits >> 1;
                there = there && !(what == 1 && v[k] == 0) && !(what == 2 && v[k] != res - 1);
                cell = (v[k] - (what == 1 ? 1u : 0u)) + cell * res;
                corner |= (what != 0 ? 1u : 0u) << k;
            }
            if (!there) continue;
            const float* at = base + (static_cast<size_t>(cell) * C::ROWS + corner) * F;
            for (int c = 0; c < copies; ++c, at += static_cast<size_t>(n) * C::ELEMENTS) {
                if constexpr (F == 2) {
                    const float2 x = *reinterpret_cast<const float2*>(at);
                    sum[0] += x.x; sum[1] += x.y;
                } else {
#pragma unroll
                    for (int e = 0; e < F; e += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(at + e);
                        sum[e] += x.x; sum[e + 1] += x.y; sum[e + 2] += x.z; sum[e + 3] += x.w;
                    }
                }
            }
        }
        bool any = false;
        float total[F];
#pragma unroll
        for (int e = 0; e < F; ++e) {
            total[e] = static_cast<float>(sum[e]);
            any = any || total[e] != 0.f;   // (also true of NaN)
        }
        if (any) grid_scatter_row<F>(g.grad, grid_checked_index<D, F>(g, lv, grid_vertex_index<D, F>(v, lv)), g.vecOk != 0, 1.f, total);
    }
}

// elements of level l of a table of `levels` levels (levels with copies are small: 32 bits hold every index into them)
__device__ __forceinline__ int grid_level_elements(const GridP& g, int l, int levels)
{
    return static_cast<int>((l + 1 < levels ? g.levels[l + 1].offset : static_cast<unsigned int>(g.tableCount)) - g.levels[l].offset);
}
// where this CTA adds the gradient of level l (level `group` over all grids), seen from element offset 0 of the whole table:
// the table itself or, with copies, one of them
__device__ __forceinline__ float* grid_grad_of_cta(const GridP& g, const GradReplicas& r, int group, int l, int levels)
{
    if (group >= MAX_GRID_LEVELS || r.log2Copies[group] == 0) return g.grad;
    const int n = grid_level_elements(g, l, levels);
    if (BOUNDS_CHECK && n <= 0) return g.grad;   // (a table declared shorter than it is)
    return r.base + r.offset[group] + (blockIdx.x & ((1u << r.log2Copies[group]) - 1u)) * n - g.levels[l].offset;
}
// where this CTA adds up level `group` by cell, null: it does not
template <int D, int F>
__device__ __forceinline__ float* grid_records_of_cta(const GridP& g, const GradReplicas& r, int group, int l)
{
    if constexpr (GridCellUnits<D, F>::USED) {
        if (group < MAX_GRID_LEVELS && r.byCell[group] != 0)
            return r.base + r.offset[group] +
                   static_cast<size_t>(blockIdx.x & ((1u << (r.byCell[group] - 1)) - 1u)) * grid_cell_count<D>(g.levels[l].resolution) * GridCellUnits<D, F>::ELEMENTS;
    }
    return nullptr;
}
// blocks of 256 threads for grid_sum_copies
template <int D, int F>
inline unsigned int grid_sum_blocks(const GridP& g, const GradReplicas& r, int group, int l)
{
    if (group >= MAX_GRID_LEVELS || !GridCellUnits<D, F>::USED || r.byCell[group] == 0) return 32;
    const unsigned int n = (grid_cell_count<D>(g.levels[l].resolution) + 255) / 256;
    return n < 32 ? 32 : (n > 1024 ? 1024 : n);
}
// sum of the copies of a level -> its gradient (grid-stride over blockIdx.x, 256 threads)
template <int D, int F>
__device__ __forceinline__ void grid_sum_copies(const GridP& g, const GradReplicas& r, int group, int l, int levels)
{
    if (group >= MAX_GRID_LEVELS || g.grad == nullptr) return;
    if constexpr (GridCellUnits<D, F>::USED) {
        if (r.byCell[group] != 0) {
            grid_sum_cells<D, F>(g, r, group, l);
            return;
        }
    }
    if (r.log2Copies[group] == 0) return;
    const int copies = 1 << r.log2Copies[group], n = grid_level_elements(g, l, levels);
    const float* src = r.base + r.offset[group];
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        float v = 0.f;
#pragma unroll 8
        for (int c = 0; c < copies; ++c) v += src[c * n + i];
        if (v != 0.f) red_add_f32(g.grad + g.levels[l].offset + i, v);
    }
}

} // namespace kernel
} // namespace qmlp
