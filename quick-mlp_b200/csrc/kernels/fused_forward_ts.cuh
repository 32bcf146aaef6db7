// Fused inference with the activations in tensor memory, for networks up to 128 channels wide whose layer-0 input is at hand
// (identity encodings, or the feature planes of encode_planes_kernel).
//
// Same contract as fused_forward_tc_kernel (replaces NetworkKernelInferenceAndForward,
// src_cpp/include/qmlp/kernels/network_forward.cuh:34-114). That kernel is bound by shared memory up to 64 channels: an MMA
// of 128 x 64 x 16 reads 4 KB of activations and 2 KB of weights at 128 bytes per clock, 48 clocks for an operation that the
// tensor core does in 32, and the epilogues write every activation there first (64-wide network of five layers: about 1570
// of the 1780 clocks a tile took). Here the epilogue writes the next operand to tensor memory (tcgen05.st), the MMA
// takes it from there, and shared memory only delivers weights.
//
//   * One persistent CTA per SM, one warpgroup per tile slot (three for wide networks, which take the blocks of 16 channels in
//     turn). A slot is 128 points in flight: an fp32 accumulator of 64 (32, 128) columns and the fp16 operand of the next
//     layer in 32 (16, 64) columns, two channels per column. 512 columns hold five (eight, two) slots and the constant
//     operand of the bias MMA. Lane = point row = TMEM lane.
//   * Per layer: wait for the accumulator, read it, activate, write the operand, meet on the slot's named barrier; then one
//     warp of the slot issues the K/16 MMAs, the bias MMA (operand [1, 0, ...] x block with the bias in its first K column) and
//     the commit. The issuing warps of the slots sit on different SM sub-partitions.
//   * The features of the slot's next tile are fetched under the layers of the current one.
// Measured, 64-wide network of five layers (relu, celu, sine, relu), 2^22 points: 204 -> 186 us; without its special-function
// operations it would take 122 us, without its MMAs 152: bound by the special-function unit (128 operations per point, 71 %
// busy) with five warps per scheduler to cover the rest. Two warpgroups per slot on four slots: 217 us.
// Every wait is bounded; on a timeout the CTA runs through without waiting and the status word is set.
#pragma once
#include "fused_train_tc.cuh"

namespace qmlp {
namespace kernel {

template <class Spec>
struct TsLayout {
    using TL = TcLayout<Spec>;
    static constexpr int NL = Spec::NUM_LAYERS;
    static constexpr int ACC = TL::maxCout() <= 32 ? 32 : TL::maxCout() <= 64 ? 64 : 128,
                         OPERAND = TL::maxCin() <= 32 ? 16 : TL::maxCin() <= 64 ? 32 : 64, ONES = 8;   // columns
    // warpgroups of a slot: 128 channels fit two slots only (192 columns each); with three warpgroups per slot (two / four) the
    // 64 -> 128 -> 128 -> 128 -> 4 layers of 2^22 points take 309 us (320 / 324; 406 with the operands in shared memory)
    static constexpr int WG = ACC == 128 ? 3 : 1;
    // slots that tensor memory and 1024 threads have room for (one layer of more than 64 outputs on few inputs: three by columns)
    static constexpr int FIT = (512 - ONES) / (ACC + OPERAND), MOST = 8 / WG, SLOTS = FIT < MOST ? FIT : MOST;
    static constexpr int THREADS = SLOTS * WG * 128;
    static_assert(SLOTS >= 1 && THREADS <= 1024, "slots of a CTA");
    __host__ __device__ static constexpr bool wideThroughout()
    {
        for (int i = 0; i + 1 < NL; ++i)
            if (Spec::COUT[i] <= 64) return false;
        return true;
    }
    // Two slots of three warpgroups pay only where every hidden layer keeps them busy: 48 -> 128 -> 64 -> 16 -> 4 with its encode pass,
    // 2^20 points, 287 us against 253 us with the operands in shared memory.
    __host__ __device__ static constexpr bool eligible() { return TL::eligible() && (ACC <= 64 || wideThroughout()); }
    // Points per SM from which the kernel is quicker than the mma.sync one: two tiles, four for networks up to 32 wide (64-wide
    // network 47360 points 7.9 against 9.0 us, 32768 points 7.1 against 6.4; 16-wide 80000 points 4.0 against 5.0, 65536 4.0 / 3.9)
    __host__ __device__ static constexpr long long pointsPerSM() { return ACC == 32 ? 4 * TC_TILE : 2 * TC_TILE; }
    // bias block of layer l: COUT rows of 16 halfs, un-swizzled (bias_block_offset)
    __host__ __device__ static constexpr int biasOffset(int l)
    {
        int o = TL::weightBytes();
        for (int i = 0; i < l; ++i) o += Spec::COUT[i] * 32;
        return o;
    }
    __host__ __device__ static constexpr int barStart() { return (biasOffset(NL) + 127) / 128 * 128; }
    __host__ __device__ static constexpr int bytes() { return barStart() + 256 + 1024; }
};

// D (+)= A * B^T with A in tensor memory
__device__ __forceinline__ void umma_f16_ts_elected(uint32_t lead, uint32_t dTmem, uint32_t aTmem, uint64_t bDesc, uint32_t iDesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(dTmem), "r"(aTmem), "l"(bDesc), "r"(iDesc), "r"(accumulate), "r"(lead) : "memory");
}
// 8 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

template <class Spec>
struct TsSlot {
    static constexpr int WG = TsLayout<Spec>::WG, STEPS = (Spec::CIN[0] / 16 + WG - 1) / WG;   // 16-channel steps this thread writes
    uint32_t tmem;          // accumulator, lane field of this warp included; the operand follows
    uint32_t full, parity;  // mbarrier the MMAs commit to
    long long point;
    uint32_t features[STEPS][2][4];   // of the next tile
};

template <class Spec, int K>
__device__ __forceinline__ void ts_fetch(const LaunchArgs& p, TsSlot<Spec>& sl, int wg, long long point)
{
    constexpr int WG = TsSlot<Spec>::WG;
    if constexpr (K * 16 < Spec::CIN[0]) {
        if (wg == K % WG) {
            fetch_piece<Spec, K * 16, K * 16 + 8>(p, point, sl.features[K / WG][0]);
            fetch_piece<Spec, K * 16 + 8, K * 16 + 16>(p, point, sl.features[K / WG][1]);
        }
        ts_fetch<Spec, K + 1>(p, sl, wg, point);
    }
}

template <class Spec, int L>
__device__ __forceinline__ void ts_issue(uint32_t lead, uint32_t smem, uint32_t slotTmem, uint32_t onesTmem, uint32_t full)
{
    using TS = TsLayout<Spec>;
    constexpr int CIN = Spec::CIN[L], COUT = Spec::COUT[L];
    constexpr uint32_t idesc = umma_idesc_f16(TC_TILE, COUT);
    const uint64_t b = umma_desc_sw128(smem + TcLayout<Spec>::wOffset(L));
#pragma unroll
    for (int k = 0; k < CIN / 16; ++k) umma_f16_ts_elected(lead, slotTmem, slotTmem + TS::ACC + k * 8, b + (((k >> 2) * (COUT * 128) + (k & 3) * 32) >> 4), idesc, k > 0 ? 1u : 0u);
    if constexpr (Spec::BOFF[L] >= 0) umma_f16_ts_elected(lead, slotTmem, onesTmem, umma_desc_k16_noswizzle(smem + TS::biasOffset(L)), idesc, 1u);
    umma_commit_elected(lead, full);
}

// Stage 0: features -> operand of layer 0. Stage L + 1: epilogue of layer L. Every stage but the last ends with the MMAs of the
// next layer.
template <class Spec, int ST>
__device__ __forceinline__ void ts_stages(const LaunchArgs& p, TsSlot<Spec>& sl, uint32_t smem, uint32_t onesTmem, int wg, int barrierId, bool issuer, uint32_t lead,
                                          long long next, volatile int* abortFlag, bool& dead)
{
    using TS = TsLayout<Spec>;
    constexpr int NL = Spec::NUM_LAYERS;
    constexpr int WG = TS::WG;
    if constexpr (ST == 0) {
        constexpr int CIN0 = Spec::CIN[0];
#pragma unroll
        for (int k = 0; k < TsSlot<Spec>::STEPS; ++k) {
            const int step = wg + k * WG;
            if (step * 16 >= CIN0) continue;
            const uint32_t (&a)[4] = sl.features[k][0], (&b)[4] = sl.features[k][1];
            const uint32_t v[8] = {a[0], a[1], a[2], a[3], b[0], b[1], b[2], b[3]};
            tmem_st8(sl.tmem + TS::ACC + step * 8, v);
        }
        if (next < p.numel) ts_fetch<Spec, 0>(p, sl, wg, next);
    } else {
        constexpr int L = ST - 1, COUT = Spec::COUT[L];
        using Act = typename Spec::template Act<L>;
        train_wait(sl.full, sl.parity, abortFlag, dead);
        sl.parity ^= 1u;
        __syncwarp();   // tcgen05.ld is warp-collective
        tc_fence_after();
        if constexpr (ST < NL) {
            // the warpgroups take the blocks of 16 columns in turn; two blocks per wait
            constexpr int BLOCKS = (COUT / 16 + WG - 1) / WG;
#pragma unroll
            for (int b0 = 0; b0 < BLOCKS; b0 += 2) {
                float v[2][16];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int col = (wg + (b0 + b) * WG) * 16;
                    if (b0 + b < BLOCKS && col < COUT) tmem_ld16(sl.tmem + col, v[b]);
                }
                tmem_wait_ld();
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int col = (wg + (b0 + b) * WG) * 16;
                    if (b0 + b >= BLOCKS || col >= COUT) continue;
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = h2_as_u32(act_forward_f32x2<Act>(v[b][2 * i], v[b][2 * i + 1], col + 2 * i));
                    tmem_st8(sl.tmem + TS::ACC + col / 2, w);
                }
            }
        } else {
            // first NUM_OUTPUTS channels -> fp32 (kernels/network_forward.cuh:103-111)
            constexpr int OUT = Spec::NUM_OUTPUTS;
#pragma unroll
            for (int c0 = 0; c0 < OUT; c0 += 8) {
                if (c0 / 8 % WG != wg) continue;
                float v[8];
                tmem_ld8(sl.tmem + c0, v);
                tmem_wait_ld();
                if (sl.point < p.numel) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __half22float2(act_forward_f32x2<Act>(v[2 * i], v[2 * i + 1], c0 + 2 * i));
                        const int c = c0 + 2 * i;
                        if (c < OUT) p.output[sl.point * p.outS0 + c * p.outS1] = f.x;
                        if (c + 1 < OUT) p.output[sl.point * p.outS0 + (c + 1) * p.outS1] = f.y;
                    }
                }
            }
        }
    }
    if constexpr (ST < NL) {
        tmem_wait_st();
        tc_fence_before();
        asm volatile("bar.sync %0, %1;" ::"r"(barrierId), "n"(WG * 128) : "memory");
        if (issuer && !dead) {
            tc_fence_after();
            ts_issue<Spec, ST>(lead, smem, sl.tmem & 0x0000ffffu, onesTmem, sl.full);
        }
        ts_stages<Spec, ST + 1>(p, sl, smem, onesTmem, wg, barrierId, issuer, lead, next, abortFlag, dead);
    }
}

// bias of layer L -> first K column of its block (whole CTA)
template <class Spec, int L>
__device__ __forceinline__ void ts_stage_bias(const LaunchArgs& p, unsigned char* smem)
{
    if constexpr (L < Spec::NUM_LAYERS) {
        constexpr int COUT = Spec::COUT[L];
        if constexpr (Spec::BOFF[L] >= 0)
            for (int i = threadIdx.x; i < COUT * 16; i += TsLayout<Spec>::THREADS) {
                const int r = i >> 4, k = i & 15;
                *reinterpret_cast<__half*>(smem + TsLayout<Spec>::biasOffset(L) + bias_block_offset(r, k)) = k == 0 ? p.weights[Spec::BOFF[L] + r] : __ushort_as_half(0);
            }
        ts_stage_bias<Spec, L + 1>(p, smem);
    }
}

template <class Spec>
__global__ void __launch_bounds__(TsLayout<Spec>::THREADS, 1)
fused_forward_ts_kernel(const __grid_constant__ LaunchArgs p, const __grid_constant__ TcWeightMaps<Spec> weightMaps)
{
    using TL = TcLayout<Spec>;
    using TS = TsLayout<Spec>;
    extern __shared__ unsigned char smemRaw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    // per slot: the MMAs' barrier and the one that drains them after a timeout; then the weight staging
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TS::barStart());
    uint64_t* weightBar = bars + 2 * TS::SLOTS;
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(weightBar + 1);
    volatile int* abortFlag = reinterpret_cast<int*>(tmemSlot + 1);
    const uint32_t smemBase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, slot = (warp >> 2) / TS::WG, wg = (warp >> 2) % TS::WG, row = threadIdx.x & 127;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(weightBar), 1);
        for (int s = 0; s < 2 * TS::SLOTS; ++s) mbar_init(smem_u32(bars + s), 1);
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(smem_u32(weightBar), TL::weightCopyBytes());
        tc_issue_weight_copies<Spec, 0>(weightMaps, smemBase, smem_u32(weightBar));
    }
    const int numTiles = static_cast<int>((p.numel + TC_TILE - 1) / TC_TILE);
    const int stride = gridDim.x;
    const int myTiles = static_cast<int>(blockIdx.x) < numTiles ? (numTiles - static_cast<int>(blockIdx.x) + stride - 1) / stride : 0;
    auto pointOf = [&](int i) { return i < myTiles ? (blockIdx.x + static_cast<long long>(i) * stride) * TC_TILE + row : p.numel; };
    // tile i of this CTA's sequence belongs to slot i % SLOTS
    TsSlot<Spec> sl;
    sl.point = pointOf(slot);
#pragma unroll
    for (int k = 0; k < TsSlot<Spec>::STEPS; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i) sl.features[k][i / 4][i % 4] = 0u;
    if (sl.point < p.numel) ts_fetch<Spec, 0>(p, sl, wg, sl.point);
    ts_stage_bias<Spec, 0>(p, smem);
    if (warp == 0) {
        tmem_alloc(smem_u32(tmemSlot), 512);
        tmem_relinquish();
    }
    fence_proxy_async();   // bias blocks written by the threads -> visible to the tensor core
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmemBase = *tmemSlot;
    const uint32_t laneField = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t onesTmem = tmemBase + TS::SLOTS * (TS::ACC + TS::OPERAND);
    if (warp < 4) {   // constant operand of the bias MMA: every row = [1, 0, ..., 0]
        const uint32_t one[8] = {0x3C00u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        tmem_st8(onesTmem + laneField, one);
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    bool dead = false;
    sl.tmem = tmemBase + slot * (TS::ACC + TS::OPERAND) + laneField;
    sl.full = smem_u32(bars + 2 * slot);
    sl.parity = 0;
    const bool issuer = wg == 0 && (warp & 3) == (slot & 3);
    const uint32_t lead = elect_one();
    train_wait(smem_u32(weightBar), 0, abortFlag, dead);
    __syncwarp();
    for (int i = slot; i < myTiles; i += TS::SLOTS) {
        const long long next = pointOf(i + TS::SLOTS);
        ts_stages<Spec, 0>(p, sl, smemBase, onesTmem, wg, 1 + slot, issuer, lead, next, abortFlag, dead);
        sl.point = next;
    }
    if (issuer && __any_sync(0xffffffffu, dead)) {   // gave up: let the MMAs in flight finish
        umma_commit_elected(lead, sl.full + 8);
        mbar_wait(sl.full + 8, 0);
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmemBase, 512);
    }
    if (threadIdx.x == 0 && *abortFlag != 0 && p.status != nullptr) atomicOr(p.status, STATUS_WAIT_TIMEOUT);
}

template <class Spec>
struct TsLaunchers {
    static cudaError_t run(const LaunchArgs& a, cudaStream_t s)
    {
        using TS = TsLayout<Spec>;
        static DeviceOnce once;
        auto k = fused_forward_ts_kernel<Spec>;
        const cudaError_t e = once.run([&] { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TS::bytes()); });
        if (e != cudaSuccess) return e;
        const TcWeightMaps<Spec>* maps = nullptr;
        const cudaError_t m = TcLaunchers<Spec>::weightMaps(a.weights, maps);
        if (m != cudaSuccess) return m;
        const long long tiles = (a.numel + TC_TILE - 1) / TC_TILE;
        const long long blocks = tiles < a.numSMs ? tiles : a.numSMs;
        k<<<static_cast<unsigned>(blocks < 1 ? 1 : blocks), TS::THREADS, TS::bytes(), s>>>(a, *maps);
        return cudaGetLastError();
    }
};

} // namespace kernel
} // namespace qmlp
