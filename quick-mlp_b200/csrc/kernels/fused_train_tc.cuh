// Layer chain of a training step on the 5th-generation tensor cores: forward, L2 loss, backward and the weight / bias
// gradients of all layers in one kernel (replaces, for the training step, the reference's
// NetworkKernelInferenceAndForward, NetworkKernelBackward and WeightUpdateSingleBlockKernel,
// src_cpp/include/qmlp/kernels/network_forward.cuh:34-114, network_backward.cuh:33-114,
// network_weight_update_block.cuh:356-494).
//
// Features come from, and their adjoints go to, the level-major planes of kernels/grid_planes.cuh. Nothing else of a point
// reaches global memory: with one kernel per phase the pre-activations and deltas of every layer were written once and read
// back twice (1.3 KB per point for 32 -> 64 -> 64 -> 1).
//
//   * One persistent CTA per SM. A tile is 128 points; the CTA has as many tile slots as shared and tensor memory hold, four of one
//     warpgroup, three of one, two of two, or one of four, and a warp that issues weight gradients. The slots run independently: the MMAs
//     of one run under the epilogues of the others. Thread = (point row, column share): the warpgroups of a slot take the
//     blocks of 8 columns of an accumulator row in turn.
//   * Shared memory, all in the 128-byte swizzled layout (rows = points, 64 channels per block): the weights (staged by
//     TMA), per slot one buffer per layer input. The delta of layer l - 1 overwrites the input of layer l, which has the same shape
//     and is dead once the weight gradient of layer l is done; the last delta lies in channels that an input leaves free.
//   * Tensor memory: per slot one accumulator for the layers and the adjoints one after the other, and packed pre-activations as far as
//     columns are left (the others stay in registers); and the weight-gradient accumulators of all layers, which stay for the whole
//     kernel and are added to the gradient vector once per CTA.
//   * Weight gradients are MMAs over K = the 128 points of the tile: both operands are the tiles above read MN-major. Either
//     delta^T * input (M = outputs) or input^T * delta (M = inputs), whichever needs fewer columns. The bias gradient is one
//     more column (or row) of the same MMA: a channel of ones in the padding of the input's block, or a block of ones behind it
//     that holds 16 points only, which each of the MMAs reads again.
//   * A slot's warps meet on a named barrier at the end of a stage, and one of them issues the MMAs of the next. The weight gradients of
//     all slots go to the same accumulators, so one warp issues all of them, in order: it reads requests from a ring in shared memory
//     (one word to watch; with a barrier per slot to poll it took 500 clocks to notice). They only have to be done when the next stage of
//     the slot overwrites their operands, and that stage computes all its deltas before it waits.
// Measured, step of 32 -> 64 -> 64 -> 1 on 2^20 points: 94 (forward) + 123 (backward) + 127 us (weight gradients) -> 137 us with two slots
// of two warpgroups -> 111 us with four of one; 48 -> 128 -> 64 -> 16 -> 4 on 2^21 points: 709 (with the gather) + 1022 (with the scatter)
// + 473 -> 577 us with accumulators computed a second time -> 576 us (111 and 564 while a slot's warps did not wait for each other at the
// end of a stage). What it spends (clocks of the first example, measured in the kernel):
// a tile's MMAs 1970, 54 % of the time per tile (K = 16 takes 40 to 49 clocks from shared memory however few columns, 33 from tensor
// memory, for which there are no columns left); a slot's stage 2000: 450 waiting for the accumulator behind other slots' MMAs, 1000
// of epilogue, 130 fences, 300 to issue. Features fetched before the last stage are spilled, and a spill waits for the load (1500 clocks).
// Every wait on the tensor core or a copy is bounded. After one that gave up the CTA runs through without them and sets the status word; what its
// warps still wait for then is each other, at barriers that each of them reaches.
//
// The second instantiation (LOSS false) is the backward pass of a forward call that stashed the encoded features only: the layers
// are computed a second time on the tensor core instead of being written by the forward kernel and read twice. 32 -> 64 -> 64 -> 1
// on 2^18 points: forward 104 -> 93 us, backward and weight gradients 71 -> 42 us.
//
// Same roundings as the separate kernels: fp16 activations, deltas and pre-activations (bias added in half), fp32 sums.
#pragma once
#include "fused_forward_tc.cuh"

namespace qmlp {
namespace kernel {

constexpr int TRAIN_BLOCK = TC_TILE * 128;   // bytes of a block: 128 points x 64 channels
constexpr int TRAIN_ONES = 2048;             // and of the block of ones: 16 points

// LOSS: the training step's kernel (features from the planes, L2 loss against targets); else the backward pass of an earlier
// forward call (features from its stash, the adjoint of the output from the caller)
template <class Spec, bool LOSS = true>
struct TrainLayout {
    using TL = TcLayout<Spec>;
    static constexpr int NL = Spec::NUM_LAYERS;
    static constexpr bool FEATURE_ADJOINT = !LOSS || table_rows_per_point<Spec>() > 0;   // the adjoint of the features is wanted
    __host__ __device__ static constexpr int blocks(int channels) { return (channels + 63) / 64; }
    __host__ __device__ static constexpr bool bias(int l) { return Spec::BOFF[l] >= 0; }
    // buffer l < NL: input of layer l (later delta of layer l - 1); buffer NL: delta of the last layer. A narrow last delta lies in the
    // last channels of the first input's block that has room for it behind the input and the channel of ones.
    __host__ __device__ static constexpr int lastHost()
    {
        for (int i = 0; i < NL; ++i)
            if (Spec::CIN[i] + 16 + Spec::COUT[NL - 1] <= 64) return i;
        return -1;
    }
    static constexpr int LAST_BUFFER = lastHost() >= 0 ? lastHost() : NL, LAST_CHUNK = lastHost() >= 0 ? 8 - Spec::COUT[NL - 1] / 8 : 0;
    __host__ __device__ static constexpr int bufOffset(int l)
    {
        int o = 0;
        for (int i = 0; i < l && i < NL; ++i) o += blocks(Spec::CIN[i]) * TRAIN_BLOCK;
        return o;   // (l == NL: behind the last input)
    }
    // byte offset of the delta of layer l in the slot (its first channel, row 0)
    __host__ __device__ static constexpr int deltaOffset(int l) { return l < NL - 1 ? bufOffset(l + 1) : bufOffset(LAST_BUFFER) + LAST_CHUNK * 16; }
    __host__ __device__ static constexpr int slotBytes() { return bufOffset(NL) + (lastHost() >= 0 ? 0 : blocks(Spec::COUT[NL - 1]) * TRAIN_BLOCK); }

    // weight gradient of layer l: columns if M = outputs / M = inputs, the bias included where it comes for free
    __host__ __device__ static constexpr int colsOut(int l) { return bias(l) ? Spec::CIN[l] + 16 : Spec::CIN[l]; }
    __host__ __device__ static constexpr int colsIn(int l) { return Spec::COUT[l] + (separateBias(l) ? 16 : 0); }
    __host__ __device__ static constexpr bool mIsOut(int l) { return colsOut(l) < colsIn(l); }
    __host__ __device__ static constexpr int wgCols(int l) { return mIsOut(l) ? colsOut(l) : colsIn(l); }
    // the bias needs an MMA of its own against the block of ones
    __host__ __device__ static constexpr bool separateBias(int l) { return bias(l) && Spec::CIN[l] == 128; }
    __host__ __device__ static constexpr int wgCol(int l)
    {
        int c = 0;
        for (int i = 0; i < l; ++i) c += wgCols(i);
        return c;
    }
    __host__ __device__ static constexpr int dBefore(int l)   // outputs of the layers before l
    {
        int c = 0;
        for (int i = 0; i < l; ++i) c += Spec::COUT[i];
        return c;
    }
    // accumulator columns of a slot: one region that the layers' outputs, their adjoints and the adjoint of the features share
    __host__ __device__ static constexpr int slotCols()
    {
        int m = Spec::COUT[NL - 1];
        for (int i = FEATURE_ADJOINT ? 0 : 1; i < NL; ++i) m = Spec::CIN[i] > m ? Spec::CIN[i] : m;
        return m;
    }
    __host__ __device__ static constexpr int slotStart() { return TL::weightBytes(); }
    __host__ __device__ static constexpr int onesStart(int slots) { return slotStart() + slots * slotBytes(); }
    __host__ __device__ static constexpr int biasStart(int slots) { return onesStart(slots) + TRAIN_ONES; }
    __host__ __device__ static constexpr int barStart(int slots) { return biasStart(slots) + (dBefore(NL) * 2 + 127) / 128 * 128; }
    // barriers, arrival counters and flags (fused_train_tc_kernel)
    __host__ __device__ static constexpr int bytes(int slots) { return barStart(slots) + 384 + 1024; }
    __host__ __device__ static constexpr int queueStart() { return barStart(SLOTS) + 8 * (2 * SLOTS + 1 + THREADS / 32); }
    __host__ __device__ static constexpr bool fits(int slots) { return slots * slotCols() + wgCol(NL) <= 512 && bytes(slots) <= 227 * 1024; }
    // The pre-activations of the layers but the last wait for the backward pass as packed halfs: in tensor memory, first layers first, as far
    // as columns are left, else in registers.
    __host__ __device__ static constexpr int spareCols(int slots) { return (512 - wgCol(NL) - slots * slotCols()) / slots / 16 * 16; }
    __host__ __device__ static constexpr int preCol(int l, int slots)   // first column behind the slot's accumulator, -1: registers
    {
        int c = 0;
        for (int i = 0; i < NL - 1; ++i) {
            const bool room = c + Spec::COUT[i] / 2 <= spareCols(slots);
            if (i == l) return room ? c : -1;
            if (room) c += Spec::COUT[i] / 2;
        }
        return -1;
    }
    __host__ __device__ static constexpr int preBefore(int l, int slots, int wg)   // registers of a thread before those of layer l
    {
        int r = 0;
        for (int i = 0; i < l; ++i)
            if (preCol(i, slots) < 0) r += (Spec::COUT[i] / 8 + wg - 1) / wg * 4;
        return r;
    }
    __host__ __device__ static constexpr int slotStride(int slots) { return slotCols() + spareCols(slots); }   // columns of a slot
    // Slots and warpgroups per slot: as many slots as there is room for, the stages of a tile being latency (see above). 17 warps have 96
    // registers a thread, 13 have 128. Also at few tiles per CTA, where half the threads work on each: 32 -> 64 -> 64 -> 1, 0.4 / 1 / 2 / 4 / 8 / 16
    // tiles per CTA, two slots of two warpgroups 14.8 / 18.9 / 22.9 / 27.0 / 33.2 / 51.3 us, four of one 14.8 / 19.0 / 22.9 / 25.0 / 29.2 / 43.4;
    // 3 -> 64 x 4 -> 1 22.3 / 27.1 / 34.7 / 49.3 / 78.2 / 135 and 22.2 / 27.0 / 29.1 / 38.6 / 57.2 / 92.1.
    __host__ __device__ static constexpr bool holds(int slots, int wg, int registers) { return fits(slots) && preBefore(NL - 1, slots, wg) <= registers; }
    static constexpr int SLOTS = holds(4, 1, 40) ? 4 : holds(3, 1, 72) ? 3 : holds(2, 2, 48) ? 2 : 1;
    static constexpr int WG = SLOTS >= 3 ? 1 : SLOTS == 2 ? 2 : 4;
    static constexpr int WARPGROUPS = SLOTS * WG, THREADS = WARPGROUPS * 128 + 32;   // the last warp issues the weight gradients
    __host__ __device__ static constexpr int preCol(int l) { return preCol(l, SLOTS); }
    __host__ __device__ static constexpr int preBefore(int l) { return preBefore(l, SLOTS, WG); }
    __host__ __device__ static constexpr int slotStride() { return slotStride(SLOTS); }
    // Stages: 0 features, 1 .. NL - 1 activations, NL loss, then the deltas of the layers NL - 2 .. 0, then the adjoint of the features.
    __host__ __device__ static constexpr int lastStage() { return 2 * NL; }
    __host__ __device__ static constexpr int stepLayer(int stage) { return 2 * NL - 1 - stage; }   // layer whose delta stage `stage` computes (NL < stage < lastStage())
    // (TcLayout: the encode pass exists for the same networks)
    __host__ __device__ static constexpr bool eligible() { return TL::eligible() && fits(1); }
};

// K-major tile or weight block read along its rows' channels (MN-major operand): 64-channel blocks `lbo` bytes apart,
// groups of 8 rows (along K) 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smemAddr, uint32_t lbo)
{
    return static_cast<uint64_t>((smemAddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) | (64ull << 32) | (1ull << 46) |
           (2ull << 61);
}
constexpr uint32_t UMMA_A_MN = 1u << 15, UMMA_B_MN = 1u << 16;

// 8 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// 4 packed words at consecutive columns
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&v)[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The whole issuing warp runs the issue code, so that descriptors and addresses live in uniform registers; only the
// elected lane's instruction takes effect. (Behind a `lane == 0` branch every operand has to be moved to a uniform register
// first: 16 MMAs with N = 64 take 773 instead of 596 clocks to issue.)
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}
__device__ __forceinline__ void umma_f16_elected(uint32_t lead, uint32_t dTmem, uint64_t aDesc, uint64_t bDesc, uint32_t iDesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(dTmem), "l"(aDesc), "l"(bDesc), "r"(iDesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ __forceinline__ void umma_commit_elected(uint32_t lead, uint32_t bar)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead) : "memory");
}
// polls of a wait before it gives up (bounds-checking instantiations: the host's, a test hook)
__device__ __forceinline__ uint32_t train_spin_limit(const LaunchArgs& p)
{
    if constexpr (BOUNDS_CHECK) return p.spinLimit;
    (void)p;
    return TC_SPIN_LIMIT;
}
// Bounded wait. When one gives up it raises the CTA's abort flag; from then on nobody waits any more (`dead`), so that the
// CTA runs through to its end.
__device__ __forceinline__ void train_wait(uint32_t bar, uint32_t parity, volatile int* abortFlag, bool& dead, uint32_t limit = TC_SPIN_LIMIT)
{
    if (dead) return;
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_test(bar, parity)) return;
        if ((i & 1023u) == 1023u && *abortFlag != 0) break;
    }
    *abortFlag = 1;
    dead = true;
}

// ---- features of a point in pieces of 8 channels ------------------------------------------------------------------------
// encoding that channel C of the encoded input belongs to (-1: padding)
template <class Spec, int C, int E = 0>
__host__ __device__ constexpr int channel_encoding()
{
    if constexpr (E >= Spec::NUM_ENCODINGS) return -1;
    else {
        using Enc = typename Spec::template Enc<E>;
        if constexpr (C >= Enc::OUT_OFF && C < Enc::OUT_OFF + Enc::NUM_OUT) return E;
        else return channel_encoding<Spec, C, E + 1>();
    }
}
// features of a grid level (one plane) from channel C on that fit one vector access and the piece
template <class Enc, int C>
__host__ __device__ constexpr int plane_vector()
{
    constexpr int i = (C - Enc::OUT_OFF) % Enc::F, left = 8 - C % 8;
    int w = 1;
    while (w < 8 && C % 2 == 0 && Enc::F % (2 * w) == 0 && i % (2 * w) == 0 && 2 * w <= left) w *= 2;
    return w;
}

// channels [C, END) of a point -> v (packed halfs, channel C % 8 first); END - 8 is a multiple of 8
template <class Spec, int C, int END>
__device__ __forceinline__ void fetch_piece(const LaunchArgs& p, long long point, uint32_t (&v)[4])
{
    if constexpr (C < END) {
        constexpr int E = channel_encoding<Spec, C>();
        constexpr int j = C % 8;
        if constexpr (E < 0) {   // padding up to the layer width
            if constexpr (j % 2 == 0) v[j / 2] = 0u;
            fetch_piece<Spec, C + 1, END>(p, point, v);
        } else {
            using Enc = typename Spec::template Enc<E>;
            if constexpr (!Enc::IS_GRID) {
                const __half h = __float2half(__ldg(p.input + point * p.inS0 + (C - Enc::OUT_OFF + Enc::START) * p.inS1));
                const uint32_t b = static_cast<uint32_t>(__half_as_ushort(h));
                v[j / 2] = j % 2 == 0 ? b : (v[j / 2] | (b << 16));
                fetch_piece<Spec, C + 1, END>(p, point, v);
            } else {
                constexpr int F = Enc::F, i = (C - Enc::OUT_OFF) % F, W = plane_vector<Enc, C>();
                const __half* at = p.planes + p.planeStride * (C - i) + point * F + i;
                if (!scratch_ok(p, at - p.planes, W, p.planeHalfs, STATUS_PLANES)) {
#pragma unroll
                    for (int w = j; w < j + W; w += 2)
                        if (w % 2 == 0) v[w / 2] = 0u;
                } else if constexpr (W == 8) {
                    const uint4 u = *reinterpret_cast<const uint4*>(at);
                    v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
                } else if constexpr (W == 4) {
                    const uint2 u = *reinterpret_cast<const uint2*>(at);
                    v[j / 2] = u.x; v[j / 2 + 1] = u.y;
                } else if constexpr (W == 2) {
                    v[j / 2] = *reinterpret_cast<const uint32_t*>(at);
                } else {
                    const uint32_t b = static_cast<uint32_t>(__half_as_ushort(*at));
                    v[j / 2] = j % 2 == 0 ? b : (v[j / 2] | (b << 16));
                }
                fetch_piece<Spec, C + W, END>(p, point, v);
            }
        }
    }
}
// adjoints of channels [C, END) -> planes of the grids (if any), gradient of the input for identity encodings (if wanted; an
// input channel may feed several encodings)
template <class Spec, int C, int END>
__device__ __forceinline__ void store_piece(const LaunchArgs& p, long long point, const uint32_t (&v)[4])
{
    if constexpr (C < END) {
        constexpr int E = channel_encoding<Spec, C>();
        constexpr int j = C % 8;
        if constexpr (E >= 0) {
            using Enc = typename Spec::template Enc<E>;
            if constexpr (!Enc::IS_GRID) {
                if (p.adjInput != nullptr)
                    red_add_f32(p.adjInput + point * p.aiS0 + (C - Enc::OUT_OFF + Enc::START) * p.aiS1,
                                __half2float(__ushort_as_half(static_cast<unsigned short>(j % 2 == 0 ? v[j / 2] & 0xffffu : v[j / 2] >> 16))));
            } else {
                constexpr int F = Enc::F, i = (C - Enc::OUT_OFF) % F, W = plane_vector<Enc, C>();
                __half* at = p.planes + p.planeStride * (C - i) + point * F + i;
                if (p.planes == nullptr || !scratch_ok(p, at - p.planes, W, p.planeHalfs, STATUS_PLANES)) {}
                else if constexpr (W == 8) *reinterpret_cast<uint4*>(at) = make_uint4(v[0], v[1], v[2], v[3]);
                else if constexpr (W == 4) *reinterpret_cast<uint2*>(at) = make_uint2(v[j / 2], v[j / 2 + 1]);
                else if constexpr (W == 2) *reinterpret_cast<uint32_t*>(at) = v[j / 2];
                else *at = __ushort_as_half(static_cast<unsigned short>(j % 2 == 0 ? v[j / 2] & 0xffffu : v[j / 2] >> 16));
                store_piece<Spec, C + W, END>(p, point, v);
                return;
            }
        }
        store_piece<Spec, C + 1, END>(p, point, v);
    }
}

// ---- MMAs (issued by one elected lane of a whole warp) --------------------------------------------------------------------------------------------
template <class Spec, bool LOSS>
struct TrainIssue {
    using TL = TcLayout<Spec>;
    using TR = TrainLayout<Spec, LOSS>;
    // outputs of layer L = input * W^T, to column `dTmem`
    template <int L>
    static __device__ __forceinline__ void forward(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t dTmem)
    {
        constexpr int CIN = Spec::CIN[L], COUT = Spec::COUT[L];
        const uint64_t a = umma_desc_sw128(slotSmem + TR::bufOffset(L)), b = umma_desc_sw128(smem + TL::wOffset(L));
#pragma unroll
        for (int k = 0; k < CIN / 16; ++k)
            umma_f16_elected(lead, dTmem, a + (((k >> 2) * TRAIN_BLOCK + (k & 3) * 32) >> 4), b + (((k >> 2) * (COUT * 128) + (k & 3) * 32) >> 4),
                             umma_idesc_f16(TC_TILE, COUT), k > 0 ? 1u : 0u);
    }
    // adjoint of the inputs of layer L = delta * W, to column `dTmem`
    template <int L>
    static __device__ __forceinline__ void adjoint(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t dTmem)
    {
        constexpr int COUT = Spec::COUT[L];
        const uint64_t a = umma_desc_sw128(slotSmem + TR::deltaOffset(L)), b = umma_desc_mn_sw128(smem + TL::wOffset(L), COUT * 128);
#pragma unroll
        for (int k = 0; k < COUT / 16; ++k)
            umma_f16_elected(lead, dTmem, a + (((k >> 2) * TRAIN_BLOCK + (k & 3) * 32) >> 4), b + ((k * 2048) >> 4),
                             umma_idesc_f16(TC_TILE, Spec::CIN[L]) | UMMA_B_MN, k > 0 ? 1u : 0u);
    }
    // weight (and bias) gradient of layer L
    template <int L>
    static __device__ __forceinline__ void gradient(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t wgTmem, uint32_t accumulate)
    {
        constexpr int CIN = Spec::CIN[L];
        const uint32_t delta = slotSmem + TR::deltaOffset(L), input = slotSmem + TR::bufOffset(L), ones = smem + TR::onesStart(TR::SLOTS);
        // The 64 channels behind an operand of one block are the block of ones: the input's channel of ones where its own block is full,
        // else rows of the result that are not read (M is always 128). It holds 16 points, which every MMA reads: its distance
        // shrinks as the operand's address grows.
        constexpr bool OUT = TR::mIsOut(L);
        constexpr bool DELTA_WIDE = Spec::COUT[L] > 64, INPUT_WIDE = CIN > 64;
        const uint64_t d = umma_desc_mn_sw128(delta, DELTA_WIDE ? TRAIN_BLOCK : ones - delta), i = umma_desc_mn_sw128(input, INPUT_WIDE ? TRAIN_BLOCK : ones - input);
        constexpr uint64_t STEP = 2048 >> 4, WIDE_STEP = STEP, NARROW_STEP = STEP - (STEP << 16);
        constexpr int N = OUT ? CIN + (TR::bias(L) && CIN != 128 ? 16 : 0) : Spec::COUT[L];
#pragma unroll
        for (int k = 0; k < TC_TILE / 16; ++k) {
            const uint64_t dk = d + k * (DELTA_WIDE ? WIDE_STEP : NARROW_STEP), ik = i + k * (INPUT_WIDE ? WIDE_STEP : NARROW_STEP);
            umma_f16_elected(lead, wgTmem + TR::wgCol(L), OUT ? dk : ik, OUT ? ik : dk, umma_idesc_f16(TC_TILE, N) | UMMA_A_MN | UMMA_B_MN, k == 0 ? accumulate : 1u);
        }
        if constexpr (TR::separateBias(L)) {
            const uint64_t o = umma_desc_mn_sw128(ones, TRAIN_BLOCK);   // (16 channels of it)
#pragma unroll
            for (int k = 0; k < TC_TILE / 16; ++k)
                umma_f16_elected(lead, wgTmem + TR::wgCol(L) + N, d + k * (DELTA_WIDE ? WIDE_STEP : NARROW_STEP), o, umma_idesc_f16(TC_TILE, 16) | UMMA_A_MN | UMMA_B_MN,
                                 k == 0 ? accumulate : 1u);
        }
    }
    // what the next stage of the slot waits for after stage ST
    template <int ST>
    static __device__ __forceinline__ void critical(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t slotTmem, uint32_t bars)
    {
        constexpr int NL = Spec::NUM_LAYERS, NEXT = ST + 1;
        if constexpr (ST < NL) {
            forward<ST>(lead, smem, slotSmem, slotTmem);
            umma_commit_elected(lead, bars);
        } else if constexpr (NEXT < TR::lastStage()) {
            adjoint<TR::stepLayer(NEXT) + 1>(lead, smem, slotSmem, slotTmem);
            umma_commit_elected(lead, bars);
        } else if constexpr (TR::FEATURE_ADJOINT) {
            adjoint<0>(lead, smem, slotSmem, slotTmem);
            umma_commit_elected(lead, bars);
        }
    }
    // layer whose delta is complete after stage ST (-1: none)
    template <int ST>
    __host__ __device__ static constexpr int graded()
    {
        constexpr int NL = Spec::NUM_LAYERS;
        if constexpr (ST < NL) return -1;
        else if constexpr (ST == NL) return NL - 1;
        else return ST < TR::lastStage() ? TR::stepLayer(ST) : -1;
    }
    // weight gradient of layer `layer`. `started`: layers whose accumulator holds sums already
    template <int L>
    static __device__ __forceinline__ void weights(uint32_t lead, int layer, uint32_t smem, uint32_t slotSmem, uint32_t wgTmem, uint32_t& started, uint32_t bars)
    {
        if constexpr (L < Spec::NUM_LAYERS) {
            if (layer != L) {
                weights<L + 1>(lead, layer, smem, slotSmem, wgTmem, started, bars);
            } else {
                gradient<L>(lead, smem, slotSmem, wgTmem, (started >> L) & 1u);
                started |= 1u << L;
                umma_commit_elected(lead, bars + 8);
            }
        }
    }
};

// ---- requests for weight gradients: a ring of entries that the issuing warps of the slots fill and the weight-gradient warp empties ----
// An entry carries its number, so that the reader of entry n knows it from the one before in its place. A slot asks for one layer at a
// time, the next time only after the gradient before is done: the ring never overruns.
constexpr int TRAIN_QUEUE = 16;
__device__ __forceinline__ void train_request(uint32_t queue, int slot, int layer)
{
    uint32_t n;
    asm volatile("atom.relaxed.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(n) : "r"(queue) : "memory");
    const uint32_t v = (n + 1) << 8 | static_cast<uint32_t>(slot) << 5 | static_cast<uint32_t>(layer);
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(queue + 4 + (n % TRAIN_QUEUE) * 4), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t train_next_request(uint32_t queue, uint32_t n)
{
    uint32_t v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(queue + 4 + (n % TRAIN_QUEUE) * 4) : "memory");
    return v;
}

// ---- one tile slot, per thread --------------------------------------------------------------------------------------------
template <class Spec, bool LOSS>
struct TrainSlot {
    static constexpr int WG = TrainLayout<Spec, LOSS>::WG;                           // warpgroups of a slot
    static constexpr int PIECES = (Spec::CIN[0] / 8 + WG - 1) / WG;                 // 8-channel pieces of the input this thread writes
    static constexpr int TARGETS = Spec::NUM_OUTPUTS <= 4 ? Spec::NUM_OUTPUTS : 0;  // prefetched by the warpgroup that takes the loss
    uint32_t row;          // shared address of this thread's row in buffer 0
    uint32_t tmem;         // base column, lane field of this warp included
    uint32_t bars;         // full: accumulator done; graded: weight gradient done
    int slot;              // its warps meet on named barrier 2 + slot at the end of a stage
    bool issuer;           // this warp issues the MMAs of the slot
    uint32_t smem, lead;
    uint32_t full, graded; // parities
    long long point;
    bool valid;
    uint32_t features[PIECES][4];
    float target[TARGETS > 0 ? TARGETS : 1];
    // pre-activations of this thread's channels, from a layer's forward to its backward stage (TrainLayout::preCol)
    static constexpr int PRE = TrainLayout<Spec, LOSS>::preBefore(Spec::NUM_LAYERS - 1);
    uint32_t pre[PRE > 0 ? PRE : 1];
};

// targets (or adjoints of the output) of a point, for the warpgroup that takes the loss
template <class Spec, bool LOSS>
__device__ __forceinline__ void train_fetch_target(const LaunchArgs& p, TrainSlot<Spec, LOSS>& sl, int wg, long long point)
{
    if constexpr (TrainSlot<Spec, LOSS>::TARGETS > 0) {
        if (wg == 0 && point < p.numel) {
#pragma unroll
            for (int c = 0; c < Spec::NUM_OUTPUTS; ++c)
                sl.target[c] = LOSS ? __ldg(p.target + point * p.tS0 + c * p.tS1) : __ldg(p.adjOutput + point * p.aoS0 + c * p.aoS1);
        }
    }
}
template <class Spec, bool LOSS, int K>
__device__ __forceinline__ void train_fetch(const LaunchArgs& p, TrainSlot<Spec, LOSS>& sl, int wg, long long point)
{
    constexpr int WG = TrainSlot<Spec, LOSS>::WG, CIN0 = Spec::CIN[0];
    if constexpr (K < TrainSlot<Spec, LOSS>::PIECES * WG) {
        if (wg == K % WG) {
            uint32_t (&v)[4] = sl.features[K / WG];
            if constexpr (K * 8 < CIN0) {
                if (point < p.numel) {
                    if constexpr (LOSS) {
                        fetch_piece<Spec, K * 8, K * 8 + 8>(p, point, v);
                    } else if (const long long at = point * CIN0 + K * 8; scratch_ok(p, at, 8, p.fwdTmpHalfs, STATUS_STASH)) {
                        const uint4 u = *reinterpret_cast<const uint4*>(p.fwdTmp + at);
                        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
                    } else {
                        v[0] = v[1] = v[2] = v[3] = 0u;
                    }
                }
                else v[0] = v[1] = v[2] = v[3] = 0u;
            }
        }
        train_fetch<Spec, LOSS, K + 1>(p, sl, wg, point);
    }
}
template <class Spec, bool LOSS, int K>
__device__ __forceinline__ void train_store_adjoint(const LaunchArgs& p, const TrainSlot<Spec, LOSS>& sl, int wg)
{
    if constexpr (K * 8 < Spec::CIN[0]) {
        if (wg == K % TrainSlot<Spec, LOSS>::WG) {
            float x[8];
            tmem_ld8(sl.tmem + K * 8, x);
            tmem_wait_ld();
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = h2_as_u32(__floats2half2_rn(x[2 * i], x[2 * i + 1]));
            if (sl.valid) store_piece<Spec, K * 8, K * 8 + 8>(p, sl.point, v);
        }
        train_store_adjoint<Spec, LOSS, K + 1>(p, sl, wg);
    }
}

// pre-activations of 8 accumulator columns: rounded to half, then the half bias is added
template <class Spec, int L>
__device__ __forceinline__ void train_pre(const float (&v)[8], const __half* bias, int col, __half2 (&pre)[4])
{
#pragma unroll
    for (int i = 0; i < 4; ++i) pre[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    if constexpr (Spec::BOFF[L] >= 0) {
        const uint4 b0 = *reinterpret_cast<const uint4*>(bias + TrainLayout<Spec>::dBefore(L) + col);
        const uint32_t w[4] = {b0.x, b0.y, b0.z, b0.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) pre[i] = __hadd2(pre[i], u32_as_h2(w[i]));
    }
}
// 8 channels at chunk CHUNK (8 channels each) + `col` / 8 of this thread's row of a buffer
template <int CHUNK = 0>
__device__ __forceinline__ void train_put(uint32_t rowAddr, int row, int col, const uint32_t (&w)[4])
{
    sts128(rowAddr + sw128_row_offset(row, CHUNK + col / 8), w[0], w[1], w[2], w[3]);
}

// One stage of a slot's tile (TrainLayout::lastStage). Every stage but the last is followed by the MMAs of the next one: the
// slot's warps meet, and one of them (the same one for all stages) issues.
template <class Spec, bool LOSS, int ST>
__device__ __forceinline__ void train_stage(const LaunchArgs& p, TrainSlot<Spec, LOSS>& sl, const __half* bias, int wg, int row, long long nextPoint,
                                            float& lossAcc, volatile int* abortFlag, bool& dead)
{
    using TR = TrainLayout<Spec, LOSS>;
    constexpr int NL = Spec::NUM_LAYERS, WG = TrainSlot<Spec, LOSS>::WG;
    if constexpr (ST == 0) {
        constexpr int CIN0 = Spec::CIN[0];
#pragma unroll
        for (int k = 0; k < TrainSlot<Spec, LOSS>::PIECES; ++k) {
            const int piece = wg + k * WG;
            if (piece * 8 < CIN0) {
                const uint32_t(&v)[4] = sl.features[k];
                sts128(sl.row + sw128_row_offset(row, piece), v[0], v[1], v[2], v[3]);
            }
        }
    } else {
        if constexpr (ST < TR::lastStage() || TR::FEATURE_ADJOINT) {
            train_wait(sl.bars, sl.full, abortFlag, dead, train_spin_limit(p));
            sl.full ^= 1u;
        }
        __syncwarp();   // tcgen05.ld is warp-collective
        tc_fence_after();
        if constexpr (ST < NL) {
            constexpr int L = ST - 1, COUT = Spec::COUT[L];
            using Act = typename Spec::template Act<L>;
#pragma unroll
            for (int k = 0; k < (COUT / 8 + WG - 1) / WG; ++k) {
                const int col = (wg + k * WG) * 8;
                if (col >= COUT) continue;
                float v[8];
                __half2 pre[4];
                uint32_t w[4];
                tmem_ld8(sl.tmem + col, v);
                tmem_wait_ld();
                train_pre<Spec, L>(v, bias, col, pre);
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = h2_as_u32(act_forward2<Act>(pre[i], col + 2 * i));
                train_put(sl.row + TR::bufOffset(L + 1), row, col, w);
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = h2_as_u32(pre[i]);
                if constexpr (TR::preCol(L) >= 0) {
                    tmem_st4(sl.tmem + TR::slotCols() + TR::preCol(L) + col / 2, w);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) sl.pre[TR::preBefore(L) + k * 4 + i] = w[i];
                }
            }
            if constexpr (TR::preCol(L) >= 0) tmem_wait_st();
        } else if constexpr (ST == NL) {
            constexpr int L = NL - 1, COUT = Spec::COUT[L];
            using Act = typename Spec::template Act<L>;
#pragma unroll
            for (int k = 0; k < (COUT / 8 + WG - 1) / WG; ++k) {
                const int col = (wg + k * WG) * 8;
                if (col >= COUT) continue;
                float v[8];
                __half2 pre[4];
                uint32_t w[4];
                tmem_ld8(sl.tmem + col, v);
                tmem_wait_ld();
                train_pre<Spec, L>(v, bias, col, pre);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float adj[2] = {0.f, 0.f};
                    if (col + 2 * i < Spec::NUM_OUTPUTS && sl.valid) {
                        const float2 out = __half22float2(act_forward2<Act>(pre[i], col + 2 * i));
                        const float o[2] = {out.x, out.y};
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int c = col + 2 * i + e;
                            if (c < Spec::NUM_OUTPUTS) {
                                float t;
                                if constexpr (TrainSlot<Spec, LOSS>::TARGETS > 0) t = sl.target[(2 * i + e) % TrainSlot<Spec, LOSS>::TARGETS];   // (here col == 0)
                                else t = LOSS ? __ldg(p.target + sl.point * p.tS0 + c * p.tS1) : __ldg(p.adjOutput + sl.point * p.aoS0 + c * p.aoS1);
                                if constexpr (LOSS) {
                                    const float d = o[e] - t;
                                    lossAcc += d * d;
                                    adj[e] = p.lossScale * d;
                                } else {
                                    adj[e] = t;
                                }
                            }
                        }
                    }
                    const __half2 d = act_adjoint2<Act>(pre[i], __floats2half2_rn(adj[0], adj[1]), col + 2 * i);
                    w[i] = sl.valid ? h2_as_u32(d) : 0u;
                }
                train_put<TR::LAST_CHUNK>(sl.row + TR::bufOffset(TR::LAST_BUFFER), row, col, w);
            }
        } else if constexpr (ST < TR::lastStage()) {
            // delta of layer L from the adjoint of layer L + 1's input
            constexpr int L = TR::stepLayer(ST), COUT = Spec::COUT[L];
            using Act = typename Spec::template Act<L>;
            // (all of them are computed under the gradient of layer L + 1, whose operand their buffer still is)
            uint32_t d[(COUT / 8 + WG - 1) / WG][4];
#pragma unroll
            for (int k = 0; k < (COUT / 8 + WG - 1) / WG; ++k) {
                const int col = (wg + k * WG) * 8;
                if (col >= COUT) continue;
                float x[8];
                tmem_ld8(sl.tmem + col, x);
                if constexpr (TR::preCol(L) >= 0) {
                    tmem_ld4(sl.tmem + TR::slotCols() + TR::preCol(L) + col / 2, d[k]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) d[k][i] = sl.pre[TR::preBefore(L) + k * 4 + i];
                }
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half2 y = act_adjoint2<Act>(u32_as_h2(d[k][i]), __floats2half2_rn(x[2 * i], x[2 * i + 1]), col + 2 * i);
                    d[k][i] = sl.valid ? h2_as_u32(y) : 0u;
                }
            }
            train_wait(sl.bars + 8, sl.graded, abortFlag, dead, train_spin_limit(p));
#pragma unroll
            for (int k = 0; k < (COUT / 8 + WG - 1) / WG; ++k) {
                const int col = (wg + k * WG) * 8;
                if (col < COUT) train_put(sl.row + TR::bufOffset(L + 1), row, col, d[k]);
            }
            sl.graded ^= 1u;
        } else {
            if constexpr (TR::FEATURE_ADJOINT) train_store_adjoint<Spec, LOSS, 0>(p, sl, wg);
            train_wait(sl.bars + 8, sl.graded, abortFlag, dead, train_spin_limit(p));   // buffer 0 is written next
            sl.graded ^= 1u;
        }
    }
    // the next tile of this slot: its features are fetched under the last stage (earlier they would be spilled, and waited for to do so)
    if constexpr (ST == TR::lastStage() - 1) {
        train_fetch<Spec, LOSS, 0>(p, sl, wg, nextPoint);
        train_fetch_target<Spec, LOSS>(p, sl, wg, nextPoint);
    }
    if constexpr (ST < TR::lastStage()) {
        using Issue = TrainIssue<Spec, LOSS>;
        tc_fence_before();
        fence_proxy_async();   // generic-proxy writes of the operands become visible to the tensor core
        __syncwarp();
        // All warps of the slot wait here, the others for an accumulator that is not computed before anyway. After a wait that gave up this
        // keeps them in step: no warp leaves a tile early, so each takes part in every meeting once. (If they only arrived, a warp that
        // waits for nothing any more would arrive for later stages too and leave the issuing warp alone in one of them for good. Layers
        // of 32 -> 64 -> 64 -> 1, 2^20 points / 48 -> 128 -> 64 -> 16 -> 4, 2^21 points: arriving only 94.7 / 564 us, meeting 94.7 / 576,
        // an arrival counter whose last warp issues 98.8 / 586.)
        asm volatile("bar.sync %0, %1;" ::"r"(2 + sl.slot), "n"(WG * 128) : "memory");
        if (sl.issuer) {
            tc_fence_after();
            if (!__any_sync(0xffffffffu, dead)) Issue::template critical<ST>(sl.lead, sl.smem, sl.smem + TR::slotStart() + sl.slot * TR::slotBytes(), sl.tmem & 0xffffu, sl.bars);
            if constexpr (Issue::template graded<ST>() >= 0)
                if ((threadIdx.x & 31) == 0) train_request(sl.smem + TR::queueStart(), sl.slot, Issue::template graded<ST>());
        }
    }
}

template <class Spec, bool LOSS, int ST>
__device__ __forceinline__ void train_stages(const LaunchArgs& p, TrainSlot<Spec, LOSS>& sl, const __half* bias, int wg, int row, long long nextPoint, float& lossAcc,
                                             volatile int* abortFlag, bool& dead)
{
    if constexpr (ST <= TrainLayout<Spec, LOSS>::lastStage()) {
        train_stage<Spec, LOSS, ST>(p, sl, bias, wg, row, nextPoint, lossAcc, abortFlag, dead);
        train_stages<Spec, LOSS, ST + 1>(p, sl, bias, wg, row, nextPoint, lossAcc, abortFlag, dead);
    }
}

// The weight-gradient warp: the MMAs of the layers' gradients in the order in which the deltas are completed. All slots add to the same
// accumulators, so one thread issues them; nobody waits for them before the slot's next stage has computed its results.
template <class Spec, bool LOSS>
__device__ __forceinline__ void train_gradients(const LaunchArgs& p, uint32_t lead, uint32_t smem, uint32_t tmemBase, uint32_t bars, uint32_t queue, int myTiles,
                                                volatile int* abortFlag, bool& dead)
{
    using TR = TrainLayout<Spec, LOSS>;
    uint32_t started = 0;
    const uint32_t requests = static_cast<uint32_t>(myTiles) * Spec::NUM_LAYERS;
    for (uint32_t n = 0; n < requests; ++n) {
        uint32_t v = 0, idle = 0;
        while (true) {
            v = __shfl_sync(0xffffffffu, train_next_request(queue, n), 0);
            if ((v >> 8) == ((n + 1) & 0xffffffu)) break;
            ++idle;
            if (idle > 4 * train_spin_limit(p) || ((idle & 1023u) == 1023u && __any_sync(0xffffffffu, *abortFlag != 0))) {
                *abortFlag = 1;
                dead = true;
                return;
            }
        }
        __syncwarp();   // (orders the elected lane's MMAs behind lane 0's acquire)
        tc_fence_after();
        // (opaque copies: the descriptors of all MMAs would be computed ahead of the loop and spilled)
        uint32_t base = smem, tmem = tmemBase;
        asm volatile("" : "+r"(base), "+r"(tmem));
        const int slot = static_cast<int>(v >> 5) & 7;
        TrainIssue<Spec, LOSS>::template weights<0>(lead, static_cast<int>(v & 31u), base, base + TR::slotStart() + slot * TR::slotBytes(), tmem + TR::SLOTS * TR::slotStride(),
                                                    started, bars + slot * 16);
    }
}

// weight-gradient accumulators of this CTA -> fp32 gradient vector
template <class Spec, bool LOSS, int L>
__device__ __forceinline__ void train_flush(const LaunchArgs& p, uint32_t wgTmem, int warpgroup, int lane)
{
    if constexpr (L < Spec::NUM_LAYERS) {
        using TR = TrainLayout<Spec, LOSS>;
        constexpr int CIN = Spec::CIN[L], COUT = Spec::COUT[L];
        constexpr bool OUT = TR::mIsOut(L), BIAS = TR::bias(L);
        constexpr int CHUNKS = TR::wgCols(L) / 16;
        float* gw = p.gradWeights + Spec::WOFF[L];
        float* gb = p.gradWeights + (BIAS ? Spec::BOFF[L] : 0);
        const bool vec = (reinterpret_cast<uintptr_t>(gw) & 15) == 0;   // (a caller's gradient vector may start anywhere)
        for (int c = warpgroup; c < CHUNKS; c += TR::WARPGROUPS) {
            const int col = c * 16;
            float v[16];
            tmem_ld16(wgTmem + TR::wgCol(L) + col, v);
            tmem_wait_ld();
            if constexpr (OUT) {            // lane = output, columns = inputs
                if (lane < COUT) {
                    if (col < CIN) {
#pragma unroll
                        for (int i = 0; i < 16; i += 4) {
                            float* at = gw + lane * CIN + col + i;
                            if (vec) red_add_v4_f32(at, v[i], v[i + 1], v[i + 2], v[i + 3]);
                            else {
#pragma unroll
                                for (int e = 0; e < 4; ++e) red_add_f32(at + e, v[i + e]);
                            }
                        }
                    } else if constexpr (BIAS) {
                        red_add_f32(gb + lane, v[0]);
                    }
                }
            } else {                        // lane = input, columns = outputs
                if (col < COUT) {
                    if (lane < CIN) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) red_add_f32(gw + (col + i) * CIN + lane, v[i]);
                    } else if (BIAS && CIN != 128 && lane == CIN) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) red_add_f32(gb + col + i, v[i]);
                    }
                } else if constexpr (BIAS) { // the bias MMA: lane = output
                    if (lane < COUT) red_add_f32(gb + lane, v[0]);
                }
            }
        }
        train_flush<Spec, LOSS, L + 1>(p, wgTmem, warpgroup, lane);
    }
}

// biases of all layers -> shared memory (whole CTA), or the channel of ones of every input buffer (one warpgroup)
template <class Spec, bool LOSS, int L, int SLOTS, bool ONES>
__device__ __forceinline__ void train_init(const LaunchArgs& p, uint32_t smemBase, __half* sBias, int row)
{
    if constexpr (L < Spec::NUM_LAYERS) {
        using TR = TrainLayout<Spec, LOSS>;
        constexpr int CIN = Spec::CIN[L], COUT = Spec::COUT[L];
        if constexpr (!ONES) {
            if constexpr (Spec::BOFF[L] >= 0)
                for (int i = threadIdx.x; i < COUT; i += TR::THREADS) sBias[TR::dBefore(L) + i] = p.weights[Spec::BOFF[L] + i];
        } else if constexpr (CIN % 64 != 0) {
#pragma unroll
            for (int s = 0; s < SLOTS; ++s)
                sts16(smemBase + TR::slotStart() + s * TR::slotBytes() + TR::bufOffset(L) + row * 128 + sw128_row_offset(row, CIN / 8), __ushort_as_half(0x3C00));
        }
        train_init<Spec, LOSS, L + 1, SLOTS, ONES>(p, smemBase, sBias, row);
    }
}

template <class Spec, bool LOSS, int SLOTS>
__global__ void __launch_bounds__(TrainLayout<Spec, LOSS>::THREADS, 1)
fused_train_tc_kernel(const __grid_constant__ LaunchArgs p, const __grid_constant__ TcWeightMaps<Spec> weightMaps)
{
    using TL = TcLayout<Spec>;
    using TR = TrainLayout<Spec, LOSS>;
    extern __shared__ unsigned char smemRaw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    __half* sBias = reinterpret_cast<__half*>(smem + TR::biasStart(SLOTS));
    // full and graded of every slot, the weight staging, the drain of every warp after a timeout; requests for weight gradients
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TR::barStart(SLOTS));
    uint64_t* weightBar = bars + 2 * SLOTS;
    uint64_t* drainBar = weightBar + 1;
    uint32_t* queue = reinterpret_cast<uint32_t*>(smem + TR::queueStart());   // number of requests so far, then the ring
    uint32_t* tmemSlot = queue + 1 + TRAIN_QUEUE;
    volatile int* abortFlag = reinterpret_cast<int*>(tmemSlot + 1);
    static_assert(8 * (2 * SLOTS + 1 + TR::THREADS / 32) + 4 * (TRAIN_QUEUE + 3) <= 384, "barrier area");
    static_assert(SLOTS <= 8 && Spec::NUM_LAYERS <= 32, "fields of a request");
    const uint32_t smemBase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, warpgroup = warp >> 2, row = threadIdx.x & 127;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(weightBar), 1);
        for (int w = 0; w < TR::THREADS / 32; ++w) mbar_init(smem_u32(drainBar + w), 1);
        for (int s = 0; s < 2 * SLOTS; ++s) mbar_init(smem_u32(bars + s), 1);     // one tcgen05.commit per phase
        for (int i = 0; i <= TRAIN_QUEUE; ++i) queue[i] = 0;
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(smem_u32(weightBar), TL::weightCopyBytes());
        tc_issue_weight_copies<Spec, 0>(weightMaps, smemBase, smem_u32(weightBar));
    }
    // Operand buffers and the block behind them start as zeros with a channel of ones: in the buffers the first padding
    // channel of the input (stages write the channels before it only), in the last block channel 0.
    for (int i = threadIdx.x; i < (TR::onesStart(SLOTS) + TRAIN_ONES - TR::slotStart()) / 16; i += TR::THREADS)
        reinterpret_cast<uint4*>(smem + TR::slotStart())[i] = make_uint4(0, 0, 0, 0);
    train_init<Spec, LOSS, 0, SLOTS, false>(p, smemBase, sBias, row);
    __syncthreads();
    if (warpgroup == 0) {
        if (row < TRAIN_ONES / 128) sts16(smemBase + TR::onesStart(SLOTS) + row * 128 + sw128_row_offset(row, 0), __ushort_as_half(0x3C00));
        train_init<Spec, LOSS, 0, SLOTS, true>(p, smemBase, sBias, row);
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(tmemSlot), 512);
        tmem_relinquish();
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmemBase = *tmemSlot;
    const uint32_t laneField = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t wgTmem = tmemBase + SLOTS * TR::slotStride();
    const int numTiles = static_cast<int>((p.numel + TC_TILE - 1) / TC_TILE);
    const int stride = gridDim.x;
    const int myTiles = static_cast<int>(blockIdx.x) < numTiles ? (numTiles - static_cast<int>(blockIdx.x) + stride - 1) / stride : 0;
    bool dead = false;
    const uint32_t lead = elect_one();
    train_wait(smem_u32(weightBar), 0, abortFlag, dead, train_spin_limit(p));
    __syncwarp();
    if (warpgroup == TR::WARPGROUPS) {
        const uint32_t smemU = __shfl_sync(0xffffffffu, smemBase, 0), tmemU = __shfl_sync(0xffffffffu, tmemBase, 0);
        if (!__any_sync(0xffffffffu, dead)) train_gradients<Spec, LOSS>(p, lead, smemU, tmemU, smemU + TR::barStart(SLOTS), smem_u32(queue), myTiles, abortFlag, dead);
    } else {
        // tile i of this CTA's sequence belongs to slot i % SLOTS
        const int slot = warpgroup / TrainSlot<Spec, LOSS>::WG, wg = warpgroup % TrainSlot<Spec, LOSS>::WG;
        auto pointOf = [&](int i) { return i < myTiles ? (blockIdx.x + static_cast<long long>(i) * stride) * TC_TILE + row : p.numel; };
        TrainSlot<Spec, LOSS> sl;
        sl.row = smemBase + TR::slotStart() + slot * TR::slotBytes() + row * 128;
        sl.tmem = tmemBase + slot * TR::slotStride() + laneField;
        sl.bars = smem_u32(bars + 2 * slot);
        sl.slot = slot;
        sl.issuer = wg == 0 && (warp & 3) == (slot & 3);   // (on different sub-partitions of the SM)
        sl.smem = smemBase;
        sl.lead = lead;
        sl.full = sl.graded = 0;
        sl.point = pointOf(slot);
        train_fetch<Spec, LOSS, 0>(p, sl, wg, sl.point);
        train_fetch_target<Spec, LOSS>(p, sl, wg, sl.point);
        float lossAcc = 0.f;
        for (int i = slot; i < myTiles; i += SLOTS) {
            sl.valid = sl.point < p.numel;
            const long long next = pointOf(i + SLOTS);
            train_stages<Spec, LOSS, 0>(p, sl, sBias, wg, row, next, lossAcc, abortFlag, dead);
            sl.point = next;
        }
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(TR::WARPGROUPS * 128) : "memory");   // every slot's weight gradients are in
        if (myTiles > 0 && !__any_sync(0xffffffffu, *abortFlag != 0)) {
            tc_fence_after();
            train_flush<Spec, LOSS, 0>(p, wgTmem + laneField, warpgroup, row);
            if (LOSS && p.lossSum != nullptr) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) lossAcc += __shfl_xor_sync(0xffffffffu, lossAcc, o);
                if ((threadIdx.x & 31) == 0 && lossAcc != 0.f) atomicAdd(p.lossSum, lossAcc);
            }
        }
    }
    __syncthreads();         // (nobody raises the flag any more)
    if (*abortFlag != 0) {   // gave up: let the copies of the weights and this warp's MMAs in flight finish
        mbar_wait(smem_u32(weightBar), 0);
        umma_commit_elected(lead, smem_u32(drainBar + warp));
        mbar_wait(smem_u32(drainBar + warp), 0);
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
struct TrainLaunchers {
    // a.numel == 0 asks whether the kernel exists for this network
    template <bool LOSS>
    static cudaError_t run(const LaunchArgs& a, cudaStream_t s)
    {
        using TR = TrainLayout<Spec, LOSS>;
        constexpr int smem = TR::bytes(TR::SLOTS);
        if (a.numel == 0) return cudaSuccess;
        static DeviceOnce once;
        auto k = fused_train_tc_kernel<Spec, LOSS, TR::SLOTS>;
        const cudaError_t e = once.run([&] { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
        if (e != cudaSuccess) return e;
        const TcWeightMaps<Spec>* maps = nullptr;
        const cudaError_t m = TcLaunchers<Spec>::weightMaps(a.weights, maps);
        if (m != cudaSuccess) return m;
        const long long tiles = (a.numel + TC_TILE - 1) / TC_TILE;
        const long long blocks = tiles < a.numSMs ? tiles : a.numSMs;
        k<<<static_cast<unsigned>(blocks), TR::THREADS, smem, s>>>(a, *maps);
        return cudaGetLastError();
    }
};

} // namespace kernel
} // namespace qmlp
