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
//   * One persistent CTA of 16 + 1 warps per SM. A tile is 128 points; the CTA has two tile slots of two warpgroups each, or
//     one of four where shared or tensor memory is short. The slots run independently: the MMAs of one run under the epilogue
//     of the other. Thread = (point row, column share): the warpgroups of a slot take the blocks of 8 columns of an
//     accumulator row in turn.
//   * Shared memory, all in the 128-byte swizzled layout (rows = points, 64 channels per block): the weights (staged by
//     TMA), per slot one buffer per layer input and one for the last delta. The delta of layer l - 1 overwrites the input
//     of layer l, which has the same shape and is dead once the weight gradient of layer l is done.
//   * Tensor memory: the accumulator of every layer of the slot stays until the backward pass has taken the activation
//     derivative from it, or is computed a second time where the columns are short (pre-activation = round to half, add the
//     half bias: taken from the fp32 accumulator instead of stored); one region for the adjoint of a layer input; and the
//     weight-gradient accumulators of all layers, which stay for the whole kernel and are added to the gradient vector
//     once per CTA.
//   * Weight gradients are MMAs over K = the 128 points of the tile: both operands are the tiles above read MN-major. Either
//     delta^T * input (M = outputs) or input^T * delta (M = inputs), whichever needs fewer columns. The bias gradient is one
//     more column (or row) of the same MMA: a channel of ones in the padding of the input's block, or a constant block of
//     ones behind it.
//   * The warp of a slot that finishes a stage last issues the MMAs that the next stage waits for (a warp of its own polling both
//     slots took several hundred clocks to notice: 606 -> 577 us in the second example below). The weight gradients of
//     all slots go to the same accumulators, so one warp issues all of them, in order; they only have to be done when the
//     next stage of the slot overwrites their operands.
// Measured, step of 32 -> 64 -> 64 -> 1 on 2^20 points: 94 (forward) + 123 (backward) + 127 us (weight gradients) -> 137 us;
// 48 -> 128 -> 64 -> 16 -> 4 on 2^21 points: 709 (with the gather) + 1022 (with the scatter) + 473 -> 577 us (655 with 16
// columns per block instead of 8: the narrow layers then leave a warpgroup idle). Bound by the latency of the stages: an MMA of
// K = 16 takes 48 clocks up to N = 64 from shared memory however few columns it has, and the round trip of a stage (arrival,
// issue, MMAs, commit, accumulator load) takes about a thousand clocks that one other slot cannot cover.
// Every wait is bounded; on a timeout the CTA runs through without waiting and the status word is set.
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

constexpr int TRAIN_WARPGROUPS = 4, TRAIN_THREADS = TRAIN_WARPGROUPS * 128 + 32;   // the last warp issues the weight gradients
constexpr int TRAIN_BLOCK = TC_TILE * 128;   // bytes of a block: 128 points x 64 channels

// LOSS: the training step's kernel (features from the planes, L2 loss against targets); else the backward pass of an earlier
// forward call (features from its stash, the adjoint of the output from the caller)
template <class Spec, bool LOSS = true>
struct TrainLayout {
    using TL = TcLayout<Spec>;
    static constexpr int NL = Spec::NUM_LAYERS;
    static constexpr bool FEATURE_ADJOINT = !LOSS || table_rows_per_point<Spec>() > 0;   // the adjoint of the features is wanted
    __host__ __device__ static constexpr int blocks(int channels) { return (channels + 63) / 64; }
    __host__ __device__ static constexpr bool bias(int l) { return Spec::BOFF[l] >= 0; }
    // buffer l < NL: input of layer l (later delta of layer l - 1); buffer NL: delta of the last layer. A narrow last delta
    // lies in the upper half of the block of a narrow last input.
    static constexpr bool SHARED_LAST = Spec::CIN[NL - 1] <= 16 && Spec::COUT[NL - 1] <= 32;
    __host__ __device__ static constexpr int bufOffset(int l)
    {
        int o = 0;
        for (int i = 0; i < l && i < NL; ++i) o += blocks(Spec::CIN[i]) * TRAIN_BLOCK;
        return o;   // (l == NL: behind the last input)
    }
    // byte offset of the delta of layer l in the slot (its first channel, row 0)
    __host__ __device__ static constexpr int deltaOffset(int l) { return l < NL - 1 ? bufOffset(l + 1) : (SHARED_LAST ? bufOffset(NL - 1) + 64 : bufOffset(NL)); }
    __host__ __device__ static constexpr int slotBytes() { return bufOffset(NL) + (SHARED_LAST ? 0 : blocks(Spec::COUT[NL - 1]) * TRAIN_BLOCK); }

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
    // Accumulator columns of a slot. Kept: every layer's accumulator stays until the backward pass has used it, then comes the
    // adjoint region, where the last layer starts as well (it is consumed before the first adjoint is computed). Recomputed:
    // all forward accumulators share 128 columns, and the backward pass runs in steps of 64 outputs, with the
    // recomputed accumulator in the first and the adjoint in the second half.
    __host__ __device__ static constexpr int keptCols()
    {
        int m = Spec::COUT[NL - 1];
        for (int i = FEATURE_ADJOINT ? 0 : 1; i < NL; ++i) m = Spec::CIN[i] > m ? Spec::CIN[i] : m;
        return dBefore(NL - 1) + m;
    }
    __host__ __device__ static constexpr int slotStart() { return TL::weightBytes(); }
    __host__ __device__ static constexpr int onesStart(int slots) { return slotStart() + slots * slotBytes(); }
    __host__ __device__ static constexpr int biasStart(int slots) { return onesStart(slots) + TRAIN_BLOCK; }
    __host__ __device__ static constexpr int barStart(int slots) { return biasStart(slots) + (dBefore(NL) * 2 + 127) / 128 * 128; }
    // barriers, arrival counters and flags (fused_train_tc_kernel)
    __host__ __device__ static constexpr int bytes(int slots) { return barStart(slots) + 384 + 1024; }
    __host__ __device__ static constexpr bool fits(int slots, bool recompute)
    {
        return slots * (recompute ? 128 : keptCols()) + wgCol(NL) <= 512 && bytes(slots) <= 227 * 1024;
    }
    // Two slots hide the MMA round trips (a few hundred clocks per stage) behind each other and are worth recomputing for.
    static constexpr int SLOTS = fits(2, false) || fits(2, true) ? 2 : 1;
    static constexpr bool RECOMPUTE = !fits(SLOTS, false);
    __host__ __device__ static constexpr int slotCols() { return RECOMPUTE ? 128 : keptCols(); }
    __host__ __device__ static constexpr int dCol(int l) { return RECOMPUTE ? 0 : dBefore(l); }
    __host__ __device__ static constexpr int adjCol() { return RECOMPUTE ? 64 : dBefore(NL - 1); }
    __host__ __device__ static constexpr int featureAdjCol() { return RECOMPUTE ? 0 : dBefore(NL - 1); }
    // Stages: 0 features, 1 .. NL - 1 activations, NL loss, then the backward steps of the layers NL - 2 .. 0 (their deltas; 64
    // outputs each when recomputing), then the adjoint of the features.
    __host__ __device__ static constexpr int steps(int l) { return RECOMPUTE ? blocks(Spec::COUT[l]) : 1; }
    __host__ __device__ static constexpr int lastStage()
    {
        int n = NL + 1;
        for (int i = 0; i < NL - 1; ++i) n += steps(i);
        return n;
    }
    __host__ __device__ static constexpr int stepLayer(int stage)   // layer whose delta stage `stage` computes (NL < stage < lastStage())
    {
        int s = NL + 1, l = NL - 2;
        while (s + steps(l) <= stage) { s += steps(l); --l; }
        return l;
    }
    __host__ __device__ static constexpr int stepIndex(int stage)
    {
        int s = NL + 1, l = NL - 2;
        while (s + steps(l) <= stage) { s += steps(l); --l; }
        return stage - s;
    }
    // (TcLayout: the encode pass exists for the same networks)
    __host__ __device__ static constexpr bool eligible() { return TL::eligible() && (fits(1, false) || fits(1, true)); }
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
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// without the suspension that a try_wait may take: for a warp that watches several barriers
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait. When one gives up it raises the CTA's abort flag; from then on nobody waits any more (`dead`), so that the
// CTA runs through to its end.
__device__ __forceinline__ void train_wait(uint32_t bar, uint32_t parity, volatile int* abortFlag, bool& dead)
{
    if (dead) return;
    for (uint32_t i = 0; i < TC_SPIN_LIMIT; ++i) {
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
template <class Spec, bool LOSS, int SLOTS>
struct TrainIssue {
    using TL = TcLayout<Spec>;
    using TR = TrainLayout<Spec, LOSS>;
    // outputs [FIRST, FIRST + N) of layer L = input * W^T, to column `dTmem`
    template <int L, int FIRST, int N>
    static __device__ __forceinline__ void forward(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t dTmem)
    {
        constexpr int CIN = Spec::CIN[L], COUT = Spec::COUT[L];
        const uint64_t a = umma_desc_sw128(slotSmem + TR::bufOffset(L)), b = umma_desc_sw128(smem + TL::wOffset(L) + FIRST * 128);
#pragma unroll
        for (int k = 0; k < CIN / 16; ++k)
            umma_f16_elected(lead, dTmem, a + (((k >> 2) * TRAIN_BLOCK + (k & 3) * 32) >> 4), b + (((k >> 2) * (COUT * 128) + (k & 3) * 32) >> 4),
                             umma_idesc_f16(TC_TILE, N), k > 0 ? 1u : 0u);
    }
    // adjoint of inputs [FIRST, FIRST + N) of layer L = delta * W, to column `dTmem`
    template <int L, int FIRST, int N>
    static __device__ __forceinline__ void adjoint(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t dTmem)
    {
        constexpr int COUT = Spec::COUT[L];
        const uint64_t a = umma_desc_sw128(slotSmem + TR::deltaOffset(L)), b = umma_desc_mn_sw128(smem + TL::wOffset(L) + FIRST / 64 * (COUT * 128), COUT * 128);
#pragma unroll
        for (int k = 0; k < COUT / 16; ++k)
            umma_f16_elected(lead, dTmem, a + (((k >> 2) * TRAIN_BLOCK + (k & 3) * 32) >> 4), b + ((k * 2048) >> 4), umma_idesc_f16(TC_TILE, N) | UMMA_B_MN,
                             k > 0 ? 1u : 0u);
    }
    // weight (and bias) gradient of layer L
    template <int L>
    static __device__ __forceinline__ void gradient(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t wgTmem, uint32_t accumulate)
    {
        constexpr int CIN = Spec::CIN[L];
        const uint32_t delta = slotSmem + TR::deltaOffset(L), input = slotSmem + TR::bufOffset(L), ones = smem + TR::onesStart(SLOTS);
        // M is always 128: the block after a 64-channel operand is whatever lies there (inside the CTA's shared memory), its rows
        // of the result are not read
        constexpr bool OUT = TR::mIsOut(L);
        const uint32_t inputLbo = CIN == 64 ? ones - input : TRAIN_BLOCK;
        const uint64_t m = OUT ? umma_desc_mn_sw128(delta, TRAIN_BLOCK) : umma_desc_mn_sw128(input, inputLbo);
        const uint64_t n = OUT ? umma_desc_mn_sw128(input, inputLbo) : umma_desc_mn_sw128(delta, TRAIN_BLOCK);
        constexpr int N = OUT ? CIN + (TR::bias(L) && CIN != 128 ? 16 : 0) : Spec::COUT[L];
#pragma unroll
        for (int k = 0; k < TC_TILE / 16; ++k)
            umma_f16_elected(lead, wgTmem + TR::wgCol(L), m + ((k * 2048) >> 4), n + ((k * 2048) >> 4), umma_idesc_f16(TC_TILE, N) | UMMA_A_MN | UMMA_B_MN,
                             k == 0 ? accumulate : 1u);
        if constexpr (TR::separateBias(L)) {
            const uint64_t d = umma_desc_mn_sw128(delta, TRAIN_BLOCK), o = umma_desc_mn_sw128(ones, TRAIN_BLOCK);
#pragma unroll
            for (int k = 0; k < TC_TILE / 16; ++k)
                umma_f16_elected(lead, wgTmem + TR::wgCol(L) + N, d + ((k * 2048) >> 4), o + ((k * 2048) >> 4),
                                 umma_idesc_f16(TC_TILE, 16) | UMMA_A_MN | UMMA_B_MN, k == 0 ? accumulate : 1u);
        }
    }
    // what the next stage of the slot waits for after stage ST
    template <int ST>
    static __device__ __forceinline__ void critical(uint32_t lead, uint32_t smem, uint32_t slotSmem, uint32_t slotTmem, uint32_t bars)
    {
        constexpr int NL = Spec::NUM_LAYERS, NEXT = ST + 1;
        if constexpr (ST < NL) {
            forward<ST, 0, Spec::COUT[ST]>(lead, smem, slotSmem, slotTmem + TR::dCol(ST));
            umma_commit_elected(lead, bars);
        } else if constexpr (NEXT < TR::lastStage()) {
            constexpr int L = TR::stepLayer(NEXT), FIRST = 64 * TR::stepIndex(NEXT), LEFT = Spec::COUT[L] - FIRST;
            constexpr int N = TR::RECOMPUTE && LEFT > 64 ? 64 : LEFT;
            if constexpr (TR::RECOMPUTE) forward<L, FIRST, N>(lead, smem, slotSmem, slotTmem);
            adjoint<L + 1, FIRST, N>(lead, smem, slotSmem, slotTmem + TR::adjCol());
            umma_commit_elected(lead, bars);
        } else if constexpr (TR::FEATURE_ADJOINT) {
            adjoint<0, 0, Spec::CIN[0]>(lead, smem, slotSmem, slotTmem + TR::featureAdjCol());
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
        else return TR::stepIndex(ST) == TR::steps(TR::stepLayer(ST)) - 1 ? TR::stepLayer(ST) : -1;
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

// ---- one tile slot, per thread --------------------------------------------------------------------------------------------
template <class Spec, bool LOSS>
struct TrainSlot {
    static constexpr int WG = TRAIN_WARPGROUPS / TrainLayout<Spec, LOSS>::SLOTS;          // warpgroups of a slot
    static constexpr int PIECES = (Spec::CIN[0] / 8 + WG - 1) / WG;                 // 8-channel pieces of the input this thread writes
    static constexpr int TARGETS = Spec::NUM_OUTPUTS <= 4 ? Spec::NUM_OUTPUTS : 0;  // prefetched by the warpgroup that takes the loss
    uint32_t row;          // shared address of this thread's row in buffer 0
    uint32_t tmem;         // base column, lane field of this warp included
    uint32_t bars;         // full: accumulator done; graded: weight gradient done; ready: a delta is complete
    uint32_t counter;      // arrivals of the slot's warps
    uint32_t smem, slotSmem, slotTmem, lead;   // what the MMAs of the slot are issued from
    uint32_t full, graded; // parities
    long long point;
    bool valid;
    uint32_t features[PIECES][4];
    float target[TARGETS > 0 ? TARGETS : 1];
};

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
            tmem_ld8(sl.tmem + TrainLayout<Spec, LOSS>::featureAdjCol() + K * 8, x);
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
// warps count their arrivals, and the last one issues.
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
        if constexpr (TrainSlot<Spec, LOSS>::TARGETS > 0) {
            if (wg == 0 && sl.valid) {
#pragma unroll
                for (int c = 0; c < Spec::NUM_OUTPUTS; ++c)
                    sl.target[c] = LOSS ? __ldg(p.target + sl.point * p.tS0 + c * p.tS1) : __ldg(p.adjOutput + sl.point * p.aoS0 + c * p.aoS1);
            }
        }
    } else {
        if constexpr (ST < TR::lastStage() || TR::FEATURE_ADJOINT) {
            train_wait(sl.bars, sl.full, abortFlag, dead);
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
                tmem_ld8(sl.tmem + TR::dCol(L) + col, v);
                tmem_wait_ld();
                train_pre<Spec, L>(v, bias, col, pre);
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = h2_as_u32(act_forward2<Act>(pre[i], col + 2 * i));
                train_put(sl.row + TR::bufOffset(L + 1), row, col, w);
            }
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
                tmem_ld8(sl.tmem + TR::dCol(L) + col, v);
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
                train_put<TR::SHARED_LAST ? 4 : 0>(sl.row + TR::bufOffset(TR::SHARED_LAST ? NL - 1 : NL), row, col, w);
            }
            // the next tile of this slot: its features are fetched under the backward pass
            train_fetch<Spec, LOSS, 0>(p, sl, wg, nextPoint);
        } else if constexpr (ST < TR::lastStage()) {
            // outputs [FIRST, FIRST + N) of the delta of layer L from the adjoint of layer L + 1's input
            constexpr int L = TR::stepLayer(ST), H = TR::stepIndex(ST), FIRST = 64 * H, LEFT = Spec::COUT[L] - FIRST,
                          N = TR::RECOMPUTE && LEFT > 64 ? 64 : LEFT;
            using Act = typename Spec::template Act<L>;
            bool graded = H > 0;
#pragma unroll
            for (int k = 0; k < (N / 8 + WG - 1) / WG; ++k) {
                const int col = (wg + k * WG) * 8;
                if (col >= N) continue;
                float v[8], x[8];
                __half2 pre[4];
                uint32_t w[4];
                tmem_ld8(sl.tmem + TR::dCol(L) + col, v);
                tmem_ld8(sl.tmem + TR::adjCol() + col, x);
                tmem_wait_ld();
                train_pre<Spec, L>(v, bias, FIRST + col, pre);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half2 d = act_adjoint2<Act>(pre[i], __floats2half2_rn(x[2 * i], x[2 * i + 1]), FIRST + col + 2 * i);
                    w[i] = sl.valid ? h2_as_u32(d) : 0u;
                }
                if (!graded) train_wait(sl.bars + 8, sl.graded, abortFlag, dead);   // the buffer still is an operand of layer L + 1's gradient
                graded = true;
                train_put(sl.row + TR::bufOffset(L + 1), row, FIRST + col, w);
            }
            if (!graded) train_wait(sl.bars + 8, sl.graded, abortFlag, dead);       // (no columns here: stay in step with the barrier)
            if constexpr (H == 0) sl.graded ^= 1u;
        } else {
            if constexpr (TR::FEATURE_ADJOINT) train_store_adjoint<Spec, LOSS, 0>(p, sl, wg);
            train_wait(sl.bars + 8, sl.graded, abortFlag, dead);   // buffer 0 is written next
            sl.graded ^= 1u;
        }
    }
    if constexpr (ST < TR::lastStage()) {
        using Issue = TrainIssue<Spec, LOSS, TR::SLOTS>;
        tc_fence_before();
        fence_proxy_async();   // generic-proxy writes of the operands become visible to the tensor core
        __syncwarp();
        uint32_t before = 0;
        if ((threadIdx.x & 31) == 0)
            asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(sl.counter) : "memory");
        before = __shfl_sync(0xffffffffu, before, 0);
        if ((before & (WG * 4 - 1)) == WG * 4 - 1) {
            tc_fence_after();
            if (!__any_sync(0xffffffffu, dead)) Issue::template critical<ST>(sl.lead, sl.smem, sl.slotSmem, sl.slotTmem, sl.bars);
            if constexpr (Issue::template graded<ST>() >= 0)
                if ((threadIdx.x & 31) == 0) mbar_arrive(sl.bars + 16);
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

// The weight-gradient warp: whenever a slot's delta is complete, the MMAs of that layer's gradient. All slots add to the same
// accumulators, so one thread issues them; nobody waits for them before the slot's next stage has computed its results.
template <class Spec, bool LOSS, int SLOTS>
__device__ __forceinline__ void train_gradients(uint32_t lead, uint32_t smem, uint32_t tmemBase, uint32_t bars, int myTiles, volatile int* abortFlag, bool& dead)
{
    using TR = TrainLayout<Spec, LOSS>;
    constexpr int NL = Spec::NUM_LAYERS;
    int layer[SLOTS], left[SLOTS], open = 0;
    uint32_t parity = 0, started = 0, idle = 0;
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        layer[j] = NL - 1;
        left[j] = myTiles > j ? (myTiles - j + SLOTS - 1) / SLOTS * NL : 0;
        open += left[j] > 0;
    }
    while (open > 0) {
        ++idle;
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            if (left[j] == 0 || !__all_sync(0xffffffffu, mbar_poll(bars + j * 24 + 16, (parity >> j) & 1u))) continue;
            tc_fence_after();
            // (opaque copies: the descriptors of all MMAs would be computed ahead of the loop and spilled)
            uint32_t base = smem, tmem = tmemBase;
            asm volatile("" : "+r"(base), "+r"(tmem));
            TrainIssue<Spec, LOSS, SLOTS>::template weights<0>(lead, layer[j], base, base + TR::slotStart() + j * TR::slotBytes(), tmem + SLOTS * TR::slotCols(), started,
                                                         bars + j * 24);
            parity ^= 1u << j;
            layer[j] = layer[j] == 0 ? NL - 1 : layer[j] - 1;
            if (--left[j] == 0) --open;
            idle = 0;
        }
        if (idle > 4 * TC_SPIN_LIMIT || ((idle & 1023u) == 1023u && __any_sync(0xffffffffu, *abortFlag != 0))) {
            *abortFlag = 1;
            dead = true;
            return;
        }
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
        for (int c = warpgroup; c < CHUNKS; c += TRAIN_WARPGROUPS) {
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
                for (int i = threadIdx.x; i < COUT; i += TRAIN_THREADS) sBias[TR::dBefore(L) + i] = p.weights[Spec::BOFF[L] + i];
        } else if constexpr (CIN % 64 != 0) {
#pragma unroll
            for (int s = 0; s < SLOTS; ++s)
                sts16(smemBase + TR::slotStart() + s * TR::slotBytes() + TR::bufOffset(L) + row * 128 + sw128_row_offset(row, CIN / 8), __ushort_as_half(0x3C00));
        }
        train_init<Spec, LOSS, L + 1, SLOTS, ONES>(p, smemBase, sBias, row);
    }
}

template <class Spec, bool LOSS, int SLOTS>
__global__ void __launch_bounds__(TRAIN_THREADS, 1)
fused_train_tc_kernel(const __grid_constant__ LaunchArgs p, const __grid_constant__ TcWeightMaps<Spec> weightMaps)
{
    using TL = TcLayout<Spec>;
    using TR = TrainLayout<Spec, LOSS>;
    extern __shared__ unsigned char smemRaw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    __half* sBias = reinterpret_cast<__half*>(smem + TR::biasStart(SLOTS));
    // full, graded and ready of every slot, the weight staging, the drain of every warp after a timeout; arrival counters
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TR::barStart(SLOTS));
    uint64_t* weightBar = bars + 3 * SLOTS;
    uint64_t* drainBar = weightBar + 1;
    uint32_t* counters = reinterpret_cast<uint32_t*>(drainBar + TRAIN_THREADS / 32);
    uint32_t* tmemSlot = counters + SLOTS;
    volatile int* abortFlag = reinterpret_cast<int*>(tmemSlot + 1);
    static_assert(8 * (3 * SLOTS + 1 + TRAIN_THREADS / 32) + 4 * (SLOTS + 2) <= 384, "barrier area");
    const uint32_t smemBase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, warpgroup = warp >> 2, row = threadIdx.x & 127;

    if (threadIdx.x == 0) {
        mbar_init(smem_u32(weightBar), 1);
        for (int w = 0; w < TRAIN_THREADS / 32; ++w) mbar_init(smem_u32(drainBar + w), 1);
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(smem_u32(bars + 3 * s), 1);                                // one tcgen05.commit per phase
            mbar_init(smem_u32(bars + 3 * s + 1), 1);
            mbar_init(smem_u32(bars + 3 * s + 2), 1);                            // the last warp of a stage that completes a delta
            counters[s] = 0;
        }
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(smem_u32(weightBar), TL::weightCopyBytes());
        tc_issue_weight_copies<Spec, 0>(weightMaps, smemBase, smem_u32(weightBar));
    }
    // Operand buffers and the block behind them start as zeros with a channel of ones: in the buffers the first padding
    // channel of the input (stages write the channels before it only), in the last block channel 0.
    for (int i = threadIdx.x; i < (TR::onesStart(SLOTS) + TRAIN_BLOCK - TR::slotStart()) / 16; i += TRAIN_THREADS)
        reinterpret_cast<uint4*>(smem + TR::slotStart())[i] = make_uint4(0, 0, 0, 0);
    train_init<Spec, LOSS, 0, SLOTS, false>(p, smemBase, sBias, row);
    __syncthreads();
    if (warpgroup == 0) {
        sts16(smemBase + TR::onesStart(SLOTS) + row * 128 + sw128_row_offset(row, 0), __ushort_as_half(0x3C00));
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
    const uint32_t wgTmem = tmemBase + SLOTS * TR::slotCols();
    const int numTiles = static_cast<int>((p.numel + TC_TILE - 1) / TC_TILE);
    const int stride = gridDim.x;
    const int myTiles = static_cast<int>(blockIdx.x) < numTiles ? (numTiles - static_cast<int>(blockIdx.x) + stride - 1) / stride : 0;
    bool dead = false;
    const uint32_t lead = elect_one();
    train_wait(smem_u32(weightBar), 0, abortFlag, dead);
    __syncwarp();
    if (warpgroup == TRAIN_WARPGROUPS) {
        const uint32_t smemU = __shfl_sync(0xffffffffu, smemBase, 0), tmemU = __shfl_sync(0xffffffffu, tmemBase, 0);
        if (!__any_sync(0xffffffffu, dead)) train_gradients<Spec, LOSS, SLOTS>(lead, smemU, tmemU, smemU + TR::barStart(SLOTS), myTiles, abortFlag, dead);
    } else {
        // tile i of this CTA's sequence belongs to slot i % SLOTS
        const int slot = warpgroup / TrainSlot<Spec, LOSS>::WG, wg = warpgroup % TrainSlot<Spec, LOSS>::WG;
        auto pointOf = [&](int i) { return i < myTiles ? (blockIdx.x + static_cast<long long>(i) * stride) * TC_TILE + row : p.numel; };
        TrainSlot<Spec, LOSS> sl;
        sl.row = smemBase + TR::slotStart() + slot * TR::slotBytes() + row * 128;
        sl.tmem = tmemBase + slot * TR::slotCols() + laneField;
        sl.bars = smem_u32(bars + 3 * slot);
        sl.counter = smem_u32(counters + slot);
        sl.smem = smemBase;
        sl.slotSmem = smemBase + TR::slotStart() + slot * TR::slotBytes();
        sl.slotTmem = tmemBase + slot * TR::slotCols();
        sl.lead = lead;
        sl.full = sl.graded = 0;
        sl.point = pointOf(slot);
        train_fetch<Spec, LOSS, 0>(p, sl, wg, sl.point);
        float lossAcc = 0.f;
        for (int i = slot; i < myTiles; i += SLOTS) {
            sl.valid = sl.point < p.numel;
            const long long next = pointOf(i + SLOTS);
            train_stages<Spec, LOSS, 0>(p, sl, sBias, wg, row, next, lossAcc, abortFlag, dead);
            sl.point = next;
        }
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(TRAIN_WARPGROUPS * 128) : "memory");   // every slot's weight gradients are in
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
    if (*abortFlag != 0) {   // gave up: let this warp's MMAs in flight finish
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
        k<<<static_cast<unsigned>(blocks), TRAIN_THREADS, smem, s>>>(a, *maps);
        return cudaGetLastError();
    }
};

} // namespace kernel
} // namespace qmlp
