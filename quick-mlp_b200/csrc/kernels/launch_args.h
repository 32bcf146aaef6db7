// Plain structs shared by the host library and the per-spec kernel instantiations.
// They replace the reference's __constant__ HashGridConfig marshalling
// (src_cpp/include/qmlp/kernels/encoding_hashgrid_config.cuh:23-38, src_cpp/src/encoding_hashgrid.cpp:204-243):
// the level table travels as a __grid_constant__ kernel parameter instead of a cuMemcpyHtoDAsync per launch.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace qmlp {
namespace kernel {

constexpr int MAX_GRID_LEVELS = 32;
constexpr int MAX_GRIDS = 4;
// Grid slots of the launch arguments as this translation unit sees them. The generated source of a network defines how many
// it uses, so that a launch copies no more: the slots (and what goes with levels) are the last members, and an instantiation reads a prefix of what the
// library passes.
#ifdef QMLP_GRIDS
constexpr int GRID_SLOTS = QMLP_GRIDS;
#else
constexpr int GRID_SLOTS = MAX_GRIDS;
#endif
constexpr int MAX_GRID_DIMS = 6;

struct GridLevelP {
    unsigned int offset;       // element offset of the level inside the table (memoryOffset)
    int resolution;            // per-side resolution
    unsigned int hashGridSize; // rows if hashed (a power of two)
    int hashed;                // 1: hashed lookup, 0: dense lookup
};

struct GridP {
    const void* table; // fp32 (reference layout) or fp16 copy: [level0 rows*F | level1 ...]
    float* grad;       // fp32 gradient table, same layout (may be null)
    float boxMin[MAX_GRID_DIMS];
    float boxInvSize[MAX_GRID_DIMS];
    float boxSize[MAX_GRID_DIMS];
    float stepsize;    // line integration only: world-space step along the ray
    int tableIsHalf;
    int vecOk; // table and grad pointers are aligned for whole-row vector access
    unsigned long long tableCount; // elements of the table (and of its gradient): what QMLP_BOUNDS_CHECK builds check rows against
    int* status;                   // the library's status word (QMLP_BOUNDS_CHECK builds report through it), may be null
    GridLevelP levels[MAX_GRID_LEVELS];
};

// Bits of the library's device status word (qmlp_device_status). Bit 0 is set by a kernel that gave up on a bounded wait;
// the others only by instantiations compiled with QMLP_BOUNDS_CHECK, which test every table row, stash offset, plane
// offset and record or copy of a grid cell against the size the host declared, skip an access that would leave it and report here instead of faulting.
constexpr int STATUS_WAIT_TIMEOUT = 1, STATUS_TABLE_ROW = 2, STATUS_STASH = 4, STATUS_PLANES = 8, STATUS_CELL = 16;
#ifdef QMLP_BOUNDS_CHECK
constexpr bool BOUNDS_CHECK = true;
#else
constexpr bool BOUNDS_CHECK = false;
#endif

// bits of LaunchArgs::flags for the backward kernel (AdjointMode of the reference,
// src_cpp/include/qmlp/fused_network.h:22-34)
constexpr int FLAG_GRAD_INPUT = 1;
constexpr int FLAG_GRAD_WEIGHTS = 2;
constexpr int FLAG_GRAD_ENCODINGS = 4;
// the backward kernel only writes the adjoint of the grid features to level-major planes (LaunchArgs::planes); the
// table gradients are scattered from there by KERNEL_SCATTER_PLANES. Only with FLAG_GRAD_ENCODINGS and without
// FLAG_GRAD_INPUT.
constexpr int FLAG_SPLIT_SCATTER = 8;
// KERNEL_ENCODE_PLANES for a pass without gradients: see grid_pair_forward
constexpr int FLAG_HALF_SUMS = 16;
// KERNEL_ENCODE_PLANES, KERNEL_ENCODING_FORWARD: fill the copies by cell (CellTables) first
constexpr int FLAG_FILL_CELLS = 32;

// Copies of small grid levels by cell: the rows of a cell's 2^D corners side by side, so that a point fetches one piece of memory
// per level instead of 2^(D-1) pairs of rows (kernels/grid.cuh, GridCellRows). Filled from the tables by every call that
// uses them.
struct CellTables {
    unsigned char* base;                    // 256-byte aligned (null: none)
    long long bytes;                        // of all copies (QMLP_BOUNDS_CHECK builds)
    unsigned int offset[MAX_GRID_LEVELS];   // first byte of a level's cells / 256, + 1; levels counted over all grids of the network; 0: no copy
};

// Copies of the gradients of small grid levels. Reductions to one 128-byte line execute one after the other in its L2 slice
// (about nine clocks each): a level of a few lines that a large batch keeps hitting holds the whole kernel up. Such
// levels are scattered into several copies, picked by the CTA, which are added up afterwards.
struct GradReplicas {
    float* base;                            // copies of all such levels, level by level (null: none)
    long long total;                        // elements
    long long capacity;                     // the same, for QMLP_BOUNDS_CHECK builds (the size the host declares)
    unsigned int offset[MAX_GRID_LEVELS];        // first element of a level's copies; levels counted over all grids of the network
    unsigned char log2Copies[MAX_GRID_LEVELS];   // 0: the level has no copies
    unsigned char byCell[MAX_GRID_LEVELS];       // 1 + log2 of the copies of a level whose gradient is added up by cell first (GridCellUnits); else 0
};

struct LevelArgs {
    GradReplicas replicas;   // KERNEL_ENCODING_ADJOINT, KERNEL_SCATTER_PLANES
    CellTables cells;        // KERNEL_ENCODE_PLANES, KERNEL_ENCODING_FORWARD
};

struct LaunchArgs {
    long long numel;
    const float* input;     long long inS0, inS1;
    float* output;          long long outS0, outS1;
    const float* adjOutput; long long aoS0, aoS1;
    float* adjInput;        long long aiS0, aiS1;
    const float* target;    long long tS0, tS1;   // fused L2 loss (training step)
    float lossScale;                               // 2 / (global points * channels)
    float* lossSum;                                // += sum (out-target)^2, may be null
    const __half* weights;                         // flat fp16 parameter vector
    float* gradWeights;                            // flat fp32 gradient vector
    __half* fwdTmp;                                // stash: encoded input + pre-activations per layer
    __half* adjTmp;                                // adjoint stash: delta per layer
    int flags;
    int numSMs;
    int numGrids;
    int forcePath;                                 // 0: best path for spec and batch, 1: mma.sync kernels only, 3: tcgen05 whenever instantiated
    int* status;                                   // device word set to 1 when a kernel gave up on a bounded wait
    __half* planes;                                // encoded features (or their adjoints) of a chunk of points, one plane per grid level
    long long planeStride;                         // points per plane (capacity of the chunk buffer)
    long long fwdTmpHalfs, adjTmpHalfs, planeHalfs; // sizes of the three scratch buffers in halfs (QMLP_BOUNDS_CHECK builds; 0: unknown)
    unsigned int spinLimit;                        // polls before a wait of the training kernel gives up (QMLP_BOUNDS_CHECK builds)
    // spatially binned training step (kernels/sorted_scatter.cuh): KERNEL_SORT_POINTS copies the points (and targets)
    // into Morton-bin order; the kernels after it read the sorted copies through `input` / `target`
    unsigned int* binCounts;                       // points per bin (sort_bin_count() entries), zeroed by the launcher
    unsigned int* binStart;                        // first sorted point of every bin, sort_bin_count() + 1 entries
    unsigned int* binCursor;                       // running insert position per bin
    float* sortedInput;                            // (numel, NUM_INPUTS) row-major
    float* sortedTarget;                           // (numel, NUM_OUTPUTS) row-major, may be null
    int scatterLevelBegin, scatterLevelEnd;        // KERNEL_SCATTER_PLANES: grid levels (counted over all grids) to scatter; 0, 0 = all
    int runAggregation;                            // 0: every point of every level scatters straight to the gradient table
    LevelArgs level[GRID_SLOTS > 0 ? 1 : 0];       // (a network without grids carries none)
    GridP grids[GRID_SLOTS];                       // the last member (GRID_SLOTS)
};

// Bins of the point sort: a regular grid of 2^sort_bin_bits(D) cells per dimension over the bounding box of the first
// grid encoding, numbered in Morton order (bit b of dimension d at bit b * D + d of the key).
__host__ __device__ constexpr int sort_bin_bits(int dims)
{
    return dims <= 1 ? 16 : dims == 2 ? 9 : dims == 3 ? 6 : dims == 4 ? 4 : 3;
}
__host__ __device__ constexpr int sort_bin_count(int dims) { return 1 << (sort_bin_bits(dims) * dims); }

// kernels a network instantiation exports through qmlp_spec_launch
enum KernelId {
    KERNEL_INFERENCE = 0,
    KERNEL_FORWARD = 1,       // forward with stash
    KERNEL_FORWARD_LOSS = 2,  // forward with stash, writes dLoss/dOut of the L2 loss instead of the output
    KERNEL_BACKWARD = 3,      // flags select the variant
    KERNEL_WGRAD = 4,
    KERNEL_ENCODING_FORWARD = 5,
    KERNEL_ENCODING_ADJOINT = 6,
    KERNEL_ACTIVATION_FORWARD = 7,
    KERNEL_ACTIVATION_ADJOINT = 8,
    KERNEL_ENCODE_PLANES = 9,      // encodings of a chunk of points -> level-major feature planes
    KERNEL_INFERENCE_PLANES = 10,  // layer chain reading the feature planes instead of running the encodings
    KERNEL_SCATTER_PLANES = 11,    // adjoint feature planes -> grid table gradients, one grid level at a time
    KERNEL_FORWARD_LOSS_PLANES = 12, // KERNEL_FORWARD_LOSS with layer 0 fed from the planes of KERNEL_ENCODE_PLANES
    KERNEL_SORT_POINTS = 13,         // points (and targets) -> Morton-bin order: count, scan, reorder
    KERNEL_TRAIN = 14,               // layers of a training step on the planes: forward, loss, backward, weight gradients; adjoints back to the planes
    KERNEL_FORWARD_FEATURES = 16,    // forward that stashes the encoded input only
    KERNEL_BACKWARD_FEATURES = 17,   // its backward pass: layers computed again, weight gradients, adjoints to the planes / the input
    KERNEL_SCATTER_SORTED = 15       // KERNEL_SCATTER_PLANES for sorted points: coarse levels summed in shared memory first
};

// arguments of the stand-alone activation kernels
struct ActivationArgs {
    long long rows, cols;
    const __half* input;     long long inS0, inS1;
    const __half* adjOutput; long long aoS0, aoS1;
    __half* output;          long long outS0, outS1; // forward: z; adjoint: adjx
};

} // namespace kernel
} // namespace qmlp

// entry points every instantiation exports
extern "C" {
typedef int (*qmlp_spec_launch_fn)(int kernel, const void* args, cudaStream_t stream, int* launches);
typedef int (*qmlp_spec_abi_fn)(void);
}
#define QMLP_SPEC_ABI_VERSION 15
