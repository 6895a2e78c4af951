// Pieces shared by the SchNet kernels (schnet.cu: E, F and W; schnet_tangent.cu: the
// parameter gradient of a force and virial loss): sizes, the packed parameter block and the
// workspace layouts, the activations, BF16 feature rows, the per-CTA tensor-core context,
// the Gaussian basis, and the feature lanes that gather and scatter rows.

#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "umma.cuh"

namespace nd {
namespace {

constexpr int kFeatures = 64;
constexpr int kHidden = 32;      // the readout's hidden layer, features / 2
constexpr int kTile = 128;       // rows per tensor-core tile = threads per CTA
constexpr int kImagesPerBlock = 10;
constexpr float kLn2 = 0.693147180559945309f;

// Status bits of the SchNet status word.
constexpr int kBadPair = 1;       // a pair index outside [0, N)
constexpr int kProductLost = 16;  // a tensor-core product did not complete in time

// Weight images of one block, in this order. The two transposes of the filter layers are part of the
// block's layout only: the reverse passes read the layers' own images the other way.
enum Image : int
{
    kB1 = 0,   // filter1.weight [64 out][K in, zero-padded to 64]
    kB2 = 1,   // filter2.weight [out][in]
    kB2T = 2,  // its transpose
    kB1T = 3,  // filter1.weight^T [K, zero-padded to 64][64]
    kA = 4,    // atoms.weight
    kAT = 5,
    kD1 = 6,   // update1.weight
    kD1T = 7,
    kD2 = 8,   // update2.weight
    kD2T = 9,
};

// Byte layout of the packed parameter block (nd_schnet_weight_bytes).
struct WeightLayout
{
    std::int64_t vectors;  // per block: b1, b2, d1, d2 (64 floats each)
    std::int64_t readout;  // R1 [32][64], e1 [32], R2 [32], e2 (padded to 32)
    std::int64_t tables;   // embedding [T][64], v0 = embedding A0^T [T][64]
    std::int64_t total;

    __host__ __device__ WeightLayout(int blocks, int types)
    {
        vectors = static_cast<std::int64_t>(blocks) * kImagesPerBlock * umma::kImageBytes;
        readout = vectors + static_cast<std::int64_t>(blocks) * 4 * kFeatures * 4;
        tables = readout + (kHidden * kFeatures + 3 * kHidden) * 4;
        total = tables + 2 * static_cast<std::int64_t>(types) * kFeatures * 4;
    }
};

__host__ __device__ inline std::int64_t align256(std::int64_t bytes)
{
    return (bytes + 255) / 256 * 256;
}

constexpr int kVirialSlots = 1024;  // per-CTA virial partials of the last reverse pass

// Byte layout of the workspace (nd_schnet_workspace_bytes).
struct Workspace
{
    std::int64_t counters, block_counts, block_offsets, pairs, geometry, x, v, h, m, grad,
        grad_m, grad_v, dedr, energy, virial, total;

    Workspace(std::int64_t atoms, std::int64_t columns, int blocks)
    {
        const std::int64_t row = atoms * kFeatures * 4;
        const std::int64_t tiles = (atoms + kTile - 1) / kTile;
        const std::int64_t column_blocks = (columns + kThreads - 1) / kThreads;
        counters = 0;
        block_counts = 256;
        block_offsets = block_counts + align256(column_blocks * 4);
        pairs = block_offsets + align256(column_blocks * 4);
        geometry = pairs + align256(columns * 8);
        x = geometry + align256(columns * 16);
        v = x + align256(row);
        h = v + blocks * align256(row);
        m = h + blocks * align256(row);  // one message buffer per block (the tangent pass reuses them)
        grad = m + blocks * align256(row);
        grad_m = grad + align256(row);
        grad_v = grad_m + align256(row);
        dedr = grad_v + align256(row);
        energy = dedr + align256(columns * 4);
        virial = energy + align256(tiles * 8);
        total = virial + align256(kVirialSlots * 9 * 8);
    }
};

constexpr float kLog2E = 1.44269504088896340736f;

// The hardware exponential and logarithm of base two, denormals flushed (one instruction each;
// without the flush the compiler adds scaling on both sides).
__device__ __forceinline__ float exp2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float log2_approx(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ln(1 + e^x) - ln 2 and its derivative, in FP32 with the hardware exp and log; the results
// feed BF16 operands. e^-|x| underflows to zero where its logarithm term is below an ulp.
__device__ __forceinline__ float softplus_shifted(float x)
{
    const float log2 = log2_approx(1.0f + exp2_approx(-fabsf(x) * kLog2E));
    return fmaxf(x, 0.0f) + log2 * kLn2 - kLn2;
}

// The Gaussian exp(-u^2 / 2). As an operand of the tensor cores it keeps denormal results: their
// sums can lose the last bit to a product that lies below it. Where FP32 arithmetic weights it, a
// value below the smallest normal number changes nothing and is zero (three operations fewer).
__device__ __forceinline__ float gaussian(float u) { return __expf(-0.5f * u * u); }

__device__ __forceinline__ float gaussian_flushed(float u)
{
    return exp2_approx(-0.5f * u * u * kLog2E);
}

// 1 / (1 + e^-x) = (1 + tanh(x / 2)) / 2, with the hardware tanh (one special-function op).
__device__ __forceinline__ float sigmoid(float x)
{
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
    return fmaf(0.5f, t, 0.5f);
}

__device__ __forceinline__ std::uint32_t pack2(float lo, float hi)
{
    __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<std::uint32_t*>(&pair);
}

// One weight image of a CTA: where it goes in shared memory and where it comes from.
struct ImageCopy
{
    unsigned char* to;
    const unsigned char* from;
};

// The per-CTA tensor-core context: tensor memory, the completion barrier and its phase, and the
// weight images, which copies of the bulk engine bring in behind whatever precedes the first
// product.
struct Cores
{
    std::uint64_t* barrier;  // [3]: products; the slot; the images' copies
    std::uint32_t* slot;
    std::uint32_t tmem;  // this warp's lanes, column 0
    unsigned phase;
    bool images_pending;  // thread 0: the first product waits for the images

    template <int kImages>
    __device__ void open(std::uint64_t* barrier_, std::uint32_t columns, int* counters_,
                         int stage_, const ImageCopy (&images)[kImages])
    {
        barrier = barrier_;
        slot = reinterpret_cast<std::uint32_t*>(barrier + 1);
        phase = 0;
        counters = counters_;
        stage = stage_;
        tile_index = -1;
        images_pending = true;
        if (threadIdx.x == 0)
        {
            umma::barrier_init(barrier);
            umma::barrier_init(barrier + 2);
            umma::expect_bytes(barrier + 2, kImages * umma::kImageBytes);
#pragma unroll
            for (int k = 0; k < kImages; ++k)
            {
                umma::bulk_load(images[k].to, images[k].from, umma::kImageBytes, barrier + 2);
            }
        }
        if (threadIdx.x < 32)
        {
            umma::allocate(slot, columns);
        }
        umma::fence_before_sync();
        __syncthreads();
        umma::fence_after_sync();
        tmem = *slot + ((32u * (threadIdx.x / 32 % 4)) << 16);
    }

    int* counters;  // [4]: pairs, status bits, first stage that gave up, its tile
    int stage;      // the kernel's stage code, for the diagnostics
    int tile_index; // the tile in work, for the diagnostics

    // D[column offset] = tile * image^T, after every thread wrote its row of the tile; waits
    // for the product. False (on every thread) when it did not complete in time; then the
    // status bit is set and the first stage and tile that gave up are recorded.
    __device__ bool run(std::uint32_t column, const unsigned char* tile, const unsigned char* image,
                        int step)
    {
        return run2(column, tile, image, 0, nullptr, nullptr, step);
    }

    // As run, with a second product D[column2] = tile2 * image2^T (when tile2 is not null)
    // issued behind the first and completing on the same commit.
    __device__ bool run2(std::uint32_t column, const unsigned char* tile, const unsigned char* image,
                         std::uint32_t column2, const unsigned char* tile2,
                         const unsigned char* image2, int step)
    {
        return issue(
            [&] {
                umma::product(*slot + column, umma::smem_address(tile), umma::smem_address(image));
                if (tile2 != nullptr)
                {
                    umma::product(*slot + column2, umma::smem_address(tile2),
                                  umma::smem_address(image2));
                }
            },
            step);
    }

    // Issues products from one thread, after every thread's operand writes, and waits for them.
    template <typename Products>
    __device__ __forceinline__ bool issue(Products products, int step)
    {
        begin(products);
        return finish(step);
    }

    template <typename Products>
    __device__ __forceinline__ void begin(Products products)
    {
        umma::fence_operands();
        umma::fence_before_sync();
        __syncthreads();
        if (threadIdx.x == 0)
        {
            umma::fence_after_sync();
            if (images_pending && !umma::barrier_wait(barrier + 2, 0))
            {
                atomicOr(counters + 1, kProductLost);
            }
            images_pending = false;
            products();
            umma::commit(barrier);
        }
    }

    // Waits for the products begun last.
    __device__ __forceinline__ bool finish(int step)
    {
        const bool done = umma::barrier_wait(barrier, phase);
        phase ^= 1u;
        const bool lost = __syncthreads_or(!done);
        umma::fence_after_sync();
        if (lost && threadIdx.x == 0)
        {
            atomicOr(counters + 1, kProductLost);
            if (atomicCAS(counters + 2, 0, 16 * stage + step) == 0)
            {
                counters[3] = tile_index;
            }
        }
        return !lost;
    }

    __device__ void close(std::uint32_t columns)
    {
        if (threadIdx.x == 0 && images_pending)
        {
            umma::barrier_wait(barrier + 2, 0);  // no product ran: the copies may be in flight
        }
        umma::fence_before_sync();
        __syncthreads();
        if (threadIdx.x < 32)
        {
            umma::fence_after_sync();
            umma::deallocate(*slot, columns);
        }
    }
};

// Gaussians g_k(r) = exp(-(r / D - k)^2 / 2) into this thread's row: every k of a word of eight
// that starts below K (the weight image is zero in columns K and up), zero above.
template <int kChunk = 128, int kGroup = 1024>
__device__ __forceinline__ void store_basis(unsigned char* tile, float r_over_width, int gaussians)
{
#pragma unroll
    for (int c = 0; c < 8; ++c)
    {
        float values[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (8 * c < gaussians)
        {
#pragma unroll
            for (int e = 0; e < 8; ++e)
            {
                values[e] = gaussian(r_over_width - static_cast<float>(8 * c + e));
            }
        }
        umma::store8<kChunk, kGroup>(tile, threadIdx.x, c, values);
    }
}

// Feature lanes. The feature rows that the pair kernels gather (v = x A^T and Gm) are kept in BF16,
// 128 bytes a row. A tile's products leave one pair per thread, but the gathers and scatters of
// feature rows (128 or 256 bytes each) want a row per few lanes: a thread per row touches 32
// lines per instruction, and those accesses, not the arithmetic, bound the pair kernels (75 %
// of the load/store unit's wavefronts). So the half's 32 columns of a pair's FP32 filter go
// through shared memory (stage4: 16 KB, chunks swizzled by row), and eight lanes take a
// row of it, four features each, four rows of the warp's 32 at a time: a gathered half row is
// one 64-byte segment, a scattered one a whole 128-byte line. A lane meets rows 8 group + i,
// i = 0 .. 7, and leaves the first atoms' side in the stage, where add_runs sums it along the
// runs, one atomic per run, warp and column.
constexpr int kLaneRows = 8;  // rows a lane meets per half tile

struct FeatureLane
{
    int group;   // 0 .. 3
    int lane;    // 0 .. 7: features 4 lane .. 4 lane + 3 of the half
    int warp_row;

    __device__ FeatureLane()
        : group((threadIdx.x & 31) >> 3), lane(threadIdx.x & 7), warp_row(threadIdx.x & ~31u)
    {
    }

    __device__ int row(int i) const { return warp_row + kLaneRows * group + i; }

    // This lane's word of a BF16 feature row's half, and of an FP32 one's.
    __device__ std::int64_t word(int atom, int half) const
    {
        return 16 * static_cast<std::int64_t>(atom) + 8 * half + lane;
    }
};

// Four features of a staged half row.
__device__ __forceinline__ float4 staged4(const float* stage, int row, int lane)
{
    return reinterpret_cast<const float4*>(stage)[row * 8 + (lane ^ (row & 7))];
}

__device__ __forceinline__ float4 widen4(const uint2& word)
{
    return make_float4(__uint_as_float(word.x << 16), __uint_as_float(word.x & 0xFFFF0000u),
                       __uint_as_float(word.y << 16), __uint_as_float(word.y & 0xFFFF0000u));
}

__device__ __forceinline__ float4 operator*(const float4& a, const float4& b)
{
    return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
}

__device__ __forceinline__ float4 operator*(const float4& a, float b)
{
    return make_float4(a.x * b, a.y * b, a.z * b, a.w * b);
}

// a b + c, rounded once: which product of a sum of two is rounded by itself is written out, since
// a compiler chooses differently from one kernel to the next.
__device__ __forceinline__ float4 fma4(const float4& a, const float4& b, const float4& c)
{
    return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z),
                       fmaf(a.w, b.w, c.w));
}

// Replaces four features of a staged half row.
__device__ __forceinline__ void restage4(float* stage, int row, int lane, float4 value)
{
    reinterpret_cast<float4*>(stage)[row * 8 + (lane ^ (row & 7))] = value;
}

// First-atom sums of a warp's 32 staged half rows from `begin` on, a lane per column: each run of
// one first atom (`first`; -1: dead rows) is summed row by row from zero and added once, to
// `target` (this lane's column of atom 0's row) moved to the run's atom. The order is part of the
// result: the sums feed BF16 operands, where an FP32 sum's last bit can turn a rounding. Sums
// kept in the feature lanes' registers, their row groups joined by shuffles, cost no pass through
// shared memory (32,768 beads: forward 129 us, reverse 242, the E/F/W call 1,287) but add the rows
// in another order; with this pass 157, 300 and 1,510. An atomic per column is faster here than
// one per four columns after shuffles (reverse 300 and 320 us).
__device__ __forceinline__ void add_runs(const float* stage, const int* first, int begin,
                                         float* target)
{
    constexpr int kAhead = 8;  // rows read before any is added
    const int lane = threadIdx.x & 31;
    const int atom = first[begin + lane];
    const int after = __shfl_down_sync(kFullMask, atom, 1);
    const unsigned ends = __ballot_sync(kFullMask, lane == 31 || after != atom);
    const float* rows = stage + begin * 32;
    float sum = 0.0f;
    auto add = [&](int r) {
        const int run = first[begin + r];
        if (run >= 0)
        {
            atomicAdd(target + static_cast<std::int64_t>(run) * kFeatures, sum);
        }
        sum = 0.0f;
    };
#pragma unroll 1
    for (int r0 = 0; r0 < 32; r0 += kAhead)
    {
        float part[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
        {
            part[k] = rows[(r0 + k) * 32 + (lane ^ (4 * k))];  // chunk (lane / 4) ^ (row % 8)
        }
        const unsigned inside = ends >> r0 & ((1u << kAhead) - 1u);
        if (inside == 0)
        {
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
            {
                sum += part[k];
            }
            continue;
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
        {
            sum += part[k];
            if (inside & (1u << k))
            {
                add(r0 + k);
            }
        }
    }
}

// Stages float4 `q` (columns 4 q .. 4 q + 3 of the half) of this thread's row.
__device__ __forceinline__ void stage4(float* stage, int q, float4 value)
{
    reinterpret_cast<float4*>(stage)[threadIdx.x * 8 + (q ^ (threadIdx.x & 7))] = value;
}

// A half (32 columns) of this thread's FP32 row, (value + bias) * scale, into the stage.
__device__ __forceinline__ void stage_half(std::uint32_t tmem, const float* bias, float scale,
                                           float* stage)
{
    float f[32];
    umma::load32(tmem, f);
    umma::wait_loads();
#pragma unroll
    for (int q = 0; q < 8; ++q)
    {
        stage4(stage, q,
               make_float4((f[4 * q] + bias[4 * q]) * scale,
                           (f[4 * q + 1] + bias[4 * q + 1]) * scale,
                           (f[4 * q + 2] + bias[4 * q + 2]) * scale,
                           (f[4 * q + 3] + bias[4 * q + 3]) * scale));
    }
}

// Resident CTAs per SM times the SM count, for a persistent grid: the least of the register
// file, shared memory (227 KB a CTA can use, 1 KB reserved per CTA) and tensor memory (512
// columns) over one CTA's needs.
int pair_grid(const void* kernel, int shared_bytes, int tmem_columns, int threads = kTile)
{
    int sms = 148;
    multiprocessors(&sms);
    int per_sm = 1;
    cudaFuncAttributes attributes{};
    if (cudaFuncGetAttributes(&attributes, kernel) == cudaSuccess)
    {
        const int registers = ((attributes.numRegs * 32 + 255) / 256) * 256 * (threads / 32);
        const int by_registers = 65536 / std::max(1, registers);
        const int by_shared =
            (228 * 1024) / (shared_bytes + static_cast<int>(attributes.sharedSizeBytes) + 1024);
        per_sm = std::max(1, std::min({by_registers, by_shared, 512 / tmem_columns}));
    }
    cudaGetLastError();
    return per_sm * std::max(1, sms);
}

}  // namespace
}  // namespace nd
