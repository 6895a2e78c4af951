// SchNet energy, forces and virial with the dense layers on BF16 tcgen05 tensor cores.
//
// The model is src/nabladyn/potential/_schnet/_potential.py:45-208 (64 features, K <= 64
// Gaussians, any number of blocks). The reference differentiates it with autograd
// (src/nabladyn/quantity.py:93-117); here the reverse pass is written out:
//
//   forward, per block b:  v = x A^T;  per pair p = (a, b) within the cutoff
//       z1 = g(r) B1^T + b1,  f_raw = ssp(z1) B2^T + b2,  f = f_raw C(r),
//       m_a += f * v_b,  m_b += f * v_a;
//     h = m D1^T + d1,  x += ssp(h) D2^T + d2;  E = sum_i ssp(x R1^T + e1) R2^T + e2
//   reverse:  G = dE/dx = (sigmoid(y) * R2) R1;  per block, last first:
//     Gh = (G D2) * sigmoid(h),  Gm = Gh D1;  per pair  Gf = Gm_a * v_b + Gm_b * v_a,
//       Gv_b += f * Gm_a,  Gv_a += f * Gm_b,
//       dE/dr += C'(r) (Gf . f_raw) + [((Gf C) B2 * sigmoid(z1)) B1] . g'(r);
//     G += Gv A
//   F_a -= dE/dr d / r,  F_b += dE/dr d / r,  W -= dE/dr d d^T / r.
//
// Every 64 x 64 product runs as a 128-row tile on the tensor cores: a [128 x 64] BF16 row
// tile (one pair per thread of a 128-thread CTA, or two threads per atom) times a BF16 image,
// FP32 accumulation in tensor memory (umma.cuh). The per-pair products (filter network
// forward, and its reverse) run in persistent CTAs that keep their weight images in shared
// memory; the atom-wise products in one CTA per 128 atoms. Everything else is FP32, the
// energy and virial sums FP64 in a fixed order. The feature rows the pair kernels gather
// (v and Gm) are stored in BF16; messages, their reverse and forces are summed in FP32, in an
// order that is fixed up to the atomics (add_runs in schnet.cuh).

#include "schnet.cuh"

namespace nd {
namespace {

// ---------------------------------------------------------------------------------------
// Pairs within the cutoff, compacted: (a, b) and (d, r), d = r_a - r_b of the minimum image
// as src/nabladyn/space.py:11-19 rounds it.

// Whether column c is a pair within the cutoff, with its atoms and geometry.
__device__ __forceinline__ bool column_pair(const float* __restrict__ positions,
                                            const float* __restrict__ cell,
                                            const std::int32_t* __restrict__ pairs,
                                            std::int64_t columns, std::int64_t c,
                                            std::int64_t atoms, float cutoff_squared, int2& ab,
                                            float4& g, int* counters)
{
    if (c >= columns)
    {
        return false;
    }
    ab = make_int2(pairs[c], pairs[columns + c]);
    if (ab.x == ab.y)
    {
        return false;
    }
    if (ab.x < 0 || ab.y < 0 || ab.x >= atoms || ab.y >= atoms)
    {
        atomicOr(counters + 1, kBadPair);
        return false;
    }
    float d[3];
#pragma unroll
    for (int axis = 0; axis < 3; ++axis)
    {
        const float length = cell[axis];
        const float left = positions[3 * ab.x + axis];
        const float right = positions[3 * ab.y + axis];
        const float raw = left - right;
        const float half = 0.5f * length;
        d[axis] = (left - (raw > half ? length : 0.0f)) - (right - (raw < -half ? length : 0.0f));
    }
    const float squared = __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])),
                                    __fmul_rn(d[2], d[2]));
    g = make_float4(d[0], d[1], d[2], sqrtf(squared));
    return squared < cutoff_squared;
}

// The compaction keeps the list's column order (count per block, scan, write), so the pairs
// of one first atom stay contiguous, as the list stores them.
__global__ void __launch_bounds__(kThreads) compact_count_kernel(
    const float* __restrict__ positions, const float* __restrict__ cell,
    const std::int32_t* __restrict__ pairs, std::int64_t columns, std::int64_t atoms,
    float cutoff_squared, int* __restrict__ block_counts, int* __restrict__ counters)
{
    int2 ab;
    float4 g;
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool keep = column_pair(positions, cell, pairs, columns, c, atoms, cutoff_squared, ab,
                                  g, counters);
    const int count = __syncthreads_count(keep);
    if (threadIdx.x == 0)
    {
        block_counts[blockIdx.x] = count;
    }
}

constexpr int kScanThreads = 1024;

__global__ void __launch_bounds__(kScanThreads) compact_scan_kernel(
    const int* __restrict__ block_counts, int blocks, int* __restrict__ block_offsets,
    int* __restrict__ counters)
{
    __shared__ int warp_totals[kScanThreads / kWarp];
    __shared__ int carry;
    if (threadIdx.x == 0)
    {
        carry = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    for (int base = 0; base < blocks; base += kScanThreads)
    {
        const int i = base + threadIdx.x;
        const int value = i < blocks ? block_counts[i] : 0;
        int inclusive = value;
#pragma unroll
        for (int offset = 1; offset < 32; offset *= 2)
        {
            const int other = __shfl_up_sync(kFullMask, inclusive, offset);
            inclusive += lane >= offset ? other : 0;
        }
        if (lane == 31)
        {
            warp_totals[warp] = inclusive;
        }
        __syncthreads();
        if (warp == 0)
        {
            int total = warp_totals[lane];
#pragma unroll
            for (int offset = 1; offset < 32; offset *= 2)
            {
                const int other = __shfl_up_sync(kFullMask, total, offset);
                total += lane >= offset ? other : 0;
            }
            warp_totals[lane] = total;  // inclusive over warps
        }
        __syncthreads();
        const int before = (warp > 0 ? warp_totals[warp - 1] : 0) + inclusive - value;
        if (i < blocks)
        {
            block_offsets[i] = carry + before;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            carry += warp_totals[kScanThreads / kWarp - 1];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        counters[0] = carry;
    }
}

__global__ void __launch_bounds__(kThreads) compact_write_kernel(
    const float* __restrict__ positions, const float* __restrict__ cell,
    const std::int32_t* __restrict__ pairs, std::int64_t columns, std::int64_t atoms,
    float cutoff_squared, const int* __restrict__ block_offsets, int2* __restrict__ kept,
    float4* __restrict__ geometry, int* __restrict__ counters)
{
    __shared__ int warp_base[kThreads / kWarp];
    int2 ab = make_int2(0, 0);
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool keep = column_pair(positions, cell, pairs, columns, c, atoms, cutoff_squared, ab,
                                  g, counters);
    const unsigned ballot = __ballot_sync(kFullMask, keep);
    const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    if (lane == 0)
    {
        warp_base[warp] = __popc(ballot);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int running = block_offsets[blockIdx.x];
        for (int w = 0; w < kThreads / kWarp; ++w)
        {
            const int count = warp_base[w];
            warp_base[w] = running;
            running += count;
        }
    }
    __syncthreads();
    if (keep)
    {
        const int slot = warp_base[warp] + __popc(ballot & ((1u << lane) - 1u));
        kept[slot] = ab;
        geometry[slot] = g;
    }
}

// x = embedding[type], v0 = (embedding A0^T)[type]; and zero in what the passes add to: every
// block's messages (`m`, `blocks` buffers of `row` float4 each), Gv and the forces. One thread
// per four features of an atom.
__global__ void __launch_bounds__(kThreads) embed_kernel(
    const std::int64_t* __restrict__ types, std::int64_t atoms, const float* __restrict__ table,
    const float* __restrict__ table_v, float* __restrict__ x, float* __restrict__ v,
    float4* __restrict__ m, int blocks, std::int64_t row, float4* __restrict__ grad_v,
    float* __restrict__ forces)
{
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= atoms * 16)
    {
        return;
    }
    const std::int64_t atom = i / 16;
    const int q = static_cast<int>(i % 16);
    const std::int64_t type = types[atom];
    reinterpret_cast<float4*>(x)[i] = reinterpret_cast<const float4*>(table)[type * 16 + q];
    const float4 value = reinterpret_cast<const float4*>(table_v)[type * 16 + q];
    reinterpret_cast<uint2*>(v)[i] = make_uint2(pack2(value.x, value.y), pack2(value.z, value.w));
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b = 0; b < blocks; ++b)
    {
        m[b * row + i] = zero;
    }
    if (grad_v != nullptr)
    {
        grad_v[i] = zero;
    }
    if (forces != nullptr && i < atoms * 3)
    {
        forces[i] = 0.0f;
    }
}

struct PairPass
{
    const int2* pairs;
    const float4* geometry;
    int* counters;
    const unsigned char* images;  // this block's ten images
    const float* b1;
    const float* b2;
    const float* v;           // [N][64] BF16: this block's x A^T
    float* m;                 // forward: messages
    const float* grad_m;      // reverse: Gm, [N][64] BF16
    float* grad_v;            // reverse: Gv (null for the first block)
    float* dedr;              // reverse: per-pair dE/dr over the blocks so far
    float* forces;            // reverse, last pass: F (null when not wanted)
    double* virial;           // reverse, last pass: per-CTA partials [gridDim.x][9]
    float width;              // Gaussian spacing D
    float phase;              // pi / r_c
    int gaussians;
    int first;                // reverse: the first pass (last block) starts dE/dr
};

// Shared memory of the pair passes: the filter layers' two weight images (the reverse pass
// reads them both ways), one row tile (each product's operand replaces the last once that
// product completed), in the reverse pass the FP32 filter's stage (the forward pass stages it
// in the row tile, free by then), biases, the pairs' atoms and envelopes, barrier and
// tensor-memory slot.
//
// What bounds the pair passes are the shared-memory passes between products (65 % of the load/store
// wavefronts forward, 54 % reverse), the special-function unit (36 %, 31-40 %) and the atomics, in
// a chain of dependent steps per tile; the tensor pipe is busy 6-8 % of the time. A row's features are gathered and scattered by eight
// lanes, 16 bytes each, so a warp's load covers four whole rows; with a thread per row each load
// touched 32. 32,768 beads, 1.19 million pairs: forward 269 -> 157 us, reverse 533 -> 300 us (the
// last pass 241), the E/F/W call 2,210 -> 1,510 us. Unrolled over the two column halves the kernels overflow the
// instruction cache, so those loops stay rolled.
//
// The reverse pass's row tile has its 16-byte chunks 144 bytes and its eight-row groups 1,216
// bytes apart: the eight lanes that write one row, four rows at a time, then spread over the
// shared-memory banks.
constexpr int kPairTail = 2 * 256 + 3 * kTile * 4 + 64;
constexpr int kReverseChunk = 144, kReverseGroup = 8 * kReverseChunk + 64;
constexpr int kReverseTileBytes = kTile / 8 * kReverseGroup;
constexpr int kPairForwardShared = 2 * umma::kImageBytes + umma::kTileBytes + kPairTail;
constexpr int kPairReverseShared =
    2 * umma::kImageBytes + kReverseTileBytes + umma::kTileBytes + kPairTail;

struct PairShared
{
    unsigned char* image_b1;
    unsigned char* image_b2;
    unsigned char* work;
    float* stage;
    float* bias1;
    float* bias2;
    int* first;       // -1: a dead row
    int* second;
    float* envelope;  // reverse
    std::uint64_t* barrier;

    __device__ PairShared(unsigned char* shared, bool reverse)
    {
        image_b1 = shared;
        image_b2 = image_b1 + umma::kImageBytes;
        work = image_b2 + umma::kImageBytes;
        stage = reinterpret_cast<float*>(reverse ? work + kReverseTileBytes : work);
        bias1 = stage + kTile * 32;
        bias2 = bias1 + kFeatures;
        first = reinterpret_cast<int*>(bias2 + kFeatures);
        second = first + kTile;
        envelope = reinterpret_cast<float*>(second + kTile);
        barrier = reinterpret_cast<std::uint64_t*>(envelope + kTile);
    }

    __device__ void load_biases(const PairPass& a)
    {
        if (threadIdx.x < kFeatures)
        {
            bias1[threadIdx.x] = a.b1[threadIdx.x];
            bias2[threadIdx.x] = a.b2[threadIdx.x];
        }
    }
};

// ssp(z + b1) of this thread's row, from tensor-memory columns 0-63, into the row tile.
template <int kChunk = 128, int kGroup = 1024>
__device__ __forceinline__ void store_softplus(std::uint32_t tmem, const float* bias1,
                                               unsigned char* tile)
{
#pragma unroll 1  // the unrolled kernel overflows the instruction cache
    for (int half = 0; half < 2; ++half)
    {
        float z[32];
        umma::load32(tmem + 32 * half, z);
        umma::wait_loads();
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            float s[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
            {
                s[e] = softplus_shifted(z[8 * c + e] + bias1[32 * half + 8 * c + e]);
            }
            umma::store8<kChunk, kGroup>(tile, threadIdx.x, 4 * half + c, s);
        }
    }
}

__global__ void __launch_bounds__(kTile, 6) pair_forward_kernel(PairPass a)
{
    extern __shared__ __align__(1024) unsigned char shared[];
    PairShared sh(shared, false);
    sh.load_biases(a);
    Cores cores;
    cores.open(sh.barrier, 64, a.counters, 1,
               {{sh.image_b1, a.images + kB1 * umma::kImageBytes},
                {sh.image_b2, a.images + kB2 * umma::kImageBytes}});
    const int count = *reinterpret_cast<volatile int*>(a.counters);
    const auto* v = reinterpret_cast<const uint2*>(a.v);
    float4* const m4 = reinterpret_cast<float4*>(a.m);
    const FeatureLane at;

    // Each tile's pair records are loaded one tile ahead, so their latency hides behind the
    // previous tile's products.
    int2 next_ab = make_int2(0, 0);
    float next_r = 1.0f;
    auto load_ahead = [&](int p) {
        const bool live = p < count;
        next_ab = live ? a.pairs[p] : make_int2(-1, 0);
        next_r = live ? a.geometry[p].w : 1.0f;
    };
    load_ahead(blockIdx.x * kTile + threadIdx.x);
    for (int tile = blockIdx.x; tile * kTile < count; tile += gridDim.x)
    {
        const float r = next_r;
        const float envelope = 0.5f * (__cosf(r * a.phase) + 1.0f);
        sh.first[threadIdx.x] = next_ab.x;
        sh.second[threadIdx.x] = next_ab.y;
        load_ahead((tile + gridDim.x) * kTile + threadIdx.x);
        cores.tile_index = tile;
        store_basis(sh.work, r / a.width, a.gaussians);
        if (!cores.run(0, sh.work, sh.image_b1, 1))
        {
            break;
        }
        store_softplus(cores.tmem, sh.bias1, sh.work);
        if (!cores.run(0, sh.work, sh.image_b2, 2))
        {
            break;
        }
        // Messages: m_a += f v_b along the lane's runs, m_b += f v_a pair by pair.
#pragma unroll 1
        for (int half = 0; half < 2; ++half)
        {
            uint2 vb[kLaneRows];
#pragma unroll
            for (int i = 0; i < kLaneRows; ++i)
            {
                vb[i] = __ldg(v + at.word(sh.second[at.row(i)], half));
            }
            stage_half(cores.tmem + 32 * half, sh.bias2 + 32 * half, envelope, sh.stage);
            __syncwarp();
            int key = sh.first[at.row(0)];
            float4 va = widen4(__ldg(v + at.word(max(key, 0), half)));
#pragma unroll
            for (int i = 0; i < kLaneRows; ++i)
            {
                const int row = at.row(i);
                const int first = sh.first[row];
                if (first != key)
                {
                    key = first;
                    va = widen4(__ldg(v + at.word(max(first, 0), half)));
                }
                const float4 f = staged4(sh.stage, row, at.lane);
                if (first >= 0)
                {
                    atomicAdd(m4 + at.word(sh.second[row], half), f * va);
                }
                restage4(sh.stage, row, at.lane, f * widen4(vb[i]));
            }
            __syncwarp();
            add_runs(sh.stage, sh.first, at.warp_row, a.m + 32 * half + (threadIdx.x & 31));
            __syncwarp();  // the stage's rows are this warp's own: its next writes come after
        }
    }
    cores.close(64);
}

// kLast: the last pass (block 0) has no Gv to scatter and applies forces and virial.
template <bool kLast>
__global__ void __launch_bounds__(kTile, 4) pair_reverse_kernel(PairPass a)
{
    extern __shared__ __align__(1024) unsigned char shared[];
    PairShared sh(shared, true);
    sh.load_biases(a);
    // Columns 0-63 keep z1 - b1 for the whole tile; 64-127 take the other products in turn.
    Cores cores;
    cores.open(sh.barrier, 128, a.counters, 2,
               {{sh.image_b1, a.images + kB1 * umma::kImageBytes},
                {sh.image_b2, a.images + kB2 * umma::kImageBytes}});
    const int count = *reinterpret_cast<volatile int*>(a.counters);
    const auto* v = reinterpret_cast<const uint2*>(a.v);
    const auto* gm = reinterpret_cast<const uint2*>(a.grad_m);
    float4* const gv4 = reinterpret_cast<float4*>(a.grad_v);
    const FeatureLane at;
    // D[64 + n] = the row tile times an image, read either way.
    auto product = [&](std::uint32_t column, const unsigned char* image, bool transposed, int step) {
        return cores.issue(
            [&] {
                const std::uint32_t tile = umma::smem_address(sh.work);
                const std::uint32_t b = umma::smem_address(image);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    umma::mma(*cores.slot + column,
                              umma::matrix_descriptor(tile + 2 * kReverseChunk * k, kReverseChunk,
                                                      kReverseGroup),
                              transposed ? umma::matrix_descriptor(b + 2048 * k, 1024, 128)
                                         : umma::matrix_descriptor(b + 256 * k),
                              k > 0 ? 1u : 0u, transposed ? umma::kTransposedB : umma::kInstruction);
                }
            },
            step);
    };
    double w[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // xx yy zz xy xz yz

    // Each tile's pair records are loaded one tile ahead (see pair_forward_kernel).
    int2 next_ab = make_int2(-1, 0);
    float4 next_g = make_float4(0.f, 0.f, 0.f, 1.f);
    auto load_ahead = [&](int p) {
        const bool live = p < count;
        next_ab = live ? a.pairs[p] : make_int2(-1, 0);
        next_g = live ? a.geometry[p] : make_float4(0.f, 0.f, 0.f, 1.f);
    };
    load_ahead(blockIdx.x * kTile + threadIdx.x);
    for (int tile = blockIdx.x; tile * kTile < count; tile += gridDim.x)
    {
        const int p = tile * kTile + threadIdx.x;
        const int2 ab = next_ab;
        const float4 g = next_g;
        load_ahead((tile + gridDim.x) * kTile + threadIdx.x);
        float sine, cosine;
        __sincosf(g.w * a.phase, &sine, &cosine);
        const float t = g.w / a.width;
        sh.first[threadIdx.x] = ab.x;
        sh.second[threadIdx.x] = ab.y;
        sh.envelope[threadIdx.x] = 0.5f * (cosine + 1.0f);
        cores.tile_index = tile;
        store_basis<kReverseChunk, kReverseGroup>(sh.work, t, a.gaussians);
        if (!product(0, sh.image_b1, false, 1))
        {
            break;
        }
        // ssp(z1) into the work tile; z1 - b1 stays in columns 0-63.
        store_softplus<kReverseChunk, kReverseGroup>(cores.tmem, sh.bias1, sh.work);
        if (!product(64, sh.image_b2, false, 2))
        {
            break;
        }
        // f_raw, Gf = Gm_a v_b + Gm_b v_a, Gf . f_raw, Gv, and Gf C into the work tile.
        float along = 0.0f;
#pragma unroll 1
        for (int half = 0; half < 2; ++half)
        {
            uint2 vb[kLaneRows], mb[kLaneRows];
#pragma unroll
            for (int i = 0; i < kLaneRows; ++i)
            {
                const std::int64_t word = at.word(sh.second[at.row(i)], half);
                vb[i] = __ldg(v + word);
                mb[i] = __ldg(gm + word);
            }
            stage_half(cores.tmem + 64 + 32 * half, sh.bias2 + 32 * half, 1.0f, sh.stage);
            __syncwarp();
            int key = sh.first[at.row(0)];
            float4 va = widen4(__ldg(v + at.word(max(key, 0), half)));
            float4 ma = widen4(__ldg(gm + at.word(max(key, 0), half)));
            float4 to_first[kLaneRows];
#pragma unroll
            for (int i = 0; i < kLaneRows; ++i)
            {
                const int row = at.row(i);
                const int first = sh.first[row];
                if (first != key)
                {
                    key = first;
                    const std::int64_t word = at.word(max(first, 0), half);
                    va = widen4(__ldg(v + word));
                    ma = widen4(__ldg(gm + word));
                }
                const float envelope = sh.envelope[row];
                const float4 raw = staged4(sh.stage, row, at.lane);
                const float4 right = widen4(vb[i]), right_gm = widen4(mb[i]);
                const float4 gf = fma4(ma, right, right_gm * va);
                restage4(sh.stage, row, at.lane, gf);
                if (!kLast)
                {
                    const float4 scaled = raw * envelope;
                    if (first >= 0)
                    {
                        atomicAdd(gv4 + at.word(sh.second[row], half), scaled * ma);
                    }
                    to_first[i] = scaled * right_gm;
                }
                *reinterpret_cast<uint2*>(sh.work + (row >> 3) * kReverseGroup +
                                          (4 * half + at.lane / 2) * kReverseChunk +
                                          (row & 7) * 16 + (at.lane & 1) * 8) =
                    make_uint2(pack2(gf.x * envelope, gf.y * envelope),
                               pack2(gf.z * envelope, gf.w * envelope));
            }
            __syncwarp();
            // Gf . f_raw of this thread's own row, in column order.
#pragma unroll
            for (int part = 0; part < 2; ++part)
            {
                float raw[16];
                umma::load16(cores.tmem + 64 + 32 * half + 16 * part, raw);
                umma::wait_loads();
                const float* bias = sh.bias2 + 32 * half + 16 * part;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                {
                    const float4 gf = staged4(sh.stage, threadIdx.x, 4 * part + q);
                    along = fmaf(gf.x, raw[4 * q] + bias[4 * q], along);
                    along = fmaf(gf.y, raw[4 * q + 1] + bias[4 * q + 1], along);
                    along = fmaf(gf.z, raw[4 * q + 2] + bias[4 * q + 2], along);
                    along = fmaf(gf.w, raw[4 * q + 3] + bias[4 * q + 3], along);
                }
            }
            __syncwarp();
            if (!kLast)
            {
#pragma unroll
                for (int i = 0; i < kLaneRows; ++i)
                {
                    restage4(sh.stage, at.row(i), at.lane, to_first[i]);
                }
                __syncwarp();
                add_runs(sh.stage, sh.first, at.warp_row,
                         a.grad_v + 32 * half + (threadIdx.x & 31));
                __syncwarp();  // the stage's rows are this warp's own: its next writes come after
            }
        }
        if (!product(64, sh.image_b2, true, 3))
        {
            break;
        }
        // ((Gf C) B2) * sigmoid(z1) into the work tile.
#pragma unroll 1
        for (int half = 0; half < 2; ++half)
        {
            float q[32];
            float z[32];
            umma::load32(cores.tmem + 64 + 32 * half, q);
            umma::load32(cores.tmem + 32 * half, z);
            umma::wait_loads();
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                float s[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                    s[e] = q[8 * c + e] * sigmoid(z[8 * c + e] + sh.bias1[32 * half + 8 * c + e]);
                }
                umma::store8<kReverseChunk, kReverseGroup>(sh.work, threadIdx.x, 4 * half + c, s);
            }
        }
        if (!product(64, sh.image_b1, true, 4))
        {
            break;
        }
        // dE/dr = C' Gf . f_raw + sum_k [..]_k g_k', g_k' = -g_k (r / D - k) / D, with the
        // Gaussians evaluated again in FP32 (columns k >= K hold zeros).
        float through = 0.0f;
#pragma unroll
        for (int half = 0; half < 2; ++half)
        {
            float u[32];
            umma::load32(cores.tmem + 64 + 32 * half, u);
            umma::wait_loads();
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                if (32 * half + 8 * c < a.gaussians)
                {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                    {
                        const float offset = t - static_cast<float>(32 * half + 8 * c + e);
                        through -= u[8 * c + e] * gaussian_flushed(offset) * offset;
                    }
                }
            }
        }
        if (ab.x >= 0)
        {
            const float slope = -0.5f * a.phase * sine;
            float total = slope * along + through / a.width;
            if (!a.first)
            {
                total += a.dedr[p];
            }
            if (!kLast)
            {
                a.dedr[p] = total;
            }
            else
            {
                const float scale = total / g.w;
                const float ux = scale * g.x, uy = scale * g.y, uz = scale * g.z;
                if (a.forces != nullptr)
                {
                    float* fa = a.forces + 3 * static_cast<std::int64_t>(ab.x);
                    float* fb = a.forces + 3 * static_cast<std::int64_t>(ab.y);
                    atomicAdd(fa, -ux);
                    atomicAdd(fa + 1, -uy);
                    atomicAdd(fa + 2, -uz);
                    atomicAdd(fb, ux);
                    atomicAdd(fb + 1, uy);
                    atomicAdd(fb + 2, uz);
                }
                w[0] -= static_cast<double>(ux) * g.x;
                w[1] -= static_cast<double>(uy) * g.y;
                w[2] -= static_cast<double>(uz) * g.z;
                w[3] -= static_cast<double>(ux) * g.y;
                w[4] -= static_cast<double>(ux) * g.z;
                w[5] -= static_cast<double>(uy) * g.z;
            }
        }
    }
    if (kLast && a.virial != nullptr)
    {
        __shared__ double sums[4][6];
#pragma unroll
        for (int k = 0; k < 6; ++k)
        {
            const double s = warp_sum(w[k]);
            if ((threadIdx.x & 31) == 0)
            {
                sums[threadIdx.x / 32][k] = s;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            double t6[6];
            for (int k = 0; k < 6; ++k)
            {
                t6[k] = ((sums[0][k] + sums[1][k]) + sums[2][k]) + sums[3][k];
            }
            double* out = a.virial + 9 * static_cast<std::int64_t>(blockIdx.x);
            out[0] = t6[0];
            out[4] = t6[1];
            out[8] = t6[2];
            out[1] = out[3] = t6[3];
            out[2] = out[6] = t6[4];
            out[5] = out[7] = t6[5];
        }
    }
    cores.close(128);
}

struct AtomPass
{
    std::int64_t atoms;
    const unsigned char* images;       // this block's images
    const unsigned char* next_images;  // forward: the next block's (for v); reverse: its (for Gv A)
    const float* d1;
    const float* d2;
    const float* m;        // forward
    float* h;              // forward: writes; reverse: reads
    float* x;              // forward: updated in place
    float* v_next;         // forward: the next block's v in BF16 (null for the last block)
    const float* readout;  // forward, last block: R1, e1, R2, e2
    float* grad;           // forward, last block: writes dE/dx; reverse: reads, updates
    float* grad_v;         // reverse: Gv of the next block, read and set to zero (null for the
                           // last block)
    float* grad_m;         // reverse: writes Gm in BF16
    double* energy;        // forward, last block: per-CTA partials
    int* counters;
};

// The atom-wise layers: one CTA of 256 threads per 128 atoms, thread t computing columns
// 32 (t / 128) .. + 31 of row t % 128. A small system has fewer tiles than SMs and one chain of
// products per tile, so what counts is the chain's length: two threads per row halve its
// row-wise part (with the sums cleared by these passes and the embedding instead of seven
// memsets, E/F/W of 2,048 beads 277 -> 252 us).
constexpr int kAtomThreads = 256;
constexpr int kHalf = kFeatures / 2;
constexpr int kReadoutFloats = kHidden * kFeatures + 3 * kHidden;
constexpr int kAtomShared =
    3 * umma::kImageBytes + umma::kTileBytes + kReadoutFloats * 4 + 2 * 256 + 64;
// The readout's exchange lies over the images and the tile, free by then: first the rows of x
// (68 floats apart: a row's 16-byte words then start in different banks), later ssp(y) and
// sigmoid(y) R2 of every hidden unit and row.
constexpr int kExchangeRow = 68;
static_assert(kTile * kExchangeRow * 4 <= 3 * umma::kImageBytes + umma::kTileBytes &&
                  2 * kHidden * kTile * 4 <= 3 * umma::kImageBytes + umma::kTileBytes,
              "the exchange fits");

struct AtomRow
{
    std::int64_t row;  // the atom
    bool live;
    int local;  // row of the tile
    int side;   // columns 32 side .. 32 side + 31

    __device__ explicit AtomRow(std::int64_t atoms)
        : local(threadIdx.x % kTile), side(threadIdx.x / kTile)
    {
        row = static_cast<std::int64_t>(blockIdx.x) * kTile + local;
        live = row < atoms;
    }

    __device__ __forceinline__ void load(const float* source, float (&out)[kHalf]) const
    {
        const float4* s4 = reinterpret_cast<const float4*>(source) + 16 * row + 8 * side;
#pragma unroll
        for (int q = 0; q < 8; ++q)
        {
            const float4 value = live ? s4[q] : make_float4(0.f, 0.f, 0.f, 0.f);
            out[4 * q] = value.x;
            out[4 * q + 1] = value.y;
            out[4 * q + 2] = value.z;
            out[4 * q + 3] = value.w;
        }
    }

    __device__ __forceinline__ void store(float* target, const float (&values)[kHalf]) const
    {
        float4* t4 = reinterpret_cast<float4*>(target) + 16 * row + 8 * side;
#pragma unroll
        for (int q = 0; q < 8; ++q)
        {
            if (live)
            {
                t4[q] = make_float4(values[4 * q], values[4 * q + 1], values[4 * q + 2],
                                    values[4 * q + 3]);
            }
        }
    }

    __device__ __forceinline__ void store_bf16(float* target, const float (&values)[kHalf]) const
    {
        uint4* t4 = reinterpret_cast<uint4*>(target) + 8 * row + 4 * side;
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            if (live)
            {
                t4[q] = umma::pack8(values + 8 * q);
            }
        }
    }

    __device__ __forceinline__ void store_tile(unsigned char* tile,
                                               const float (&values)[kHalf]) const
    {
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            umma::store8(tile, local, 4 * side + c, values + 8 * c);
        }
    }

    // The accumulator's columns of this thread.
    __device__ __forceinline__ void load_product(const Cores& cores, float (&out)[kHalf]) const
    {
        umma::load32(cores.tmem + 32 * side, out);
        umma::wait_loads();
    }
};

// e = ssp(x R1^T + e1) R2^T + e2 and dE/dx of the last block's x: each side computes half of
// the hidden units from whole rows, then half of the gradient's columns from all of them (the
// sums over features and over hidden units run in index order).
__device__ __forceinline__ float readout_row(const AtomRow& at, const float* readout,
                                             float* exchange, const float (&x)[kHalf],
                                             float (&grad)[kHalf])
{
    const float* r1 = readout;
    const float* e1 = readout + kHidden * kFeatures;
    const float* r2 = e1 + kHidden;
    const float e2 = r2[kHidden];
#pragma unroll
    for (int q = 0; q < 8; ++q)
    {
        *reinterpret_cast<float4*>(exchange + at.local * kExchangeRow + 32 * at.side + 4 * q) =
            make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
    }
    __syncthreads();
    float whole[kFeatures];
#pragma unroll
    for (int q = 0; q < 16; ++q)
    {
        const float4 value =
            *reinterpret_cast<const float4*>(exchange + at.local * kExchangeRow + 4 * q);
        whole[4 * q] = value.x;
        whole[4 * q + 1] = value.y;
        whole[4 * q + 2] = value.z;
        whole[4 * q + 3] = value.w;
    }
    __syncthreads();
    float* softplus = exchange;                   // [hidden][row]
    float* slopes = exchange + kHidden * kTile;
#pragma unroll 2
    for (int j = kHidden / 2 * at.side; j < kHidden / 2 * (at.side + 1); ++j)
    {
        float y = e1[j];
#pragma unroll
        for (int k = 0; k < kFeatures; ++k)
        {
            y = fmaf(whole[k], r1[j * kFeatures + k], y);
        }
        softplus[j * kTile + at.local] = softplus_shifted(y);
        slopes[j * kTile + at.local] = sigmoid(y) * r2[j];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kHalf; ++k)
    {
        grad[k] = 0.0f;
    }
    float e = e2;
    for (int j = 0; j < kHidden; ++j)
    {
        e += softplus[j * kTile + at.local] * r2[j];
        const float s = slopes[j * kTile + at.local];
#pragma unroll
        for (int k = 0; k < kHalf; ++k)
        {
            grad[k] = fmaf(s, r1[j * kFeatures + 32 * at.side + k], grad[k]);
        }
    }
    return e;
}

// h = m D1^T + d1, x += ssp(h) D2^T + d2, then v' = x A'^T, or on the last block the readout:
// e = ssp(x R1^T + e1) R2^T + e2 and dE/dx.
template <bool kLast>
__global__ void __launch_bounds__(kAtomThreads) atom_forward_kernel(AtomPass a)
{
    extern __shared__ __align__(1024) unsigned char shared[];
    unsigned char* image_d1 = shared;
    unsigned char* image_d2 = image_d1 + umma::kImageBytes;
    unsigned char* image_a = image_d2 + umma::kImageBytes;
    unsigned char* tile = image_a + umma::kImageBytes;
    float* readout = reinterpret_cast<float*>(tile + umma::kTileBytes);
    float* bias1 = readout + kReadoutFloats;
    float* bias2 = bias1 + kFeatures;
    auto* barrier = reinterpret_cast<std::uint64_t*>(bias2 + kFeatures);

    const AtomRow at(a.atoms);
    float values[kHalf], x[kHalf];
    at.load(a.m, values);
    at.load(a.x, x);
    if (kLast)
    {
        for (int i = threadIdx.x; i < kReadoutFloats; i += kAtomThreads)
        {
            readout[i] = a.readout[i];
        }
    }
    if (threadIdx.x < kFeatures)
    {
        bias1[threadIdx.x] = a.d1[threadIdx.x];
        bias2[threadIdx.x] = a.d2[threadIdx.x];
    }
    Cores cores;
    const ImageCopy d1{image_d1, a.images + kD1 * umma::kImageBytes};
    const ImageCopy d2{image_d2, a.images + kD2 * umma::kImageBytes};
    if constexpr (kLast)
    {
        cores.open(barrier, 64, a.counters, 3, {d1, d2});
    }
    else
    {
        cores.open(barrier, 64, a.counters, 3,
                   {d1, d2, {image_a, a.next_images + kA * umma::kImageBytes}});
    }
    cores.tile_index = blockIdx.x;
    double energy = 0.0;
    at.store_tile(tile, values);
    bool ok = cores.run(0, tile, image_d1, 1);
    if (ok)
    {
        at.load_product(cores, values);
#pragma unroll
        for (int k = 0; k < kHalf; ++k)
        {
            values[k] += bias1[32 * at.side + k];
        }
        at.store(a.h, values);
#pragma unroll
        for (int k = 0; k < kHalf; ++k)
        {
            values[k] = softplus_shifted(values[k]);
        }
        at.store_tile(tile, values);
        ok = cores.run(0, tile, image_d2, 2);
    }
    if (ok)
    {
        at.load_product(cores, values);
#pragma unroll
        for (int k = 0; k < kHalf; ++k)
        {
            x[k] += values[k] + bias2[32 * at.side + k];
        }
        if (!kLast)
        {
            at.store(a.x, x);
            at.store_tile(tile, x);
            ok = cores.run(0, tile, image_a, 3);
            if (ok)
            {
                at.load_product(cores, values);
                at.store_bf16(a.v_next, values);
            }
        }
        else
        {
            const float e = readout_row(at, readout, reinterpret_cast<float*>(shared), x, values);
            at.store(a.grad, values);
            energy = at.live && at.side == 0 ? e : 0.0;
        }
    }
    if (kLast)
    {
        __shared__ double sums[4];
        const double s = warp_sum(energy);
        if ((threadIdx.x & 31) == 0 && at.side == 0)
        {
            sums[threadIdx.x / 32] = s;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            a.energy[blockIdx.x] = ((sums[0] + sums[1]) + sums[2]) + sums[3];
        }
    }
    cores.close(64);
}

// Reverse of one block's atom-wise layers: G += Gv' A' (the next block's messages; Gv' goes
// back to zero for this block's pair pass), then Gh = (G D2) * sigmoid(h) and Gm = Gh D1.
__global__ void __launch_bounds__(kAtomThreads) atom_reverse_kernel(AtomPass a)
{
    extern __shared__ __align__(1024) unsigned char shared[];
    unsigned char* image_d2t = shared;
    unsigned char* image_d1t = image_d2t + umma::kImageBytes;
    unsigned char* image_at = image_d1t + umma::kImageBytes;
    unsigned char* tile = image_at + umma::kImageBytes;
    auto* barrier = reinterpret_cast<std::uint64_t*>(tile + umma::kTileBytes);

    const bool chained = a.grad_v != nullptr;
    const AtomRow at(a.atoms);
    float grad[kHalf], values[kHalf], h[kHalf];
    at.load(a.grad, grad);
    at.load(a.h, h);
    if (chained)
    {
        at.load(a.grad_v, values);
    }
    Cores cores;
    const ImageCopy d2t{image_d2t, a.images + kD2T * umma::kImageBytes};
    const ImageCopy d1t{image_d1t, a.images + kD1T * umma::kImageBytes};
    if (chained)
    {
        cores.open(barrier, 64, a.counters, 4,
                   {d2t, d1t, {image_at, a.next_images + kAT * umma::kImageBytes}});
    }
    else
    {
        cores.open(barrier, 64, a.counters, 4, {d2t, d1t});
    }
    cores.tile_index = blockIdx.x;
    bool ok = true;
    if (chained)
    {
        at.store_tile(tile, values);
        const float zeros[kHalf] = {};
        at.store(a.grad_v, zeros);
        ok = cores.run(0, tile, image_at, 1);
        if (ok)
        {
            at.load_product(cores, values);
#pragma unroll
            for (int k = 0; k < kHalf; ++k)
            {
                grad[k] += values[k];
            }
            at.store(a.grad, grad);
        }
    }
    if (ok)
    {
        at.store_tile(tile, grad);
        ok = cores.run(0, tile, image_d2t, 2);
    }
    if (ok)
    {
        at.load_product(cores, values);
#pragma unroll
        for (int k = 0; k < kHalf; ++k)
        {
            values[k] *= sigmoid(h[k]);
        }
        at.store_tile(tile, values);
        ok = cores.run(0, tile, image_d1t, 3);
    }
    if (ok)
    {
        at.load_product(cores, values);
        at.store_bf16(a.grad_m, values);
    }
    cores.close(64);
}

// E and W from the per-CTA partials in a fixed order: a warp per sum.
constexpr int kFinalizeWarps = 10;
// Partials a lane loads before it adds any: all of its own when the last pass runs 592 CTAs (four
// per SM). Loaded as they are added they were a chain of round trips to L2: 7.5 -> 2.5 us, at the
// end of an evaluation whose every launch waits for the one before.
constexpr int kFinalizeLoads = 19;

__global__ void __launch_bounds__(kFinalizeWarps * 32) finalize_kernel(
    const double* __restrict__ energy_partials, int energy_count,
    const double* __restrict__ virial_partials, int virial_count, double* energy, double* virial)
{
    const int lane = threadIdx.x & 31;
    const int sum = threadIdx.x / 32;  // 0: E, 1 + c: component c of W
    const double* from = sum == 0 ? energy_partials : virial_partials + (sum - 1);
    const int count = sum == 0 ? energy_count : virial_count, stride = sum == 0 ? 1 : 9;
    double value = 0.0;
    for (int base = lane; base < count; base += 32 * kFinalizeLoads)
    {
        double part[kFinalizeLoads];
#pragma unroll
        for (int k = 0; k < kFinalizeLoads; ++k)
        {
            const int i = base + 32 * k;
            part[k] = i < count ? from[static_cast<std::int64_t>(stride) * i] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kFinalizeLoads; ++k)
        {
            value += part[k];
        }
    }
    value = warp_sum(value);
    double* to = sum == 0 ? energy : (virial != nullptr ? virial + (sum - 1) : nullptr);
    if (lane == 0 && to != nullptr)
    {
        *to = value;
    }
}

}  // namespace
}  // namespace nd

extern "C" {

int64_t nd_schnet_weight_bytes(int32_t interactions, int32_t num_types)
{
    if (interactions < 1 || num_types < 1)
    {
        return -1;
    }
    return nd::WeightLayout(interactions, num_types).total;
}

int64_t nd_schnet_workspace_bytes(int64_t num_atoms, int64_t num_columns, int32_t interactions)
{
    if (num_atoms < 1 || num_columns < 0 || interactions < 1)
    {
        return -1;
    }
    return nd::Workspace(num_atoms, num_columns, interactions).total;
}

int nd_schnet_energy_force_virial(const nd_schnet_args* args, nd_stream_t stream_handle)
{
    using namespace nd;
    ND_REQUIRE(args != nullptr, "args is null");
    const nd_schnet_args& s = *args;
    ND_REQUIRE(s.num_atoms >= 1 && s.num_atoms <= (int64_t{1} << 30), "num_atoms out of range");
    ND_REQUIRE(s.num_columns >= 0 && s.num_columns < (int64_t{1} << 31), "num_columns out of range");
    ND_REQUIRE(s.interactions >= 1 && s.interactions <= 64, "interactions out of range");
    ND_REQUIRE(s.num_types >= 1, "num_types must be positive");
    ND_REQUIRE(s.gaussians >= 2 && s.gaussians <= 64, "gaussians must lie in [2, 64]");
    ND_REQUIRE(s.cutoff > 0.0, "cutoff must be positive");
    ND_REQUIRE(s.positions && s.cell && s.atom_types && s.weights && s.workspace && s.status,
               "a required buffer is null");
    ND_REQUIRE(s.num_columns == 0 || s.pairs != nullptr, "pairs is null");
    ND_REQUIRE(reinterpret_cast<std::uintptr_t>(s.workspace) % 256 == 0 &&
                   reinterpret_cast<std::uintptr_t>(s.weights) % 256 == 0,
               "weights and workspace must be 256-byte aligned");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_handle);
    const WeightLayout wl(s.interactions, s.num_types);
    const Workspace ws(s.num_atoms, s.num_columns, s.interactions);
    auto* weights = static_cast<const unsigned char*>(s.weights);
    auto* base = static_cast<unsigned char*>(s.workspace);
    auto at = [&](std::int64_t offset) { return base + offset; };
    const std::int64_t row_bytes = align256(s.num_atoms * kFeatures * 4);
    auto block_images = [&](int b) { return weights + static_cast<std::int64_t>(b) * kImagesPerBlock * umma::kImageBytes; };
    auto block_vector = [&](int b, int j) {
        return reinterpret_cast<const float*>(weights + wl.vectors + (static_cast<std::int64_t>(b) * 4 + j) * kFeatures * 4);
    };
    int* counters = reinterpret_cast<int*>(at(ws.counters));
    auto* pairs = reinterpret_cast<int2*>(at(ws.pairs));
    auto* geometry = reinterpret_cast<float4*>(at(ws.geometry));
    auto* x = reinterpret_cast<float*>(at(ws.x));
    auto v = [&](int b) { return reinterpret_cast<float*>(at(ws.v + b * row_bytes)); };
    auto h = [&](int b) { return reinterpret_cast<float*>(at(ws.h + b * row_bytes)); };
    auto m = [&](int b) { return reinterpret_cast<float*>(at(ws.m + b * row_bytes)); };
    auto* grad = reinterpret_cast<float*>(at(ws.grad));
    auto* grad_m = reinterpret_cast<float*>(at(ws.grad_m));
    auto* grad_v = reinterpret_cast<float*>(at(ws.grad_v));
    auto* dedr = reinterpret_cast<float*>(at(ws.dedr));
    auto* energy_partials = reinterpret_cast<double*>(at(ws.energy));
    auto* virial_partials = reinterpret_cast<double*>(at(ws.virial));
    const int atom_tiles = static_cast<int>((s.num_atoms + kTile - 1) / kTile);
    const bool reverse = s.forces != nullptr || s.virial != nullptr;

    // The kernels' attributes, set once per device (they belong to its instance of a kernel).
    static DeviceOnce configured;  // per device, retried after a failure
    ND_CUDA_TRY(configured.run([] {
        cudaError_t rc = cudaFuncSetAttribute(pair_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairForwardShared);
        auto then = [&rc](cudaError_t next) { rc = rc != cudaSuccess ? rc : next; };
        then(cudaFuncSetAttribute(pair_reverse_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairReverseShared));
        then(cudaFuncSetAttribute(pair_reverse_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairReverseShared));
        then(cudaFuncSetAttribute(atom_forward_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAtomShared));
        then(cudaFuncSetAttribute(atom_forward_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAtomShared));
        then(cudaFuncSetAttribute(atom_reverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAtomShared));
        then(cudaFuncSetAttribute(pair_forward_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        then(cudaFuncSetAttribute(pair_reverse_kernel<false>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        then(cudaFuncSetAttribute(pair_reverse_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        return rc;
    }));
    const int forward_grid = pair_grid(reinterpret_cast<const void*>(pair_forward_kernel), kPairForwardShared, 64);
    const int reverse_grid = pair_grid(reinterpret_cast<const void*>(pair_reverse_kernel<false>), kPairReverseShared, 128);
    const int last_grid = std::min(kVirialSlots, pair_grid(reinterpret_cast<const void*>(pair_reverse_kernel<true>), kPairReverseShared, 128));

    ND_CUDA_TRY(cudaMemsetAsync(counters, 0, 256, stream));
    if (s.num_columns > 0)
    {
        const unsigned column_blocks = blocks_for(s.num_columns);
        auto* block_counts = reinterpret_cast<int*>(at(ws.block_counts));
        auto* block_offsets = reinterpret_cast<int*>(at(ws.block_offsets));
        const float cutoff_squared = static_cast<float>(s.cutoff * s.cutoff);
        compact_count_kernel<<<column_blocks, kThreads, 0, stream>>>(
            s.positions, s.cell, s.pairs, s.num_columns, s.num_atoms, cutoff_squared,
            block_counts, counters);
        ND_LAUNCH_CHECK();
        compact_scan_kernel<<<1, kScanThreads, 0, stream>>>(
            block_counts, static_cast<int>(column_blocks), block_offsets, counters);
        ND_LAUNCH_CHECK();
        compact_write_kernel<<<column_blocks, kThreads, 0, stream>>>(
            s.positions, s.cell, s.pairs, s.num_columns, s.num_atoms, cutoff_squared,
            block_offsets, pairs, geometry, counters);
        ND_LAUNCH_CHECK();
    }
    embed_kernel<<<blocks_for(s.num_atoms * 16), kThreads, 0, stream>>>(
        s.atom_types, s.num_atoms, reinterpret_cast<const float*>(weights + wl.tables),
        reinterpret_cast<const float*>(weights + wl.tables + s.num_types * kFeatures * 4), x, v(0),
        reinterpret_cast<float4*>(m(0)), s.interactions, row_bytes / 16,
        reverse ? reinterpret_cast<float4*>(grad_v) : nullptr, s.forces);
    ND_LAUNCH_CHECK();

    PairPass pass{};
    pass.pairs = pairs;
    pass.geometry = geometry;
    pass.counters = counters;
    pass.width = static_cast<float>(s.cutoff / (s.gaussians - 1));
    pass.phase = static_cast<float>(3.14159265358979323846 / s.cutoff);
    pass.gaussians = s.gaussians;
    const float* readout = reinterpret_cast<const float*>(weights + wl.readout);
    for (int b = 0; b < s.interactions; ++b)
    {
        const bool last = b == s.interactions - 1;
        pass.images = block_images(b);
        pass.b1 = block_vector(b, 0);
        pass.b2 = block_vector(b, 1);
        pass.v = v(b);
        pass.m = m(b);
        pair_forward_kernel<<<forward_grid, kTile, kPairForwardShared, stream>>>(pass);
        ND_LAUNCH_CHECK();
        AtomPass atoms{};
        atoms.atoms = s.num_atoms;
        atoms.images = block_images(b);
        atoms.next_images = last ? nullptr : block_images(b + 1);
        atoms.d1 = block_vector(b, 2);
        atoms.d2 = block_vector(b, 3);
        atoms.m = m(b);
        atoms.h = h(b);
        atoms.x = x;
        atoms.v_next = last ? nullptr : v(b + 1);
        atoms.readout = readout;
        atoms.grad = grad;
        atoms.energy = energy_partials;
        atoms.counters = counters;
        if (last)
        {
            atom_forward_kernel<true><<<atom_tiles, kAtomThreads, kAtomShared, stream>>>(atoms);
        }
        else
        {
            atom_forward_kernel<false><<<atom_tiles, kAtomThreads, kAtomShared, stream>>>(atoms);
        }
        ND_LAUNCH_CHECK();
    }
    if (reverse)
    {
        for (int b = s.interactions - 1; b >= 0; --b)
        {
            const bool last = b == s.interactions - 1;
            AtomPass atoms{};
            atoms.atoms = s.num_atoms;
            atoms.images = block_images(b);
            atoms.next_images = last ? nullptr : block_images(b + 1);
            atoms.h = h(b);
            atoms.grad = grad;
            atoms.grad_v = last ? nullptr : grad_v;
            atoms.grad_m = grad_m;
            atoms.counters = counters;
            atom_reverse_kernel<<<atom_tiles, kAtomThreads, kAtomShared, stream>>>(atoms);
            ND_LAUNCH_CHECK();
            pass.images = block_images(b);
            pass.b1 = block_vector(b, 0);
            pass.b2 = block_vector(b, 1);
            pass.v = v(b);
            pass.grad_m = grad_m;
            pass.grad_v = b > 0 ? grad_v : nullptr;
            pass.dedr = dedr;
            pass.first = last ? 1 : 0;
            pass.forces = s.forces;
            pass.virial = virial_partials;
            if (b > 0)
            {
                pair_reverse_kernel<false><<<reverse_grid, kTile, kPairReverseShared, stream>>>(pass);
            }
            else
            {
                pair_reverse_kernel<true><<<last_grid, kTile, kPairReverseShared, stream>>>(pass);
            }
            ND_LAUNCH_CHECK();
        }
    }
    finalize_kernel<<<1, kFinalizeWarps * 32, 0, stream>>>(energy_partials, atom_tiles, virial_partials,
                                           reverse ? last_grid : 0, s.energy,
                                           reverse ? s.virial : nullptr);
    ND_LAUNCH_CHECK();
    ND_CUDA_TRY(cudaMemcpyAsync(s.status, counters, 4 * sizeof(int), cudaMemcpyDeviceToDevice, stream));
    return ND_OK;
}

}  // extern "C"
