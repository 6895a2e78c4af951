// The per-pair passes of the SchNet parameter gradient of a training loss over E, F and W.
//
// The reference differentiates its loss with torch.func through a double backward
// (src/nabladyn/training/_fit.py:245-271, _loss.py:49-102). Written out: with the loss's
// adjoints e_bar = dL/dE, f_bar = dL/dF [N, 3] and w_bar = dL/dW [3, 3], F = -dE/dr and
// W = -dE/d(strain) make f_bar . F + w_bar : W the derivative of -E along a direction in which
// each pair's distance moves at
//     rdot = (d . (f_bar_a - f_bar_b) + d^T w_bar d) / r,
// so dL/dtheta = d/dtheta (e_bar E - Edot): a forward pass carrying beside each value its
// derivative along rdot, then one reverse pass over both streams. Per block, the pair work:
//
//   forward:  g, g_dot = g * (-(r / D - k) / D) rdot;  z, z_dot = (g, g_dot) B1^T (+ b1 on z);
//             s = ssp(z), s_dot = sigmoid(z) z_dot;  u, u_dot = (s, s_dot) B2^T (+ b2 on u);
//             f = u C, f_dot = u_dot C + u C' rdot;
//             m_dot_a += f_dot v_b + f v_dot_b, m_dot_b likewise (m itself, f v of the other
//             atom, is the E/F/W call's, copied from its workspace);
//   reverse, given m_bar and m_dot_bar from the atom-wise layers:
//             fb = m_bar_a v_b + m_bar_b v_a + m_dot_bar_a v_dot_b + m_dot_bar_b v_dot_a,
//             fdb = m_dot_bar_a v_b + m_dot_bar_b v_a;
//             v_bar_b += f m_bar_a + f_dot m_dot_bar_a, v_dot_bar_b += f m_dot_bar_a, and for a;
//             u_bar = fb C + fdb C' rdot, u_dot_bar = fdb C;
//             (s_bar, s_dot_bar) = (u_bar, u_dot_bar) B2;
//             z_bar = s_bar sigmoid(z) + s_dot_bar z_dot sigmoid'(z), z_dot_bar = s_dot_bar sigmoid(z).
//
// The reverse pass writes every pair's BF16 rows g, g_dot, s, s_dot, z_bar, z_dot_bar, u_bar,
// u_dot_bar, so the filter weights' gradients, sums over pairs (B1: z_bar^T g + z_dot_bar^T
// g_dot, B2: u_bar^T s + u_dot_bar^T s_dot, the biases the column sums of z_bar and u_bar), are
// plain GEMMs for the caller, as are the atom-wise 64 x 64 layers. With fewer than 64
// Gaussians the g row's last column holds 1, so column 63 of z_bar^T g is the sum of z_bar.
// Each product runs with its tangent as two 128 x 64 x 64 BF16 tcgen05 products on one commit;
// the tiles' rows are pairs in the compacted order of the preceding
// nd_schnet_energy_force_virial call, whose workspace this pass reads.

#include "schnet.cuh"

namespace nd {
namespace {

// Per-pair rows of the reverse pass, in this order, [8][capacity][64] BF16.
enum Row : int
{
    kRowG = 0,
    kRowGDot = 1,
    kRowS = 2,
    kRowSDot = 3,
    kRowZBar = 4,
    kRowZDotBar = 5,
    kRowUBar = 6,
    kRowUDotBar = 7,
};

struct TangentPass
{
    const int2* pairs;
    const float4* geometry;
    int* counters;
    const unsigned char* images;  // this block's ten images
    const float* b1;
    const float* b2;
    const float* force_adjoint;    // [N][3]
    const double* virial_adjoint;  // [9]
    const uint4* v;                // [N][64] BF16, 8 features a word
    const uint4* v_dot;
    float* m;                      // forward: [N][64], added to
    float* m_dot;
    const uint4* m_bar;            // reverse: [N][64] BF16
    const uint4* m_dot_bar;
    float* v_bar;                  // reverse: [N][64], added to
    float* v_dot_bar;
    uint4* rows;                   // reverse: [8][capacity][64] BF16 as 16-byte words
    std::int64_t capacity;
    float width;  // Gaussian spacing D
    float phase;  // pi / r_c
    int gaussians;
};

// The pair's geometry and the rate rdot at which the loss's direction moves its distance.
struct PairTerms
{
    int2 ab;
    float4 g;        // d, r
    bool live;
    float envelope;  // C(r)
    float moving;    // C'(r) rdot
    float rate;      // rdot
};

__device__ __forceinline__ PairTerms pair_terms(const TangentPass& a, const float* wbar, int p,
                                                int count)
{
    PairTerms t;
    t.live = p < count;
    t.ab = make_int2(0, 0);
    t.g = make_float4(0.f, 0.f, 0.f, 1.f);
    t.rate = 0.0f;
    if (t.live)
    {
        t.ab = a.pairs[p];
        t.g = a.geometry[p];
        const float* fa = a.force_adjoint + 3 * static_cast<std::int64_t>(t.ab.x);
        const float* fb = a.force_adjoint + 3 * static_cast<std::int64_t>(t.ab.y);
        const float d[3] = {t.g.x, t.g.y, t.g.z};
        float along = 0.0f;
#pragma unroll
        for (int i = 0; i < 3; ++i)
        {
            along += d[i] * (__ldg(fa + i) - __ldg(fb + i));
#pragma unroll
            for (int j = 0; j < 3; ++j)
            {
                along += d[i] * wbar[3 * i + j] * d[j];
            }
        }
        t.rate = along / t.g.w;
    }
    float sine, cosine;
    __sincosf(t.g.w * a.phase, &sine, &cosine);
    t.envelope = t.live ? 0.5f * (cosine + 1.0f) : 0.0f;
    t.moving = t.live ? -0.5f * a.phase * sine * t.rate : 0.0f;
    return t;
}

// g_k = exp(-(t - k)^2 / 2) (zero for k >= K) and g_dot_k = g_k (t - k) scale, scale = -rdot / D,
// into this thread's row of two tiles.
__device__ __forceinline__ void store_basis_tangent(unsigned char* tile, unsigned char* tile_dot,
                                                    float t, float scale, int gaussians)
{
#pragma unroll
    for (int c = 0; c < 8; ++c)
    {
        float g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float gd[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (8 * c < gaussians)  // the weight image is zero in columns K and up
        {
#pragma unroll
            for (int e = 0; e < 8; ++e)
            {
                const float u = t - static_cast<float>(8 * c + e);
                g[e] = gaussian(u);
                gd[e] = g[e] * u * scale;
            }
        }
        umma::store8(tile, threadIdx.x, c, g);
        umma::store8(tile_dot, threadIdx.x, c, gd);
    }
}

// s = ssp(z + b1) and s_dot = sigmoid(z + b1) z_dot from tensor-memory columns 0-63 (z - b1) and
// 64-127 (z_dot) into this thread's row of two tiles.
__device__ __forceinline__ void store_activations(std::uint32_t tmem, const float* bias1,
                                                  unsigned char* tile, unsigned char* tile_dot)
{
#pragma unroll 1  // the unrolled kernel overflows the instruction cache
    for (int part = 0; part < 4; ++part)
    {
        float z[16], zd[16];
        umma::load16(tmem + 16 * part, z);
        umma::load16(tmem + 64 + 16 * part, zd);
        umma::wait_loads();
#pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            float s[8];
            float sd[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
            {
                const float x = z[8 * c + e] + bias1[16 * part + 8 * c + e];
                s[e] = softplus_shifted(x);
                sd[e] = sigmoid(x) * zd[8 * c + e];
            }
            umma::store8(tile, threadIdx.x, 2 * part + c, s);
            umma::store8(tile_dot, threadIdx.x, 2 * part + c, sd);
        }
    }
}

constexpr int kTangentForwardShared =
    2 * umma::kImageBytes + 2 * umma::kTileBytes + 2 * 256 + 2 * kTile * 4 + 64;

__global__ void __launch_bounds__(kTile, 4) tangent_forward_kernel(TangentPass a)
{
    extern __shared__ __align__(1024) unsigned char shared[];
    unsigned char* image_b1 = shared;
    unsigned char* image_b2 = image_b1 + umma::kImageBytes;
    unsigned char* tile = image_b2 + umma::kImageBytes;
    unsigned char* tile_dot = tile + umma::kTileBytes;
    // f and f_dot, a half at a time, in the row tiles once the products are done
    float* stage = reinterpret_cast<float*>(tile);
    float* stage_dot = reinterpret_cast<float*>(tile_dot);
    float* bias1 = reinterpret_cast<float*>(tile_dot + umma::kTileBytes);
    float* bias2 = bias1 + kFeatures;
    int* first = reinterpret_cast<int*>(bias2 + kFeatures);
    int* second = first + kTile;
    auto* barrier = reinterpret_cast<std::uint64_t*>(second + kTile);
    __shared__ float wbar[9];

    if (threadIdx.x < kFeatures)
    {
        bias1[threadIdx.x] = a.b1[threadIdx.x];
        bias2[threadIdx.x] = a.b2[threadIdx.x];
    }
    if (threadIdx.x < 9)
    {
        wbar[threadIdx.x] = static_cast<float>(a.virial_adjoint[threadIdx.x]);
    }
    // Columns 0-63: z, then u; 64-127: z_dot, then u_dot.
    Cores cores;
    cores.open(barrier, 128, a.counters, 5,
               {{image_b1, a.images + kB1 * umma::kImageBytes},
                {image_b2, a.images + kB2 * umma::kImageBytes}});
    const int count = *reinterpret_cast<volatile int*>(a.counters);
    const auto* v = reinterpret_cast<const uint2*>(a.v);
    const auto* v_dot = reinterpret_cast<const uint2*>(a.v_dot);
    float4* const md4 = reinterpret_cast<float4*>(a.m_dot);
    const FeatureLane at;

    for (int index = blockIdx.x; index * kTile < count; index += gridDim.x)
    {
        const int p = index * kTile + threadIdx.x;
        const PairTerms t = pair_terms(a, wbar, p, count);
        first[threadIdx.x] = t.live ? t.ab.x : -1;
        second[threadIdx.x] = t.ab.y;
        cores.tile_index = index;
        store_basis_tangent(tile, tile_dot, t.g.w / a.width, -t.rate / a.width, a.gaussians);
        if (!cores.run2(0, tile, image_b1, 64, tile_dot, image_b1, 1))
        {
            break;
        }
        store_activations(cores.tmem, bias1, tile, tile_dot);
        if (!cores.run2(0, tile, image_b2, 64, tile_dot, image_b2, 2))
        {
            break;
        }
        // m_dot_a += f_dot v_b + f v_dot_b along the runs, m_dot_b += f_dot v_a + f v_dot_a.
#pragma unroll 1
        for (int half = 0; half < 2; ++half)
        {
            uint2 vb[kLaneRows], vdb[kLaneRows];
#pragma unroll
            for (int i = 0; i < kLaneRows; ++i)
            {
                const std::int64_t word = at.word(second[at.row(i)], half);
                vb[i] = __ldg(v + word);
                vdb[i] = __ldg(v_dot + word);
            }
            {
                float u[32], ud[32];
                umma::load32(cores.tmem + 32 * half, u);
                umma::load32(cores.tmem + 64 + 32 * half, ud);
                umma::wait_loads();
                const float* bias = bias2 + 32 * half;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                {
                    float f[4], fd[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                    {
                        const float raw_filter = u[4 * q + e] + bias[4 * q + e];
                        f[e] = raw_filter * t.envelope;
                        // The reverse pass fuses the other product; each as it always has.
                        fd[e] = fmaf(raw_filter, t.moving, ud[4 * q + e] * t.envelope);
                    }
                    stage4(stage, q, make_float4(f[0], f[1], f[2], f[3]));
                    stage4(stage_dot, q, make_float4(fd[0], fd[1], fd[2], fd[3]));
                }
            }
            __syncwarp();
            int key = first[at.row(0)];
            float4 va = widen4(__ldg(v + at.word(max(key, 0), half)));
            float4 vda = widen4(__ldg(v_dot + at.word(max(key, 0), half)));
#pragma unroll
            for (int i = 0; i < kLaneRows; ++i)
            {
                const int row = at.row(i);
                const int atom = first[row];
                if (atom != key)
                {
                    key = atom;
                    va = widen4(__ldg(v + at.word(max(atom, 0), half)));
                    vda = widen4(__ldg(v_dot + at.word(max(atom, 0), half)));
                }
                const float4 f = staged4(stage, row, at.lane), fd = staged4(stage_dot, row, at.lane);
                if (atom >= 0)
                {
                    atomicAdd(md4 + at.word(second[row], half), fma4(fd, va, f * vda));
                }
                restage4(stage, row, at.lane, fma4(fd, widen4(vb[i]), f * widen4(vdb[i])));
            }
            __syncwarp();
            add_runs(stage, first, at.warp_row, a.m_dot + 32 * half + (threadIdx.x & 31));
            __syncwarp();  // the stages' rows are this warp's own: its next writes come after
        }
    }
    cores.close(128);
}

// The reverse pass. 32,768 beads, 1.19 million pairs: 1,200 -> 615 us (the forward pass 520 ->
// 253 us), bound by the latency of a tile's steps and the shared-memory passes (61 % of the
// wavefronts), then by the 1.3 GB of rows it writes (27 % of the DRAM's peak).
//
// A tile's steps form one long chain (four products with row-wise work between
// them), so two CTAs share an SM (tensor memory holds no more: z, z_dot, u and u_dot are 256
// columns) and each gives a tile 256 threads: thread t computes columns 32 (t / 128) .. + 31 of
// row t % 128 in the row-wise steps. In the scatter, eight lanes take a row's 32 staged columns
// (columns 16 step .. + 15 of both halves, step 0 and 1), four rows of the warp's 16 at a time.
// The eight BF16 rows of a pair leave from the operand tiles in whole lines while the tensor
// cores read them; with chunks 144 bytes and eight-row groups 1,184 bytes apart both that and
// the lanes' writes of four rows spread over the shared-memory banks.
constexpr int kReverseThreads = 256;
constexpr int kRowChunk = 144, kRowGroup = 8 * kRowChunk + 32;  // of the row tiles
constexpr int kRowTileBytes = kTile / 8 * kRowGroup;
constexpr int kTangentReverseShared = 2 * umma::kImageBytes + 2 * kRowTileBytes +
                                      2 * kTile * 32 * 4 + 2 * 256 + 6 * kTile * 4 + 128;

__device__ __forceinline__ unsigned char* row_word(unsigned char* tile, int row, int c)
{
    return tile + (row >> 3) * kRowGroup + c * kRowChunk + (row & 7) * 16;
}

__global__ void __launch_bounds__(kReverseThreads, 2) tangent_reverse_kernel(TangentPass a)
{
    extern __shared__ __align__(1024) unsigned char shared[];
    unsigned char* image_b1 = shared;
    unsigned char* image_b2 = image_b1 + umma::kImageBytes;
    unsigned char* tile = image_b2 + umma::kImageBytes;
    unsigned char* tile_dot = tile + kRowTileBytes;
    float* stage = reinterpret_cast<float*>(tile_dot + kRowTileBytes);  // f
    float* stage_dot = stage + kTile * 32;                              // f_dot
    float* bias1 = stage_dot + kTile * 32;
    float* bias2 = bias1 + kFeatures;
    int* first = reinterpret_cast<int*>(bias2 + kFeatures);
    int* second = first + kTile;
    float* envelopes = reinterpret_cast<float*>(second + kTile);
    float* movings = envelopes + kTile;
    float* offsets = movings + kTile;  // r / D
    float* scales = offsets + kTile;   // -rdot / D
    float* wbar = scales + kTile;
    auto* barrier = reinterpret_cast<std::uint64_t*>(wbar + 10);

    if (threadIdx.x < kFeatures)
    {
        bias1[threadIdx.x] = a.b1[threadIdx.x];
        bias2[threadIdx.x] = a.b2[threadIdx.x];
    }
    if (threadIdx.x < 9)
    {
        wbar[threadIdx.x] = static_cast<float>(a.virial_adjoint[threadIdx.x]);
    }
    // Columns 0-63 keep z - b1 and 64-127 z_dot for the whole tile; 128-191 take u, then s_bar;
    // 192-255 u_dot, then s_dot_bar.
    Cores cores;
    cores.open(barrier, 256, a.counters, 6,
               {{image_b1, a.images + kB1 * umma::kImageBytes},
                {image_b2, a.images + kB2 * umma::kImageBytes}});
    const std::uint32_t tmem = *cores.slot;
    const int count = *reinterpret_cast<volatile int*>(a.counters);
    const auto* v = reinterpret_cast<const uint2*>(a.v);
    const auto* v_dot = reinterpret_cast<const uint2*>(a.v_dot);
    const auto* m_bar = reinterpret_cast<const uint2*>(a.m_bar);
    const auto* m_dot_bar = reinterpret_cast<const uint2*>(a.m_dot_bar);
    float4* const vbar4 = reinterpret_cast<float4*>(a.v_bar);
    float4* const vdbar4 = reinterpret_cast<float4*>(a.v_dot_bar);
    const int row = threadIdx.x % kTile, side = threadIdx.x / kTile;
    // The scatter's rows: 16 of the 32 that this warp and the one of the other side staged.
    const int lane = threadIdx.x % 8;
    const int lane_row = 32 * (threadIdx.x / 32 % 4) + 16 * side + 4 * (threadIdx.x % 32 / 8);

    // Both streams' products of the tiles with an image (read the other way when transposed).
    auto products = [&](std::uint32_t column, const unsigned char* image, bool transposed) {
        const std::uint32_t b = umma::smem_address(image);
#pragma unroll
        for (int stream = 0; stream < 2; ++stream)
        {
            const std::uint32_t from = umma::smem_address(stream == 0 ? tile : tile_dot);
#pragma unroll
            for (int step = 0; step < 4; ++step)
            {
                umma::mma(tmem + column + 64 * stream,
                          umma::matrix_descriptor(from + 2 * kRowChunk * step, kRowChunk, kRowGroup),
                          transposed ? umma::matrix_descriptor(b + 2048 * step, 1024, 128)
                                     : umma::matrix_descriptor(b + 256 * step),
                          step > 0 ? 1u : 0u,
                          transposed ? umma::kTransposedB : umma::kInstruction);
            }
        }
    };
    // The tiles' live rows to the per-pair arrays `kind` and `kind` + 1, eight lanes a row. The
    // Gaussians' HBM row holds 1 in column 63 when K < 64 (a column the products never use).
    auto copy_rows = [&](int kind, int index, bool ones) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const int r = (k * kReverseThreads + threadIdx.x) / 8, c = threadIdx.x % 8;
            const int p = index * kTile + r;
            if (p < count)
            {
                uint4 word = *reinterpret_cast<const uint4*>(row_word(tile, r, c));
                if (ones && c == 7)
                {
                    word.w = (word.w & 0xFFFFu) | 0x3F800000u;
                }
                a.rows[(static_cast<std::int64_t>(kind) * a.capacity + p) * 8 + c] = word;
                a.rows[(static_cast<std::int64_t>(kind + 1) * a.capacity + p) * 8 + c] =
                    *reinterpret_cast<const uint4*>(row_word(tile_dot, r, c));
            }
        }
    };

    for (int index = blockIdx.x; index * kTile < count; index += gridDim.x)
    {
        cores.tile_index = index;
        if (side == 0)
        {
            const PairTerms t = pair_terms(a, wbar, index * kTile + row, count);
            first[row] = t.live ? t.ab.x : -1;
            second[row] = t.ab.y;
            envelopes[row] = t.envelope;
            movings[row] = t.moving;
            offsets[row] = t.g.w / a.width;
            scales[row] = -t.rate / a.width;
        }
        __syncthreads();  // and the last tile's rows have left
        {
            const float t = offsets[row], scale = scales[row];
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                const int k0 = 32 * side + 8 * c;
                float g[8], gd[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                    const float u = t - static_cast<float>(k0 + e);
                    g[e] = k0 + e < a.gaussians ? gaussian(u) : 0.0f;
                    gd[e] = g[e] * u * scale;
                }
                *reinterpret_cast<uint4*>(row_word(tile, row, 4 * side + c)) = umma::pack8(g);
                *reinterpret_cast<uint4*>(row_word(tile_dot, row, 4 * side + c)) = umma::pack8(gd);
            }
        }
        cores.begin([&] { products(0, image_b1, false); });
        copy_rows(kRowG, index, a.gaussians < 64);
        if (!cores.finish(1))
        {
            break;
        }
        // s = ssp(z + b1) and s_dot = sigmoid(z + b1) z_dot.
#pragma unroll 1
        for (int half = 0; half < 2; ++half)
        {
            float z[16], zd[16];
            const int column = 32 * side + 16 * half;
            umma::load16(cores.tmem + column, z);
            umma::load16(cores.tmem + 64 + column, zd);
            umma::wait_loads();
#pragma unroll
            for (int c = 0; c < 2; ++c)
            {
                float s[8], sd[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                    const float x = z[8 * c + e] + bias1[column + 8 * c + e];
                    s[e] = softplus_shifted(x);
                    sd[e] = sigmoid(x) * zd[8 * c + e];
                }
                *reinterpret_cast<uint4*>(row_word(tile, row, column / 8 + c)) = umma::pack8(s);
                *reinterpret_cast<uint4*>(row_word(tile_dot, row, column / 8 + c)) = umma::pack8(sd);
            }
        }
        cores.begin([&] { products(128, image_b2, false); });
        copy_rows(kRowS, index, false);
        if (!cores.finish(2))
        {
            break;
        }
#pragma unroll 1
        for (int step = 0; step < 2; ++step)
        {
            // This lane's word of a feature row: columns 16 step + 4 lane of the first half, or
            // of the second half for lanes 4 .. 7.
            const int place = 8 * (lane / 4) + 4 * step + lane % 4;
            uint2 vb[4], vdb[4], mb[4], mdb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const std::int64_t word =
                    16 * static_cast<std::int64_t>(second[lane_row + i]) + place;
                vb[i] = __ldg(v + word);
                vdb[i] = __ldg(v_dot + word);
                mb[i] = __ldg(m_bar + word);
                mdb[i] = __ldg(m_dot_bar + word);
            }
            {
                float u[16], ud[16];
                const int column = 32 * side + 16 * step;
                umma::load16(cores.tmem + 128 + column, u);
                umma::load16(cores.tmem + 192 + column, ud);
                umma::wait_loads();
                const float envelope = envelopes[row], moving = movings[row];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                {
                    float f[4], fd[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                    {
                        const float raw_filter = u[4 * q + e] + bias2[column + 4 * q + e];
                        f[e] = raw_filter * envelope;
                        fd[e] = fmaf(ud[4 * q + e], envelope, raw_filter * moving);
                    }
                    const int at = row * 8 + ((4 * side + q) ^ (row & 7));
                    reinterpret_cast<float4*>(stage)[at] = make_float4(f[0], f[1], f[2], f[3]);
                    reinterpret_cast<float4*>(stage_dot)[at] = make_float4(fd[0], fd[1], fd[2], fd[3]);
                }
            }
            umma::fence_before_sync();
            __syncthreads();
            int key = first[lane_row];
            float4 va, vda, ma, mda;
            auto load_first = [&](int atom) {
                const std::int64_t word = 16 * static_cast<std::int64_t>(max(atom, 0)) + place;
                va = widen4(__ldg(v + word));
                vda = widen4(__ldg(v_dot + word));
                ma = widen4(__ldg(m_bar + word));
                mda = widen4(__ldg(m_dot_bar + word));
            };
            load_first(key);
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const int r = lane_row + i;
                const int atom = first[r];
                if (atom != key)
                {
                    key = atom;
                    load_first(atom);
                }
                const float envelope = envelopes[r], moving = movings[r];
                const float4 f = staged4(stage, r, lane), fd = staged4(stage_dot, r, lane);
                const float4 right_v = widen4(vb[i]), right_vd = widen4(vdb[i]);
                const float4 right_m = widen4(mb[i]), right_md = widen4(mdb[i]);
                const float4 fb = fma4(right_md, vda, fma4(mda, right_vd, fma4(ma, right_v, right_m * va)));
                const float4 fdb = fma4(mda, right_v, right_md * va);
                if (atom >= 0)
                {
                    const std::int64_t word = 16 * static_cast<std::int64_t>(second[r]) + place;
                    atomicAdd(vbar4 + word, fma4(f, ma, fd * mda));
                    atomicAdd(vdbar4 + word, f * mda);
                }
                restage4(stage, r, lane, fma4(f, right_m, fd * right_md));
                restage4(stage_dot, r, lane, f * right_md);
                const float4 udb = fdb * envelope;
                const float4 ub = fma4(fb, make_float4(envelope, envelope, envelope, envelope), fdb * moving);
                const int to = 8 * (place & 1);
                *reinterpret_cast<uint2*>(row_word(tile, r, place / 2) + to) =
                    make_uint2(pack2(ub.x, ub.y), pack2(ub.z, ub.w));
                *reinterpret_cast<uint2*>(row_word(tile_dot, r, place / 2) + to) =
                    make_uint2(pack2(udb.x, udb.y), pack2(udb.z, udb.w));
            }
            __syncthreads();
            // A warp sums 32 rows of one of the two stages: v_bar's or v_dot_bar's.
            add_runs(side == 0 ? stage : stage_dot, first, 32 * (threadIdx.x / 32 % 4),
                     (side == 0 ? a.v_bar : a.v_dot_bar) + 16 * step +
                         32 * (threadIdx.x % 32 / 16) + threadIdx.x % 16);
            __syncthreads();  // the stages are written again, or the tiles read
        }
        cores.begin([&] { products(128, image_b2, true); });
        copy_rows(kRowUBar, index, false);
        if (!cores.finish(3))
        {
            break;
        }
#pragma unroll 1
        for (int half = 0; half < 2; ++half)
        {
            float sb[16], sdb[16], z[16], zd[16];
            const int column = 32 * side + 16 * half;
            umma::load16(cores.tmem + 128 + column, sb);
            umma::load16(cores.tmem + 192 + column, sdb);
            umma::load16(cores.tmem + column, z);
            umma::load16(cores.tmem + 64 + column, zd);
            umma::wait_loads();
#pragma unroll
            for (int c = 0; c < 2; ++c)
            {
                float zb[8], zdb[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                {
                    const int i = 8 * c + e;
                    const float sg = sigmoid(z[i] + bias1[column + i]);
                    zb[e] = sb[i] * sg + sdb[i] * zd[i] * sg * (1.0f - sg);
                    zdb[e] = sdb[i] * sg;
                }
                *reinterpret_cast<uint4*>(row_word(tile, row, column / 8 + c)) = umma::pack8(zb);
                *reinterpret_cast<uint4*>(row_word(tile_dot, row, column / 8 + c)) = umma::pack8(zdb);
            }
        }
        umma::fence_before_sync();
        __syncthreads();
        copy_rows(kRowZBar, index, false);
    }
    cores.close(256);
}

// Rows [count, capacity) of the eight per-pair arrays set to zero, the pair count read from the
// workspace's counters, so sums over every row of an array equal sums over the pairs.
__global__ void zero_tail_kernel(uint4* rows, std::int64_t capacity, const int* counters)
{
    const std::int64_t count = *reinterpret_cast<const volatile int*>(counters);
    const std::int64_t words = (capacity - count) * 8;  // 16-byte words past the count, per array
    const std::int64_t stride = static_cast<std::int64_t>(gridDim.x) * blockDim.x;
    for (std::int64_t i = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x;
         i < 8 * words; i += stride)
    {
        const std::int64_t array = i / words;
        rows[(array * capacity + count) * 8 + i % words] = make_uint4(0u, 0u, 0u, 0u);
    }
}

}  // namespace
}  // namespace nd

extern "C" {

int nd_schnet_tangent(const nd_schnet_tangent_args* args, int32_t direction,
                      nd_stream_t stream_handle)
{
    using namespace nd;
    ND_REQUIRE(args != nullptr, "args is null");
    ND_REQUIRE(direction == 0 || direction == 1, "direction must be 0 (forward) or 1 (reverse)");
    const nd_schnet_tangent_args& s = *args;
    ND_REQUIRE(s.num_atoms >= 1 && s.num_atoms <= (int64_t{1} << 30), "num_atoms out of range");
    ND_REQUIRE(s.num_columns >= 0 && s.num_columns < (int64_t{1} << 31), "num_columns out of range");
    ND_REQUIRE(s.interactions >= 1 && s.interactions <= 64, "interactions out of range");
    ND_REQUIRE(s.block >= 0 && s.block < s.interactions, "block out of range");
    ND_REQUIRE(s.num_types >= 1, "num_types must be positive");
    ND_REQUIRE(s.gaussians >= 2 && s.gaussians <= 64, "gaussians must lie in [2, 64]");
    ND_REQUIRE(s.cutoff > 0.0, "cutoff must be positive");
    ND_REQUIRE(s.weights && s.workspace && s.force_adjoint && s.virial_adjoint && s.v && s.v_dot &&
                   s.status,
               "a required buffer is null");
    ND_REQUIRE(reinterpret_cast<std::uintptr_t>(s.workspace) % 256 == 0 &&
                   reinterpret_cast<std::uintptr_t>(s.weights) % 256 == 0,
               "weights and workspace must be 256-byte aligned");
    auto aligned16 = [](const void* pointer) {
        return reinterpret_cast<std::uintptr_t>(pointer) % 16 == 0;
    };
    ND_REQUIRE(aligned16(s.v) && aligned16(s.v_dot) && aligned16(s.m) && aligned16(s.m_dot) &&
                   aligned16(s.m_bar) && aligned16(s.m_dot_bar) && aligned16(s.v_bar) &&
                   aligned16(s.v_dot_bar),
               "feature rows must be 16-byte aligned");
    if (direction == 0)
    {
        ND_REQUIRE(s.m && s.m_dot, "the forward pass needs m and m_dot");
    }
    else
    {
        ND_REQUIRE(s.m_bar && s.m_dot_bar && s.v_bar && s.v_dot_bar && s.pair_rows,
                   "the reverse pass needs m_bar, m_dot_bar, v_bar, v_dot_bar and pair_rows");
        ND_REQUIRE(s.capacity >= s.num_columns, "capacity must be at least num_columns");
        ND_REQUIRE(reinterpret_cast<std::uintptr_t>(s.pair_rows) % 16 == 0,
                   "pair_rows must be 16-byte aligned");
    }
    cudaStream_t stream = static_cast<cudaStream_t>(stream_handle);
    const WeightLayout wl(s.interactions, s.num_types);
    const Workspace ws(s.num_atoms, s.num_columns, s.interactions);
    auto* weights = static_cast<const unsigned char*>(s.weights);
    auto* base = static_cast<unsigned char*>(s.workspace);

    TangentPass pass{};
    pass.pairs = reinterpret_cast<const int2*>(base + ws.pairs);
    pass.geometry = reinterpret_cast<const float4*>(base + ws.geometry);
    pass.counters = reinterpret_cast<int*>(base + ws.counters);
    pass.images = weights + static_cast<std::int64_t>(s.block) * kImagesPerBlock * umma::kImageBytes;
    pass.b1 = reinterpret_cast<const float*>(weights + wl.vectors + (static_cast<std::int64_t>(s.block) * 4) * kFeatures * 4);
    pass.b2 = reinterpret_cast<const float*>(weights + wl.vectors + (static_cast<std::int64_t>(s.block) * 4 + 1) * kFeatures * 4);
    pass.force_adjoint = s.force_adjoint;
    pass.virial_adjoint = s.virial_adjoint;
    pass.v = static_cast<const uint4*>(s.v);
    pass.v_dot = static_cast<const uint4*>(s.v_dot);
    pass.m = s.m;
    pass.m_dot = s.m_dot;
    pass.m_bar = static_cast<const uint4*>(s.m_bar);
    pass.m_dot_bar = static_cast<const uint4*>(s.m_dot_bar);
    pass.v_bar = s.v_bar;
    pass.v_dot_bar = s.v_dot_bar;
    pass.rows = static_cast<uint4*>(s.pair_rows);
    pass.capacity = s.capacity;
    pass.width = static_cast<float>(s.cutoff / (s.gaussians - 1));
    pass.phase = static_cast<float>(3.14159265358979323846 / s.cutoff);
    pass.gaussians = s.gaussians;

    // The kernels' attributes, set once per device (they belong to its instance of a kernel).
    static DeviceOnce configured;  // per device, retried after a failure
    ND_CUDA_TRY(configured.run([] {
        cudaError_t rc = cudaFuncSetAttribute(tangent_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTangentForwardShared);
        auto then = [&rc](cudaError_t next) { rc = rc != cudaSuccess ? rc : next; };
        then(cudaFuncSetAttribute(tangent_reverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTangentReverseShared));
        then(cudaFuncSetAttribute(tangent_forward_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        then(cudaFuncSetAttribute(tangent_reverse_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        return rc;
    }));
    if (direction == 0)
    {
        // The messages m are the E/F/W call's for this block; only their tangent is computed.
        const std::int64_t row_bytes = align256(s.num_atoms * kFeatures * 4);
        ND_CUDA_TRY(cudaMemcpyAsync(s.m, base + ws.m + s.block * row_bytes,
                                    s.num_atoms * kFeatures * sizeof(float),
                                    cudaMemcpyDeviceToDevice, stream));
        const int grid = pair_grid(reinterpret_cast<const void*>(tangent_forward_kernel), kTangentForwardShared, 128);
        tangent_forward_kernel<<<grid, kTile, kTangentForwardShared, stream>>>(pass);
    }
    else
    {
        const int grid = pair_grid(reinterpret_cast<const void*>(tangent_reverse_kernel), kTangentReverseShared, 256, kReverseThreads);
        tangent_reverse_kernel<<<grid, kReverseThreads, kTangentReverseShared, stream>>>(pass);
        ND_LAUNCH_CHECK();
        zero_tail_kernel<<<std::min<std::int64_t>(1184, blocks_for(s.capacity * 8)), kThreads, 0, stream>>>(
            pass.rows, s.capacity, pass.counters);
    }
    ND_LAUNCH_CHECK();
    ND_CUDA_TRY(cudaMemcpyAsync(s.status, pass.counters, 4 * sizeof(int), cudaMemcpyDeviceToDevice, stream));
    return ND_OK;
}

}  // extern "C"
