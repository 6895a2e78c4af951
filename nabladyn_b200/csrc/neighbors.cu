// The neighbor operator: a cell-list half list of the pairs closer than the list radius,
// with the on-GPU skin-reuse check, behind the C-ABI of include/nabladyn_b200.h.
//
// The contract is the reference's (src/nabladyn/neighbors/csrc/ops.h:12-89,
// runtime/entry_points.cu:284-508): the same 15 buffers, the same status bits, the same pair
// set (each pair once, listed from the atom earlier in bin order), pair columns grouped by that
// atom from its offset in the scan of the counts, padding column k = (k mod N, k mod N), and
// every rebuild kernel gated by a device flag so one CUDA Graph holds a whole update. Two
// rules decide the pair set bit for bit and are kept: the grid (bins of width L / n_a, atoms
// ordered by bin, then by id) and the rounding of a displacement and its square (one rounding
// per difference, r^2 = fma(dz, dz, fma(dx, dx, dy * dy))).
//
// How the GPU builds it is this file's own design:
//   * binning takes each atom's in-bin slot from the counting atomic, and one warp per bin
//     orders the bin by id with shuffles while gathering the sorted positions;
//   * the pairs are built per HOME BIN, one CTA each. Every candidate of a home bin's atoms
//     sits in the home bin itself (after the atom) or in a stencil bin that comes later in bin
//     order; the CTA stages exactly those bins into shared memory as (x, y, z, id) slots, each
//     bin's coordinates already moved by its image where the move is exact, tests each staged
//     candidate against 32 of the bin's atoms at a time into words of hit bits, and either
//     counts the bits or turns them into columns in shared memory that leave in whole lines;
//   * small boxes (at most three bins per axis) keep a word-major bit matrix: one thread per
//     (center, 32-candidate word) with the word's candidates staged in shared memory, so
//     threads of a block store consecutive words;
//   * the update opens with one warp that checks the cell and sets the grid and the reuse
//     threshold, checks reuse with one atomic per warp, and commits the new reference frame
//     inside the fill; the scans are our own gated kernels (scan.cuh), so an update that
//     reuses its pairs runs no scan; the pair total and the padding share one launch.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <limits>

#include "common.cuh"
#include "geometry.cuh"
#include "scan.cuh"

namespace nd {

// A staged candidate: coordinates in the list's dtype and the atom id in the fourth word.
template <typename T>
struct alignas(4 * sizeof(T)) Slot
{
    T x, y, z, w;
};

__device__ __forceinline__ float id_word(float, index_t id) { return __int_as_float(id); }
__device__ __forceinline__ double id_word(double, index_t id)
{
    return __longlong_as_double(static_cast<long long>(id));
}
__device__ __forceinline__ index_t word_id(float w) { return __float_as_int(w); }
__device__ __forceinline__ index_t word_id(double w)
{
    return static_cast<index_t>(__double_as_longlong(w));
}

// ---------------------------------------------------------------------------------------
// Grid: counting sort of the atoms by bin, ordered by atom id inside each bin.

// Bins each atom and takes its slot in the bin from the counting atomic. The slots are parked
// in `slots` (the pair_counts buffer, rewritten by the count that follows).
template <typename T>
__global__ void bin_atoms_kernel(
    const T* __restrict__ positions,
    const index_t* __restrict__ dims,
    const T* __restrict__ widths,
    index_t num_atoms,
    index_t* __restrict__ atom_bin,
    index_t* __restrict__ bin_counts,
    index_t* __restrict__ slots,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status
)
{
    const std::int64_t atom = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (atom >= num_atoms || !rebuilding(rebuild, status))
    {
        return;
    }
    const T* p = positions + 3 * atom;
    const index_t nx = dims[0], ny = dims[1], nz = dims[2];
    const index_t bin = axis_bin(p[0], widths[0], nx) +
                        nx * (axis_bin(p[1], widths[1], ny) + ny * axis_bin(p[2], widths[2], nz));
    atom_bin[atom] = bin;
    slots[atom] = atomicAdd(bin_counts + bin, 1);
}

// Places each atom at its bin's offset plus its slot and returns the counts to zero for the
// next build.
__global__ void place_atoms_kernel(
    const index_t* __restrict__ atom_bin,
    const index_t* __restrict__ slots,
    const index_t* __restrict__ bin_offsets,
    index_t num_atoms,
    index_t* __restrict__ bin_counts,
    index_t* __restrict__ unordered_ids,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status
)
{
    const std::int64_t atom = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (atom >= num_atoms || !rebuilding(rebuild, status))
    {
        return;
    }
    const index_t bin = atom_bin[atom];
    unordered_ids[bin_offsets[bin] + slots[atom]] = static_cast<index_t>(atom);
    bin_counts[bin] = 0;
}

// One warp per bin: each atom's rank is the number of smaller ids in its bin, counted with
// shuffles; the warp writes the sorted ids and gathers the sorted positions.
template <typename T>
__global__ void order_bins_kernel(
    const T* __restrict__ positions,
    const index_t* __restrict__ unordered_ids,
    const index_t* __restrict__ bin_offsets,
    std::int64_t num_bins,
    index_t* __restrict__ sorted_ids,
    T* __restrict__ sorted_positions,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status
)
{
    const std::int64_t bin =
        (static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / kWarp;
    const int lane = threadIdx.x % kWarp;
    if (bin >= num_bins || !rebuilding(rebuild, status))
    {
        return;  // whole warps return together
    }
    const index_t begin = bin_offsets[bin];
    const index_t count = bin_offsets[bin + 1] - begin;
    for (index_t mine = 0; mine < count; mine += kWarp)
    {
        const bool active = mine + lane < count;
        const index_t id = active ? unordered_ids[begin + mine + lane] : 0;
        index_t rank = 0;
        for (index_t base = 0; base < count; base += kWarp)
        {
            const index_t other =
                base + lane < count ? unordered_ids[begin + base + lane] : 0x7fffffff;
            const int valid = count - base < kWarp ? count - base : kWarp;
            for (int s = 0; s < valid; ++s)
            {
                rank += __shfl_sync(kFullMask, other, s) < id;
            }
        }
        if (active)
        {
            const index_t slot = begin + rank;
            sorted_ids[slot] = id;
            sorted_positions[3LL * slot] = positions[3LL * id];
            sorted_positions[3LL * slot + 1] = positions[3LL * id + 1];
            sorted_positions[3LL * slot + 2] = positions[3LL * id + 2];
        }
    }
}

// ---------------------------------------------------------------------------------------
// Pairs on the grid path: one CTA per home bin.
//
// What bounds a build is the distance tests (about 410 candidates for each of a bin's 30 atoms
// in a liquid, 15 % of them hits) and, in the fill, the appends. So a candidate is read once
// from shared memory for 32 centers: a lane holds two centers, the two halves of a warp take
// alternate words of 32 candidates, and in float32 the two centers are the halves of packed
// f32x2 instructions whose sign bits a funnel shift collects. The four warps share a bin's
// words, so the few bins of a small system still fill a CTA, and the hits of a word are
// appended by a thread of their own: a center's words find their columns by a 16-lane scan.
// A bin's columns are one contiguous range, so entries go to shared memory first and leave in
// whole lines. 1,048,576 atoms, float32, the whole update: 1,710 us with a warp per home bin and
// appends by the centers' lanes, 903 us so (count 216, fill with the padding 537: issue 73 and
// 78 % busy). Without the padding the fill took 519; a warp per center with a lane per candidate
// (ranks by popcounts) took 575, ten or twelve CTAs per SM (48 or 40 registers, spilling) 545 and
// 528 us.

// Threads per CTA: four warps share a bin's words where the bins fill the GPU (7 CTAs per SM);
// with at most two bins per SM eight warps shorten the one wave there is (64 bins of a
// 2,003-atom float64 frame: count 16 -> 12 us, fill 35 -> 25 us).
constexpr int kHoodThreads = 128;
constexpr int kHoodFewThreads = 256;
constexpr std::int64_t kHoodFewBins = 2 * 148;
// Where bins outnumber atoms most are empty, and a CTA that finds so costs what the bin's pairs
// would: a CTA then takes up to 32 bins (kManyCtas of them keep the GPU full; 100,000 atoms among
// 27 million bins, update: 31.8 ms with a bin per CTA, 3.4 ms). In a gas also the bins with atoms
// hold few, so a warp takes one by itself (0.7 atoms a bin, float64: 952 us, 586; 2.9 atoms a bin:
// 461, 349). By the columns, because a droplet in a large box has as many empty bins but full ones
// too, which want four warps (100,000 atoms of a liquid among 46,000 bins: 227 us, with a warp per
// bin 690).
constexpr std::int64_t kManyCtas = 148 * 32;
constexpr std::int64_t kGasBins = 4;      // a bin for at most four atoms
constexpr std::int64_t kGasColumns = 12;  // columns per atom at most
constexpr int kHoodBins = 27;      // the home bin and its stencil, at most
// Candidates staged at once (a liquid needs about 410), and pairs of 32 centers (2,000); few for
// the one-warp CTAs of sparse bins, of which an SM then holds 32.
constexpr int kHoodSlots = 512;
constexpr int kHoodEntries = 3072;
constexpr int kSparseSlots = 128;
constexpr int kSparseEntries = 512;

// The part of a home bin's stencil that holds candidates: the home bin (its atoms after the
// center) and each stencil bin that comes later in bin order (all its atoms). With three or
// more bins per axis each bin has a fixed image: `ahead` marks the axes on which the bin lies
// past the upper face, where the center moves by -L (the rounding of center - L, then of the
// difference), `behind` those on which it lies past the lower face, where the candidate moves
// by -L when staged. Otherwise every candidate takes the minimum image per axis.
struct Hood
{
    int count;                    // bins kept, the home bin first
    int total;                    // candidates in them
    int first[kHoodBins];         // sorted index of each bin's first atom
    int size[kHoodBins];          // atoms per bin
    int slot[kHoodBins + 1];      // first slot of each bin in the staged list
    unsigned char ahead[kHoodBins];
    unsigned char behind[kHoodBins];
    int any_ahead;
};

// One warp lists the home bin's stencil. Lane s takes stencil bin s; the kept bins follow the
// home bin in stencil order, placed by a ballot.
__device__ __forceinline__ void plan_hood(
    Hood& hood,
    index_t home,
    const index_t* __restrict__ dims,
    const index_t* __restrict__ bin_offsets,
    bool fixed_images
)
{
    const int lane = threadIdx.x % kWarp;
    const index_t n[3] = {dims[0], dims[1], dims[2]};
    const index_t h[3] = {home % n[0], (home / n[0]) % n[1], home / (n[0] * n[1])};
    // Stencil bins per axis: three around home, or the whole axis when it has fewer bins.
    int span[3];
    for (int a = 0; a < 3; ++a)
    {
        span[a] = n[a] >= 3 ? 3 : n[a];
    }
    bool keep = false;
    index_t bin = 0;
    unsigned ahead = 0, behind = 0;
    if (lane < span[0] * span[1] * span[2])
    {
        const int s[3] = {lane % span[0], (lane / span[0]) % span[1], lane / (span[0] * span[1])};
        index_t b[3];
        for (int a = 0; a < 3; ++a)
        {
            if (n[a] >= 3)
            {
                const index_t raw = h[a] + s[a] - 1;
                b[a] = raw < 0 ? raw + n[a] : (raw >= n[a] ? raw - n[a] : raw);
                if (fixed_images)
                {
                    ahead |= raw >= n[a] ? 1u << a : 0u;
                    behind |= raw < 0 ? 1u << a : 0u;
                }
            }
            else
            {
                b[a] = s[a];
            }
        }
        bin = b[0] + n[0] * (b[1] + n[1] * b[2]);
        keep = bin > home;
    }
    const unsigned kept = __ballot_sync(kFullMask, keep);
    const unsigned ahead_lanes = __ballot_sync(kFullMask, keep && ahead != 0);
    const int count = 1 + __popc(kept);
    if (keep)
    {
        const int at = 1 + __popc(kept & ((1u << lane) - 1u));
        const index_t begin = bin_offsets[bin];
        hood.first[at] = begin;
        hood.size[at] = bin_offsets[bin + 1] - begin;
        hood.ahead[at] = static_cast<unsigned char>(ahead);
        hood.behind[at] = static_cast<unsigned char>(behind);
    }
    if (lane == 0)
    {
        const index_t begin = bin_offsets[home];
        hood.first[0] = begin;
        hood.size[0] = bin_offsets[home + 1] - begin;
        hood.ahead[0] = 0;
        hood.behind[0] = 0;
        hood.count = count;
        hood.any_ahead = ahead_lanes != 0;
    }
    __syncwarp();
    // Slots: an exclusive scan of the kept bins' sizes, in their order.
    const int value = lane < count ? hood.size[lane] : 0;
    int inclusive = value;
#pragma unroll
    for (int offset = 1; offset < kWarp; offset *= 2)
    {
        const int up = __shfl_up_sync(kFullMask, inclusive, offset);
        inclusive += lane >= offset ? up : 0;
    }
    if (lane < count)
    {
        hood.slot[lane] = inclusive - value;
    }
    if (lane == count - 1)
    {
        hood.slot[count] = inclusive;
        hood.total = inclusive;
    }
    __syncwarp();
}

// Candidate `k` of kept bin `g`, in the list's arithmetic: the coordinate moved by -L on the
// axes where the bin lies past the lower face (an exact move), and the atom id.
template <typename T>
__device__ __forceinline__ Slot<T> hood_candidate(
    const Hood& hood, int g, int k,
    const T* __restrict__ sorted_positions,
    const index_t* __restrict__ sorted_ids,
    T lx, T ly, T lz
)
{
    const std::int64_t atom = hood.first[g] + k;
    const T* p = sorted_positions + 3 * atom;
    const unsigned behind = hood.behind[g];
    Slot<T> out;
    out.x = (behind & 1u) ? p[0] + (-lx) : p[0];
    out.y = (behind & 2u) ? p[1] + (-ly) : p[1];
    out.z = (behind & 4u) ? p[2] + (-lz) : p[2];
    out.w = id_word(T(0), sorted_ids[atom]);
    return out;
}

// How a home bin's displacements are taken (one choice per CTA).
enum HoodImages : int
{
    kPlain,    // fixed images, no kept bin past an upper face: center - candidate
    kAhead,    // fixed images: the center moves by -L towards bins past an upper face
    kMinimum,  // an axis of fewer than three bins: the minimum image per candidate
};

// A lane's two centers. For kAhead also the centers moved by -L, rounded once.
template <typename T>
struct CenterPair
{
    T x0, y0, z0, x1, y1, z1;
};

// Shifts into the bits of two centers from the right: set when the candidate lies closer than
// the radius (r^2 - R^2 is negative exactly when r^2 < R^2).
template <typename T>
__device__ __forceinline__ void shift_in_hits(T x0, T y0, T z0, T x1, T y1, T z1,
                                              const Slot<T>& p, T radius_squared,
                                              unsigned& bits0, unsigned& bits1)
{
    const T r0 = squared_norm(x0 - p.x, y0 - p.y, z0 - p.z);
    const T r1 = squared_norm(x1 - p.x, y1 - p.y, z1 - p.z);
    bits0 = (bits0 << 1) | static_cast<unsigned>(r0 < radius_squared);
    bits1 = (bits1 << 1) | static_cast<unsigned>(r1 < radius_squared);
}

// The two centers as the halves of packed f32x2 instructions: each half rounds as the scalar
// test, p - x being the exact negative of x - p.
__device__ __forceinline__ void shift_in_hits(float x0, float y0, float z0, float x1, float y1,
                                              float z1, const Slot<float>& p,
                                              float radius_squared, unsigned& bits0,
                                              unsigned& bits1)
{
    const float2 dx = __fadd2_rn(make_float2(p.x, p.x), make_float2(-x0, -x1));
    const float2 dy = __fadd2_rn(make_float2(p.y, p.y), make_float2(-y0, -y1));
    const float2 dz = __fadd2_rn(make_float2(p.z, p.z), make_float2(-z0, -z1));
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
    const float2 d = __fadd2_rn(r2, make_float2(-radius_squared, -radius_squared));
    bits0 = __funnelshift_l(__float_as_uint(d.x), bits0, 1);
    bits1 = __funnelshift_l(__float_as_uint(d.y), bits1, 1);
}

// The hits of a lane's two centers among the 32 staged candidates from slot `base`: bit 31 - j
// for candidate base + j, so the first candidate is the highest bit (one instruction finds it).
// Of the warp's last words the first `groups` groups of eight candidates are tested.
constexpr int kHoodGroup = 8;

template <typename T, int kImages>
__device__ __forceinline__ void hit_words(
    const Slot<T>* __restrict__ staged, const unsigned char* __restrict__ ahead, int base,
    int groups, const CenterPair<T>& c, T lx, T ly, T lz, T radius_squared, unsigned& hits0,
    unsigned& hits1)
{
    hits0 = hits1 = 0;
#pragma unroll 8
    for (int j = 0; j < kHoodGroup * groups; ++j)
    {
        const Slot<T> p = staged[base + j];
        if (kImages == kMinimum)
        {
            const T r0 = squared_norm(min_image(c.x0, p.x, lx), min_image(c.y0, p.y, ly),
                                      min_image(c.z0, p.z, lz));
            const T r1 = squared_norm(min_image(c.x1, p.x, lx), min_image(c.y1, p.y, ly),
                                      min_image(c.z1, p.z, lz));
            hits0 = (hits0 << 1) | static_cast<unsigned>(r0 < radius_squared);
            hits1 = (hits1 << 1) | static_cast<unsigned>(r1 < radius_squared);
        }
        else if (kImages == kAhead)
        {
            const unsigned moved = ahead[base + j];
            const T sx = (moved & 1u) ? lx : T(0), sy = (moved & 2u) ? ly : T(0),
                    sz = (moved & 4u) ? lz : T(0);
            shift_in_hits(c.x0 - sx, c.y0 - sy, c.z0 - sz, c.x1 - sx, c.y1 - sy, c.z1 - sz, p,
                          radius_squared, hits0, hits1);
        }
        else
        {
            shift_in_hits(c.x0, c.y0, c.z0, c.x1, c.y1, c.z1, p, radius_squared, hits0, hits1);
        }
    }
    hits0 <<= kWarp - kHoodGroup * groups;
    hits1 <<= kWarp - kHoodGroup * groups;
}

// Bits of a word from slot `first` on whose candidates come after center `h` (slots and
// centers count from the home bin's first atom) and before slot `end`.
__device__ __forceinline__ unsigned word_mask(int first, int h, int end)
{
    const int above = h + 1 - first, size = end - first;
    const unsigned after = above <= 0 ? ~0u : (above >= kWarp ? 0u : ~0u >> above);
    const unsigned before = size >= kWarp ? ~0u : (size <= 0 ? 0u : ~(~0u >> size));
    return after & before;
}

// Takes the first candidate's position out of a word.
__device__ __forceinline__ int next_hit(unsigned& hits)
{
    const int j = __clz(static_cast<int>(hits));
    hits &= ~(0x80000000u >> j);
    return j;
}

// Pads the columns from the total on, by `threads` threads: column k holds the self-pair
// (k mod N, k mod N), spreading their zero gradients over the atoms; the threads start at the
// total and step together, so each takes one remainder and the stores are whole lines.
__device__ __forceinline__ void pad_columns(index_t total, index_t num_atoms, index_t capacity,
                                            index_t* __restrict__ pairs, unsigned thread,
                                            unsigned threads)
{
    if (total >= capacity)
    {
        return;
    }
    const unsigned n = static_cast<unsigned>(num_atoms);
    const unsigned end = static_cast<unsigned>(capacity);
    const unsigned step = threads % n;
    unsigned column = static_cast<unsigned>(total) + thread;  // below 2^32: the grid is bounded
    unsigned atom = column % n;
    for (; column < end; column += threads)
    {
        pairs[column] = static_cast<index_t>(atom);
        pairs[static_cast<std::int64_t>(capacity) + column] = static_cast<index_t>(atom);
        atom += step;
        atom -= atom >= n ? n : 0u;
    }
}

// Counts (kFill false) or writes (kFill true) the pairs of one home bin. The fill of an update
// also stores the frame it was built from, each CTA its home atoms' positions.
//
// The candidates, home bin first, are staged kHoodSlots at a time (once, in all but very dense
// bins) and tested against the bin's atoms 32 at a time.
template <typename T, bool kFill, int kThreadCount>
__device__ __forceinline__ void hood_bin(
    index_t home,
    const T* __restrict__ sorted_positions,
    const index_t* __restrict__ sorted_ids,
    const index_t* __restrict__ bin_offsets,
    const index_t* __restrict__ dims,
    const T* __restrict__ cell,
    T radius_squared,
    index_t* __restrict__ pair_counts,
    const index_t* __restrict__ pair_offsets,
    index_t capacity,
    index_t* __restrict__ pairs,
    const T* __restrict__ positions,
    T* __restrict__ reference_positions
)
{
    constexpr bool kSparse = kThreadCount == kWarp;
    constexpr int kSlots = kSparse ? kSparseSlots : kHoodSlots, kWords = kSlots / kWarp;
    constexpr int kEntries = kSparse ? kSparseEntries : kHoodEntries;
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const index_t begin = bin_offsets[home];
    const int homes = bin_offsets[home + 1] - begin;
    if (kFill && reference_positions != nullptr)
    {
        for (int k = threadIdx.x; k < 3 * homes; k += kThreadCount)
        {
            const std::int64_t id = sorted_ids[begin + k / 3];
            reference_positions[3 * id + k % 3] = positions[3 * id + k % 3];
        }
    }
    if (homes == 0)
    {
        return;  // the whole CTA
    }
    __shared__ Hood hood;
    __shared__ Slot<T> staged[kSlots];
    __shared__ unsigned char ahead[kSlots];
    __shared__ unsigned words[kFill ? kWords : 1][kWarp + 1];  // one center apart: no conflicts
    __shared__ std::uint16_t entries[kFill ? kEntries : 1];    // center << 9 | slot
    __shared__ int cursors[kWarp];                                 // fill: each center's next column
    __shared__ int warp_counts[kThreadCount / kWarp][kWarp];
    const T lx = cell[0], ly = cell[1], lz = cell[2];
    const bool fixed = dims[0] >= 3 && dims[1] >= 3 && dims[2] >= 3;
    if (warp == 0)
    {
        plan_hood(hood, home, dims, bin_offsets, fixed);
    }
    __syncthreads();
    const int images = !fixed ? kMinimum : (hood.any_ahead ? kAhead : kPlain);
    const int total = hood.total;
    const bool once = total <= kSlots;
    const int half = lane / 16, q = lane % 16;
    for (int group = 0; group < homes; group += kWarp)
    {
        const int centers = homes - group < kWarp ? homes - group : kWarp;
        const int h0 = group + 2 * q, h1 = h0 + 1;
        CenterPair<T> c;
        {
            const T* p0 = sorted_positions + 3LL * (begin + (h0 < homes ? h0 : group));
            const T* p1 = sorted_positions + 3LL * (begin + (h1 < homes ? h1 : group));
            c = {p0[0], p0[1], p0[2], p1[0], p1[1], p1[2]};
        }
        int count0 = 0, count1 = 0;
        index_t region = 0;
        int region_size = 0;
        if (kFill)
        {
            // The group's columns are one range: its centers follow one another.
            region = pair_offsets[begin + group];
            const index_t last = begin + group + centers - 1;
            region_size = pair_offsets[last] + pair_counts[last] - region;
            if (threadIdx.x < centers)
            {
                cursors[threadIdx.x] = pair_offsets[begin + group + threadIdx.x];
            }
        }
        const bool packed = kFill && once && region_size <= kEntries;
        for (int chunk = 0; chunk < total; chunk += kSlots)
        {
            const int size = total - chunk < kSlots ? total - chunk : kSlots;
            if (group == 0 || !once)
            {
                __syncthreads();  // the last chunk's readers are done
                for (int g = warp; g < hood.count; g += kThreadCount / kWarp)
                {
                    const int from = hood.slot[g] - chunk;  // the bin's first slot
                    int k = lane;
                    if (from < 0)
                    {
                        k += -from / kWarp * kWarp;
                    }
                    for (; k < hood.size[g] && from + k < size; k += kWarp)
                    {
                        if (from + k >= 0)
                        {
                            staged[from + k] = hood_candidate(hood, g, k, sorted_positions,
                                                              sorted_ids, lx, ly, lz);
                            ahead[from + k] = hood.ahead[g];
                        }
                    }
                }
                __syncthreads();
            }
            const int used = (size + kWarp - 1) / kWarp;
            for (int pair = warp; 2 * pair < used; pair += kThreadCount / kWarp)
            {
                const int w = 2 * pair + half;  // at most kWords - 1
                // Of a sparse bin's few candidates the groups there are; a liquid's words are full.
                const int left = size - 2 * kWarp * pair;  // of the first half's word on
                const int groups = kSparse ? min(kWarp, left + kHoodGroup - 1) / kHoodGroup
                                           : kWarp / kHoodGroup;
                unsigned hits0, hits1;
                if (images == kPlain)
                {
                    hit_words<T, kPlain>(staged, ahead, kWarp * w, groups, c, lx, ly, lz,
                                         radius_squared, hits0, hits1);
                }
                else if (images == kAhead)
                {
                    hit_words<T, kAhead>(staged, ahead, kWarp * w, groups, c, lx, ly, lz,
                                         radius_squared, hits0, hits1);
                }
                else
                {
                    hit_words<T, kMinimum>(staged, ahead, kWarp * w, groups, c, lx, ly, lz,
                                           radius_squared, hits0, hits1);
                }
                const int slot = chunk + kWarp * w;
                hits0 &= h0 < homes ? word_mask(slot, h0, chunk + size) : 0u;
                hits1 &= h1 < homes ? word_mask(slot, h1, chunk + size) : 0u;
                if (kFill)
                {
                    words[w][2 * q] = hits0;
                    words[w][2 * q + 1] = hits1;
                }
                else
                {
                    count0 += __popc(hits0);
                    count1 += __popc(hits1);
                }
            }
            if (!kFill)
            {
                continue;
            }
            __syncthreads();
            // A lane per (center, word): its hits follow those of the center's earlier words.
            for (int pair = warp; 2 * pair < centers; pair += kThreadCount / kWarp)
            {
                const int center = 2 * pair + half, w = q;
                unsigned hits = center < centers && w < used ? words[w][center] : 0u;
                const int count = __popc(hits);
                int inclusive = count;
#pragma unroll
                for (int offset = 1; offset < 16; offset *= 2)
                {
                    const int up = __shfl_up_sync(kFullMask, inclusive, offset, 16);
                    inclusive += w >= offset ? up : 0;
                }
                index_t column = (center < centers ? cursors[center] : 0) + inclusive - count;
                __syncwarp();
                if (w == 15 && center < centers)
                {
                    cursors[center] += inclusive;
                }
                if (packed)
                {
                    int at = column - region;
                    const int tag = center << 9 | (kWarp * w);
                    while (hits != 0)
                    {
                        const int j = next_hit(hits);
                        if (static_cast<unsigned>(at) < static_cast<unsigned>(kEntries))
                        {
                            entries[at] = static_cast<std::uint16_t>(tag + j);
                        }
                        ++at;
                    }
                }
                else
                {
                    const index_t id = hits != 0 ? sorted_ids[begin + group + center] : 0;
                    while (hits != 0)
                    {
                        const int j = next_hit(hits);
                        if (static_cast<unsigned>(column) < static_cast<unsigned>(capacity))
                        {
                            pairs[column] = id;
                            pairs[static_cast<std::int64_t>(capacity) + column] =
                                word_id(staged[kWarp * w + j].w);
                        }
                        ++column;
                    }
                }
            }
            __syncthreads();
            if (packed)
            {
                for (int e = threadIdx.x; e < region_size; e += kThreadCount)
                {
                    const index_t column = region + e;
                    const unsigned entry = entries[e];
                    if (static_cast<unsigned>(column) < static_cast<unsigned>(capacity))
                    {
                        pairs[column] = word_id(staged[group + (entry >> 9)].w);
                        pairs[static_cast<std::int64_t>(capacity) + column] =
                            word_id(staged[entry & 511u].w);
                    }
                }
            }
        }
        if (!kFill)
        {
            count0 += __shfl_xor_sync(kFullMask, count0, 16);
            count1 += __shfl_xor_sync(kFullMask, count1, 16);
            if (half == 0)
            {
                warp_counts[warp][2 * q] = count0;
                warp_counts[warp][2 * q + 1] = count1;
            }
            __syncthreads();
            if (threadIdx.x < centers)
            {
                index_t sum = 0;
#pragma unroll
                for (int w = 0; w < kThreadCount / kWarp; ++w)
                {
                    sum += warp_counts[w][threadIdx.x];
                }
                pair_counts[begin + group + threadIdx.x] = sum;
            }
        }
        __syncthreads();  // the next group's cursors, words and counts
    }
}

// A home bin per CTA, or with kMany up to 32 bins, of which it takes those with atoms. An
// update's fill stores the cell and the rebuild count in its first bin's CTA. The fill's first
// `pad_ctas` CTAs write the padding columns instead: those stores are bound by memory and the fill
// by instruction issue, so one hides the other (1,048,576 atoms, update: fill 519 us and padding
// after it 73 us, together 537 us).
template <typename T, bool kFill, int kThreadCount, bool kMany>
__global__ void __launch_bounds__(kThreadCount) hood_pairs_kernel(
    const T* __restrict__ sorted_positions,
    const index_t* __restrict__ sorted_ids,
    const index_t* __restrict__ bin_offsets,
    const index_t* __restrict__ dims,
    const T* __restrict__ cell,
    T radius_squared,
    index_t* __restrict__ pair_counts,
    const index_t* __restrict__ pair_offsets,
    index_t capacity,
    index_t* __restrict__ pairs,
    const T* __restrict__ positions,
    T* __restrict__ reference_positions,
    T* __restrict__ reference_cell,
    index_t* __restrict__ rebuild_count,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status,
    index_t num_atoms,
    int pad_ctas,
    index_t num_bins
)
{
    if (!rebuilding(rebuild, status))
    {
        return;
    }
    if (kFill && static_cast<int>(blockIdx.x) < pad_ctas)
    {
        pad_columns(pair_offsets[num_atoms - 1] + pair_counts[num_atoms - 1], num_atoms, capacity,
                    pairs, blockIdx.x * kThreadCount + threadIdx.x, pad_ctas * kThreadCount);
        return;
    }
    const index_t cta = static_cast<index_t>(blockIdx.x) - (kFill ? pad_ctas : 0);
    if (kFill && reference_positions != nullptr && cta == 0)
    {
        if (threadIdx.x < 3)
        {
            reference_cell[threadIdx.x] = cell[threadIdx.x];
        }
        if (threadIdx.x == 0)
        {
            ++rebuild_count[0];
        }
    }
    if (!kMany)
    {
        hood_bin<T, kFill, kThreadCount>(cta, sorted_positions, sorted_ids, bin_offsets, dims, cell,
                                         radius_squared, pair_counts, pair_offsets, capacity,
                                         pairs, positions, reference_positions);
        return;
    }
    // A CTA's bins lie `ctas` apart, so the bins of a droplet go to many CTAs.
    const std::int64_t ctas = gridDim.x - (kFill ? pad_ctas : 0);
    const std::int64_t mine = cta + ctas * static_cast<std::int64_t>(threadIdx.x % kWarp);
    const bool some = mine < num_bins && bin_offsets[mine] != bin_offsets[mine + 1];
    for (unsigned bins = __ballot_sync(kFullMask, some); bins != 0; bins &= bins - 1)
    {
        const auto home = static_cast<index_t>(cta + ctas * (__ffs(static_cast<int>(bins)) - 1));
        hood_bin<T, kFill, kThreadCount>(home, sorted_positions, sorted_ids, bin_offsets, dims,
                                         cell, radius_squared, pair_counts, pair_offsets, capacity,
                                         pairs, positions, reference_positions);
    }
}

// ---------------------------------------------------------------------------------------
// The all-pairs path, for lists whose first grid has at most three bins on every axis.
//
// The hits live in a word-major bit matrix: word w of atom i, bits[w * N + i], holds bit b for
// atom 32 w + b, set when that atom comes after i and lies closer than the radius (minimum
// image per axis). Words that hold no atom after i are never written nor read.

__host__ __device__ __forceinline__ std::int64_t bit_words(std::int64_t num_atoms)
{
    return (num_atoms + kWarp - 1) / kWarp;
}

constexpr int kWordThreads = 128;

// Grid (centers / 128, words): the block stages word w's 32 candidates in shared memory and
// each thread builds one center's word from them.
template <typename T>
__global__ void __launch_bounds__(kWordThreads) pair_words_kernel(
    const T* __restrict__ positions,
    const T* __restrict__ cell,
    T radius_squared,
    index_t num_atoms,
    std::uint32_t* __restrict__ bits,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status
)
{
    const std::int64_t word = blockIdx.y;
    const std::int64_t first_center = static_cast<std::int64_t>(blockIdx.x) * kWordThreads;
    if (first_center >= 32 * (word + 1) - 1 || !rebuilding(rebuild, status))
    {
        return;  // every center of the block comes at or after the word's last atom
    }
    __shared__ T candidates[3][kWarp];
    if (threadIdx.x < kWarp)
    {
        const std::int64_t j = 32 * word + threadIdx.x;
        const bool real = j < num_atoms;
        for (int a = 0; a < 3; ++a)
        {
            candidates[a][threadIdx.x] = real ? positions[3 * j + a] : T(0);
        }
    }
    __syncthreads();
    const std::int64_t center = first_center + threadIdx.x;
    if (center >= num_atoms || center >= 32 * (word + 1) - 1)
    {
        return;
    }
    const T cx = positions[3 * center], cy = positions[3 * center + 1],
            cz = positions[3 * center + 2];
    const T lx = cell[0], ly = cell[1], lz = cell[2];
    std::uint32_t hits = 0;
#pragma unroll 8
    for (int b = 0; b < kWarp; ++b)
    {
        const std::int64_t j = 32 * word + b;
        const T dx = min_image(cx, candidates[0][b], lx);
        const T dy = min_image(cy, candidates[1][b], ly);
        const T dz = min_image(cz, candidates[2][b], lz);
        const bool hit = j > center && j < num_atoms && squared_norm(dx, dy, dz) < radius_squared;
        hits |= hit ? 1u << b : 0u;
    }
    bits[word * num_atoms + center] = hits;
}

// One thread per center: its pair count from its words.
__global__ void row_counts_kernel(
    const std::uint32_t* __restrict__ bits,
    index_t num_atoms,
    index_t* __restrict__ pair_counts,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status
)
{
    const std::int64_t center = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (center >= num_atoms || !rebuilding(rebuild, status))
    {
        return;
    }
    const std::int64_t words = bit_words(num_atoms);
    index_t count = 0;
    for (std::int64_t w = (center + 1) / kWarp; w < words; ++w)
    {
        count += __popc(bits[w * num_atoms + center]);
    }
    pair_counts[center] = count;
}

// One thread per center: its pairs from its words, in atom order, from its first column. The
// fill of an update also stores the center's position, and thread 0 the cell and the count.
template <typename T>
__global__ void row_fill_kernel(
    const std::uint32_t* __restrict__ bits,
    const index_t* __restrict__ pair_offsets,
    index_t num_atoms,
    index_t capacity,
    index_t* __restrict__ pairs,
    const T* __restrict__ positions,
    const T* __restrict__ cell,
    T* __restrict__ reference_positions,
    T* __restrict__ reference_cell,
    index_t* __restrict__ rebuild_count,
    const index_t* __restrict__ rebuild,
    const index_t* __restrict__ status
)
{
    const std::int64_t center = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (center >= num_atoms || !rebuilding(rebuild, status))
    {
        return;
    }
    if (reference_positions != nullptr)
    {
        for (int a = 0; a < 3; ++a)
        {
            reference_positions[3 * center + a] = positions[3 * center + a];
        }
        if (center == 0)
        {
            for (int a = 0; a < 3; ++a)
            {
                reference_cell[a] = cell[a];
            }
            ++rebuild_count[0];
        }
    }
    const std::int64_t words = bit_words(num_atoms);
    std::int64_t column = pair_offsets[center];
    for (std::int64_t w = (center + 1) / kWarp; w < words; ++w)
    {
        std::uint32_t hits = bits[w * num_atoms + center];
        while (hits != 0)
        {
            const int b = __ffs(hits) - 1;
            hits &= hits - 1;
            if (column < capacity)
            {
                pairs[column] = static_cast<index_t>(center);
                pairs[capacity + column] = static_cast<index_t>(32 * w + b);
            }
            ++column;
        }
    }
}

// ---------------------------------------------------------------------------------------
// Total, overflow and padding, in one launch over the capacity.

// Every thread derives the total from the last count and offset. The first thread stores the
// total and, above the capacity, the overflow bit and the pairs needed; with an overflow there is
// no padding column, so the gate's read of the status cannot race. A list whose fill has padded
// already (`pad` zero) needs the first thread only.
__global__ void total_and_pad_kernel(
    const index_t* __restrict__ pair_counts,
    const index_t* __restrict__ pair_offsets,
    index_t num_atoms,
    index_t capacity,
    index_t* __restrict__ pair_total,
    index_t* __restrict__ pairs,
    index_t* __restrict__ status,
    const index_t* __restrict__ rebuild,
    int pad
)
{
    if (!rebuilding(rebuild, status))
    {
        return;
    }
    const index_t total = pair_offsets[num_atoms - 1] + pair_counts[num_atoms - 1];
    const unsigned thread = blockIdx.x * blockDim.x + threadIdx.x;
    if (thread == 0)
    {
        pair_total[0] = total;
        if (total > capacity)
        {
            status[0] |= kOverflow;
            status[1] = total > status[1] ? total : status[1];
        }
    }
    if (pad)
    {
        pad_columns(total, num_atoms, capacity, pairs, thread, gridDim.x * blockDim.x);
    }
}

constexpr std::int64_t kPadBlocks = 148 * 8;  // every SM full; more columns take more steps

// The fill's CTAs that pad: few, because each takes a slot from the fill, and one more per 2^21
// columns of capacity, so that a roomy list's padding does not outlast the fill (1,048,576 atoms,
// fill and padding: 24 CTAs 537 us, 48 CTAs 539 us, 148 CTAs 583 us, a launch of its own 592 us).
constexpr std::int64_t kPadCtas = 37;
constexpr std::int64_t kPadColumns = 1 << 21;

// ---------------------------------------------------------------------------------------
// The update's gate (the rule of src/nabladyn/neighbors/csrc/update/update.cuh:13-20).
//
// A build stores the wrapped positions x0 and the cell L0. In a cell L, with s = L / L0 per
// axis, atom i has moved d_i = min image of x_i - s x0_i; the pairs are reused while every
// |d_i|^2 < ((R min(s) - cutoff - 32 eps L_max) / 2)^2. Entries of `reuse`: the squared
// threshold, then s per axis.

// One warp: lane a < 3 checks axis a of the cell and sets its grid (at most the first grid's
// bins, each wider than the radius with a margin of a few roundings of L) and its scale; lane 0
// then sets the threshold, or asks for a rebuild when there is no room to move. A list whose
// status holds an error stays as it is until it is allocated again.
template <typename T>
__global__ void open_update_kernel(
    const T* __restrict__ cell,
    const T* __restrict__ reference_cell,
    T cutoff,
    T radius,
    T epsilon,
    const index_t* __restrict__ limits,
    index_t* __restrict__ dims,
    T* __restrict__ widths,
    T* __restrict__ reuse,
    index_t* __restrict__ rebuild,
    index_t* __restrict__ status
)
{
    const int lane = threadIdx.x;
    const bool sound = status[0] == 0;
    if (lane == 0)
    {
        rebuild[0] = 0;
    }
    const int axis = lane < 3 ? lane : 0;
    const T length = cell[axis];
    const T scale = length / reference_cell[axis];
    const bool valid = isfinite(length) && length > 2 * cutoff;
    const bool all_valid = __all_sync(kFullMask, valid);
    if (!sound)
    {
        return;
    }
    if (!all_valid)
    {
        if (lane == 0)
        {
            status[0] |= kInvalidCell;
        }
        return;
    }
    if (lane < 3)
    {
        reuse[1 + axis] = scale;
        const T fit = floor(length / fma(T(4) * epsilon, length, radius));
        const index_t count =
            fit < 1 ? 1 : (fit > limits[axis] ? limits[axis] : static_cast<index_t>(fit));
        dims[axis] = count;
        widths[axis] = length / count;
    }
    // The smallest scale and the longest length, over the three axes in lane order.
    const T s0 = __shfl_sync(kFullMask, scale, 0), s1 = __shfl_sync(kFullMask, scale, 1),
            s2 = __shfl_sync(kFullMask, scale, 2);
    const T l0 = __shfl_sync(kFullMask, length, 0), l1 = __shfl_sync(kFullMask, length, 1),
            l2 = __shfl_sync(kFullMask, length, 2);
    if (lane == 0)
    {
        T smallest = s0 < s1 ? s0 : s1;
        smallest = s2 < smallest ? s2 : smallest;
        T longest = l1 > l0 ? l1 : l0;
        longest = l2 > longest ? l2 : longest;
        const T allowance = fma(-(T(32) * epsilon), longest, fma(radius, smallest, -cutoff));
        if (allowance <= 0)
        {
            rebuild[0] = 1;
            return;
        }
        reuse[0] = allowance * allowance / 4;
    }
}

// One thread per atom, one atomic per warp: the non-finite bit, then the rebuild request when
// an atom has moved past the threshold.
template <typename T>
__global__ void reuse_check_kernel(
    const T* __restrict__ positions,
    const T* __restrict__ reference_positions,
    const T* __restrict__ cell,
    const T* __restrict__ reuse,
    index_t num_atoms,
    index_t* __restrict__ rebuild,
    index_t* __restrict__ status
)
{
    const std::int64_t atom = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (status[0] != 0)
    {
        return;  // uniform: the open's verdict, read after its launch
    }
    const int lane = threadIdx.x % kWarp;
    bool bad = false, moved_far = false;
    if (atom < num_atoms)
    {
        const T* x = positions + 3 * atom;
        const T* x0 = reference_positions + 3 * atom;
        bad = !(isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]));
        T moved = 0;
        for (int axis = 0; axis < 3; ++axis)
        {
            const T d = min_image(x[axis], reuse[1 + axis] * x0[axis], cell[axis]);
            moved = fma(d, d, moved);
        }
        moved_far = !bad && moved >= reuse[0];
    }
    const unsigned bad_lanes = __ballot_sync(kFullMask, bad);
    const unsigned far_lanes = __ballot_sync(kFullMask, moved_far);
    if (lane == 0 && bad_lanes != 0)
    {
        atomicOr(status, kNonFinite);
    }
    if (lane == 0 && far_lanes != 0)
    {
        rebuild[0] = 1;  // every writer stores the same value
    }
}

// ---------------------------------------------------------------------------------------
// A list's first frame.

// Wraps the frame into the reference positions (space.wrap's rounding) and gives every small
// buffer its starting value, in one launch. `dims` are the first grid's bins per axis, each of
// width L / n; a non-finite coordinate sets `non_finite` (zero before the launch). A small list's
// first build is bound by its launches: 30 device operations became 14 (2,003 atoms in float64,
// the whole call 342 -> 192 us).
template <typename T>
__global__ void __launch_bounds__(kThreads) start_list_kernel(
    const T* __restrict__ positions, const T* __restrict__ cell, std::int64_t num_atoms,
    int nx, int ny, int nz, index_t* __restrict__ dims, T* __restrict__ widths,
    index_t* __restrict__ bin_counts, std::int64_t bin_slots, index_t* __restrict__ pair_total,
    index_t* __restrict__ status, T* __restrict__ reference_positions,
    T* __restrict__ reference_cell, index_t* __restrict__ limits, T* __restrict__ reuse,
    index_t* __restrict__ rebuild, index_t* __restrict__ rebuild_count,
    index_t* __restrict__ non_finite)
{
    const std::int64_t k = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    bool bad = false;
    if (k < 3 * num_atoms)
    {
        const T x = positions[k];
        bad = !isfinite(x);
        // The host refuses a frame with a non-finite coordinate only after the count; until
        // then the coordinate is spread over the cell, so such atoms do not fill one bin.
        const T spread = static_cast<T>(static_cast<unsigned>(k) * 2654435769u >> 8) / T(1 << 24);
        reference_positions[k] = bad ? spread * cell[k % 3] : wrap_separately(x, cell[k % 3]);
    }
    if (k < bin_slots)
    {
        bin_counts[k] = 0;
    }
    if (k < 4)
    {
        reuse[k] = T(0);
    }
    if (k < 3)
    {
        const index_t n = k == 0 ? nx : (k == 1 ? ny : nz);
        dims[k] = limits[k] = n;
        widths[k] = static_cast<T>(static_cast<double>(cell[k]) / n);
        reference_cell[k] = cell[k];
    }
    if (k < 2)
    {
        status[k] = 0;
    }
    if (k == 0)
    {
        pair_total[0] = 0;
        rebuild[0] = 0;
        rebuild_count[0] = 1;
    }
    if (__any_sync(kFullMask, bad) && threadIdx.x % kWarp == 0)
    {
        *non_finite = 1;  // every writer stores the same value
    }
}

// ---------------------------------------------------------------------------------------
// Host launchers.

struct List
{
    const nd_neighbor_buffers* b;
    const index_t* rebuild;  // null: a build from allocate, which always runs

    bool all_pairs() const { return b->bits_numel > 0; }
};

// Where an update's fill stores the frame it was built from; all null for allocate.
template <typename T>
struct Commit
{
    const T* positions = nullptr;
    T* reference_positions = nullptr;
    T* reference_cell = nullptr;
    index_t* rebuild_count = nullptr;
};

template <typename T>
int launch_grid(const T* positions, std::int64_t n, const List& list, cudaStream_t stream)
{
    const nd_neighbor_buffers& b = *list.b;
    const auto num_atoms = static_cast<index_t>(n);
    bin_atoms_kernel<T><<<blocks_for(n), kThreads, 0, stream>>>(
        positions, b.dims, static_cast<const T*>(b.widths), num_atoms, b.atom_bin, b.bin_counts,
        b.pair_counts, list.rebuild, b.status);
    ND_LAUNCH_CHECK();
    ND_CUDA_TRY(scan_exclusive(b.bin_counts, b.bin_offsets, b.num_bin_slots, b.scan_temp,
                               list.rebuild, b.status, stream));
    place_atoms_kernel<<<blocks_for(n), kThreads, 0, stream>>>(
        b.atom_bin, b.pair_counts, b.bin_offsets, num_atoms, b.bin_counts, b.unordered_ids,
        list.rebuild, b.status);
    ND_LAUNCH_CHECK();
    const std::int64_t bins = b.num_bin_slots - 1;
    order_bins_kernel<T><<<blocks_for(bins * kWarp), kThreads, 0, stream>>>(
        positions, b.unordered_ids, b.bin_offsets, bins, b.sorted_ids,
        static_cast<T*>(b.sorted_positions), list.rebuild, b.status);
    ND_LAUNCH_CHECK();
    return ND_OK;
}

template <typename T, bool kFill>
void launch_hood(const T* cell, std::int64_t n, double radius, const List& list,
                 const Commit<T>& commit, cudaStream_t stream)
{
    const nd_neighbor_buffers& b = *list.b;
    const T r = static_cast<T>(radius);
    const std::int64_t bins = b.num_bin_slots - 1;
    const std::int64_t most = std::min<std::int64_t>(blocks_for(b.capacity), kPadBlocks);
    const std::int64_t pad =
        kFill ? std::min(most, std::max(kPadCtas, b.capacity / kPadColumns)) : 0;
    // A list that has its pairs says by its columns whether its atoms are a gas; a first count
    // does not know, and may be of a droplet in a large box.
    const bool gas = b.capacity > 1 && b.capacity <= kGasColumns * n && kGasBins * bins > n;
    const std::int64_t per_cta =
        gas || bins > n
            ? std::min<std::int64_t>(kWarp, std::max<std::int64_t>(1, bins / kManyCtas))
            : 1;
    const std::int64_t ctas = (bins + per_cta - 1) / per_cta;
    auto launch = [&](auto kernel, int threads) {
        kernel<<<static_cast<unsigned>(ctas + pad), threads, 0, stream>>>(
            static_cast<const T*>(b.sorted_positions), b.sorted_ids, b.bin_offsets, b.dims, cell,
            r * r, b.pair_counts, b.pair_offsets, static_cast<index_t>(b.capacity), b.pairs,
            commit.positions, commit.reference_positions, commit.reference_cell,
            commit.rebuild_count, list.rebuild, b.status, static_cast<index_t>(n),
            static_cast<int>(pad), static_cast<index_t>(bins));
    };
    if (gas)
    {
        launch(hood_pairs_kernel<T, kFill, kWarp, true>, kWarp);
    }
    else if (per_cta > 1)
    {
        launch(hood_pairs_kernel<T, kFill, kHoodThreads, true>, kHoodThreads);
    }
    else if (bins <= kHoodFewBins)
    {
        launch(hood_pairs_kernel<T, kFill, kHoodFewThreads, false>, kHoodFewThreads);
    }
    else
    {
        launch(hood_pairs_kernel<T, kFill, kHoodThreads, false>, kHoodThreads);
    }
}

template <typename T>
int launch_count(const T* positions, const T* cell, std::int64_t n, double radius,
                 const List& list, cudaStream_t stream)
{
    const nd_neighbor_buffers& b = *list.b;
    const auto num_atoms = static_cast<index_t>(n);
    const T r = static_cast<T>(radius);
    if (list.all_pairs())
    {
        auto* bits = reinterpret_cast<std::uint32_t*>(b.bits);
        const dim3 grid(blocks_for(n, kWordThreads), static_cast<unsigned>(bit_words(n)));
        pair_words_kernel<T><<<grid, kWordThreads, 0, stream>>>(positions, cell, r * r,
                                                               num_atoms, bits, list.rebuild,
                                                               b.status);
        ND_LAUNCH_CHECK();
        row_counts_kernel<<<blocks_for(n), kThreads, 0, stream>>>(bits, num_atoms, b.pair_counts,
                                                                  list.rebuild, b.status);
    }
    else
    {
        launch_hood<T, false>(cell, n, radius, list, Commit<T>{}, stream);
    }
    ND_LAUNCH_CHECK();
    ND_CUDA_TRY(scan_exclusive(b.pair_counts, b.pair_offsets, n, b.scan_temp, list.rebuild,
                               b.status, stream));
    return ND_OK;
}

template <typename T>
int launch_fill(const T* cell, std::int64_t n, double radius, const List& list,
                const Commit<T>& commit, cudaStream_t stream)
{
    const nd_neighbor_buffers& b = *list.b;
    const auto num_atoms = static_cast<index_t>(n);
    const auto capacity = static_cast<index_t>(b.capacity);
    if (list.all_pairs())
    {
        row_fill_kernel<T><<<blocks_for(n), kThreads, 0, stream>>>(
            reinterpret_cast<const std::uint32_t*>(b.bits), b.pair_offsets, num_atoms, capacity,
            b.pairs, commit.positions, cell, commit.reference_positions, commit.reference_cell,
            commit.rebuild_count, list.rebuild, b.status);
    }
    else
    {
        launch_hood<T, true>(cell, n, radius, list, commit, stream);
    }
    ND_LAUNCH_CHECK();
    const bool pad = list.all_pairs();  // the grid's fill has padded
    const std::int64_t pad_blocks =
        pad ? std::min<std::int64_t>(blocks_for(b.capacity), kPadBlocks) : 1;
    total_and_pad_kernel<<<static_cast<unsigned>(pad_blocks), kThreads, 0, stream>>>(
        b.pair_counts, b.pair_offsets, num_atoms, capacity, b.pair_total, b.pairs, b.status,
        list.rebuild, pad);
    ND_LAUNCH_CHECK();
    return ND_OK;
}

int check_buffers(int dtype, std::int64_t n, const nd_neighbor_buffers* b)
{
    ND_REQUIRE(dtype == ND_FLOAT32 || dtype == ND_FLOAT64, "positions must be float32 or float64");
    ND_REQUIRE(b != nullptr, "the list's buffers are missing");
    ND_REQUIRE(n >= 1 && n <= INT32_MAX, "positions must have shape [N, 3] with 1 <= N < 2**31");
    ND_REQUIRE(b->num_bin_slots >= 2 && b->num_bin_slots <= INT32_MAX,
               "the list's buffers do not match the positions");
    ND_REQUIRE(b->capacity >= 1 && b->capacity <= INT32_MAX, "pairs must be [2, C] with int32 C");
    ND_REQUIRE(b->bits_numel == 0 || b->bits_numel == n * bit_words(n),
               "bits must be empty or hold N rows of ceil(N / 32) words");
    ND_REQUIRE(b->bits_numel == 0 || bit_words(n) <= 65535,
               "the all-pairs path takes at most 2,097,120 atoms");
    const std::int64_t need = scan_scratch_bytes(b->num_bin_slots > n ? b->num_bin_slots : n);
    ND_REQUIRE(b->scan_temp_bytes >= need, "scan_temp is smaller than scan_temp_bytes asks");
    ND_REQUIRE(b->dims && b->widths && b->atom_bin && b->bin_counts && b->bin_offsets &&
                   b->unordered_ids && b->sorted_ids && b->sorted_positions && b->scan_temp &&
                   b->pair_counts && b->pair_offsets && b->pair_total && b->status && b->pairs &&
                   (b->bits_numel == 0 || b->bits),
               "a buffer of the list is null");
    return ND_OK;
}

template <typename T>
int count_first_frame(const void* positions, const void* cell, std::int64_t n, double radius,
                      const nd_neighbor_buffers* b, cudaStream_t stream)
{
    const List list{b, nullptr};
    const auto* x = static_cast<const T*>(positions);
    if (!list.all_pairs())
    {
        const int rc = launch_grid<T>(x, n, list, stream);
        if (rc != ND_OK)
        {
            return rc;
        }
    }
    return launch_count<T>(x, static_cast<const T*>(cell), n, radius, list, stream);
}

template <typename T>
int update(const void* positions, const void* cell, std::int64_t n, double cutoff, double radius,
           const nd_reuse_buffers* r, const nd_neighbor_buffers* b, cudaStream_t stream)
{
    const List list{b, r->rebuild};
    const auto* x = static_cast<const T*>(positions);
    const auto* box = static_cast<const T*>(cell);
    const auto num_atoms = static_cast<index_t>(n);
    open_update_kernel<T><<<1, kWarp, 0, stream>>>(
        box, static_cast<const T*>(r->reference_cell), static_cast<T>(cutoff),
        static_cast<T>(radius), std::numeric_limits<T>::epsilon(), r->limits, b->dims,
        static_cast<T*>(b->widths), static_cast<T*>(r->reuse), r->rebuild, b->status);
    ND_LAUNCH_CHECK();
    reuse_check_kernel<T><<<blocks_for(n), kThreads, 0, stream>>>(
        x, static_cast<const T*>(r->reference_positions), box, static_cast<const T*>(r->reuse),
        num_atoms, r->rebuild, b->status);
    ND_LAUNCH_CHECK();
    int rc = ND_OK;
    if (!list.all_pairs() && (rc = launch_grid<T>(x, n, list, stream)) != ND_OK)
    {
        return rc;
    }
    if ((rc = launch_count<T>(x, box, n, radius, list, stream)) != ND_OK)
    {
        return rc;
    }
    Commit<T> commit;
    commit.positions = x;
    commit.reference_positions = static_cast<T*>(r->reference_positions);
    commit.reference_cell = static_cast<T*>(r->reference_cell);
    commit.rebuild_count = r->rebuild_count;
    return launch_fill<T>(box, n, radius, list, commit, stream);
}

}  // namespace nd

// ---------------------------------------------------------------------------------------
// C-ABI.

extern "C" {

int nd_neighbors_scan_temp_bytes(std::int64_t items, std::int64_t* bytes)
{
    ND_REQUIRE(items > 0 && items <= INT32_MAX, "the scan length must fit int32");
    ND_REQUIRE(bytes != nullptr, "bytes is null");
    *bytes = nd::scan_scratch_bytes(items);
    return ND_OK;
}

int nd_neighbors_count_first_frame(int dtype, const void* positions, const void* cell,
                                   std::int64_t num_atoms, double radius,
                                   const nd_neighbor_buffers* buffers, nd_stream_t stream)
{
    const int rc = nd::check_buffers(dtype, num_atoms, buffers);
    if (rc != ND_OK)
    {
        return rc;
    }
    ND_REQUIRE(positions && cell, "positions and cell must not be null");
    auto s = static_cast<cudaStream_t>(stream);
    return dtype == ND_FLOAT32
               ? nd::count_first_frame<float>(positions, cell, num_atoms, radius, buffers, s)
               : nd::count_first_frame<double>(positions, cell, num_atoms, radius, buffers, s);
}

int nd_neighbors_start(int dtype, const void* positions, const void* cell, std::int64_t num_atoms,
                       const std::int32_t* dims, const nd_reuse_buffers* reuse,
                       const nd_neighbor_buffers* buffers, std::int32_t* non_finite,
                       nd_stream_t stream)
{
    ND_REQUIRE(dtype == ND_FLOAT32 || dtype == ND_FLOAT64, "positions must be float32 or float64");
    ND_REQUIRE(num_atoms >= 1 && num_atoms <= INT32_MAX,
               "positions must have shape [N, 3] with 1 <= N < 2**31");
    ND_REQUIRE(positions && cell && dims && reuse && buffers && non_finite,
               "a required pointer is null");
    const nd_neighbor_buffers& b = *buffers;
    const nd_reuse_buffers& r = *reuse;
    ND_REQUIRE(dims[0] >= 1 && dims[1] >= 1 && dims[2] >= 1, "dims must be positive");
    ND_REQUIRE(b.num_bin_slots >= 2 && b.num_bin_slots <= INT32_MAX && b.dims && b.widths &&
                   b.bin_counts && b.pair_total && b.status && r.reference_positions &&
                   r.reference_cell && r.limits && r.reuse && r.rebuild && r.rebuild_count,
               "a buffer of the list is null");
    auto s = static_cast<cudaStream_t>(stream);
    ND_CUDA_TRY(cudaMemsetAsync(non_finite, 0, sizeof(std::int32_t), s));
    const std::int64_t items = std::max<std::int64_t>(3 * num_atoms, b.num_bin_slots);
    auto launch = [&](auto zero) {
        using T = decltype(zero);
        nd::start_list_kernel<T><<<nd::blocks_for(items), nd::kThreads, 0, s>>>(
            static_cast<const T*>(positions), static_cast<const T*>(cell), num_atoms, dims[0],
            dims[1], dims[2], b.dims, static_cast<T*>(b.widths), b.bin_counts, b.num_bin_slots,
            b.pair_total, b.status, static_cast<T*>(r.reference_positions),
            static_cast<T*>(r.reference_cell), const_cast<std::int32_t*>(r.limits),
            static_cast<T*>(r.reuse), r.rebuild, r.rebuild_count, non_finite);
    };
    dtype == ND_FLOAT32 ? launch(float{}) : launch(double{});
    ND_LAUNCH_CHECK();
    return ND_OK;
}

int nd_neighbors_fill_first_frame(int dtype, const void* positions, const void* cell,
                                  std::int64_t num_atoms, double radius,
                                  const nd_neighbor_buffers* buffers, nd_stream_t stream)
{
    const int rc = nd::check_buffers(dtype, num_atoms, buffers);
    if (rc != ND_OK)
    {
        return rc;
    }
    ND_REQUIRE(positions && cell, "positions and cell must not be null");
    const nd::List list{buffers, nullptr};
    auto s = static_cast<cudaStream_t>(stream);
    return dtype == ND_FLOAT32
               ? nd::launch_fill<float>(static_cast<const float*>(cell), num_atoms, radius, list,
                                        nd::Commit<float>{}, s)
               : nd::launch_fill<double>(static_cast<const double*>(cell), num_atoms, radius,
                                         list, nd::Commit<double>{}, s);
}

int nd_neighbors_update(int dtype, const void* positions, const void* cell,
                        std::int64_t num_atoms, double cutoff, double radius,
                        const nd_reuse_buffers* reuse, const nd_neighbor_buffers* buffers,
                        nd_stream_t stream)
{
    const int rc = nd::check_buffers(dtype, num_atoms, buffers);
    if (rc != ND_OK)
    {
        return rc;
    }
    ND_REQUIRE(positions && cell, "positions and cell must not be null");
    ND_REQUIRE(reuse && reuse->reference_positions && reuse->reference_cell && reuse->limits &&
                   reuse->reuse && reuse->rebuild && reuse->rebuild_count,
               "the list's update buffers do not match the positions");
    auto s = static_cast<cudaStream_t>(stream);
    return dtype == ND_FLOAT32
               ? nd::update<float>(positions, cell, num_atoms, cutoff, radius, reuse, buffers, s)
               : nd::update<double>(positions, cell, num_atoms, cutoff, radius, reuse, buffers,
                                    s);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// The pair build without allocation.
//
// Some callers cannot call cudaMalloc at all: code running inside another framework's CUDA
// Graph capture or memory pool, plugins whose host forbids allocation, or embedded drivers
// with a fixed memory map. For them, nd_neighbors_build_no_alloc builds one frame's pair list
// with every intermediate buffer (bins, sorted ids and positions, counts, offsets, scan tiles,
// the all-pairs bit matrix) in one file-scope device array of fixed size, kNoAllocBytes, which
// every GPU that loads this library holds until the process exits. The caller passes only
// the positions, the cell and the outputs.

namespace nd {

constexpr std::int64_t kNoAllocMaxAtoms = 16384;
constexpr std::int64_t kNoAllocMaxBins = 16384;
constexpr std::int64_t kNoAllocMaxAllPairsAtoms = 2048;

constexpr std::int64_t round_up_256(std::int64_t bytes)
{
    return (bytes + 255) / 256 * 256;
}

// The layout of the array, in bytes from its start.
struct NoAllocLayout
{
    static constexpr std::int64_t dims = 0;
    static constexpr std::int64_t go = 128;      // the build's gate, set by store_grid_kernel
    static constexpr std::int64_t widths = 256;  // three doubles at most
    static constexpr std::int64_t atom_bin = 512;
    static constexpr std::int64_t bin_counts = atom_bin + round_up_256(4 * kNoAllocMaxAtoms);
    static constexpr std::int64_t bin_offsets = bin_counts + round_up_256(4 * (kNoAllocMaxBins + 1));
    static constexpr std::int64_t unordered_ids =
        bin_offsets + round_up_256(4 * (kNoAllocMaxBins + 1));
    static constexpr std::int64_t sorted_ids = unordered_ids + round_up_256(4 * kNoAllocMaxAtoms);
    static constexpr std::int64_t sorted_positions =
        sorted_ids + round_up_256(4 * kNoAllocMaxAtoms);
    static constexpr std::int64_t pair_counts =
        sorted_positions + round_up_256(3 * 8 * kNoAllocMaxAtoms);
    static constexpr std::int64_t pair_offsets = pair_counts + round_up_256(4 * kNoAllocMaxAtoms);
    static constexpr std::int64_t scan_temp = pair_offsets + round_up_256(4 * kNoAllocMaxAtoms);
    static constexpr std::int64_t bits =
        scan_temp + round_up_256((kNoAllocMaxAtoms + 1 + kTileItems - 1) / kTileItems * 4 + 16);
    static constexpr std::int64_t size =
        bits + round_up_256(4 * kNoAllocMaxAllPairsAtoms * ((kNoAllocMaxAllPairsAtoms + 31) / 32));
};

constexpr std::int64_t kNoAllocBytes = NoAllocLayout::size;

// The scratch itself. In host code this name is only a stand-in for the symbol: its device
// address comes from cudaGetSymbolAddress, per device.
static __device__ __align__(256) unsigned char no_alloc_scratch[kNoAllocBytes];

// The grid of the frame: the caller's bins per axis, each of width L / n as allocate chooses.
// A bin narrower than the radius would lose pairs: the build is then not run and the status
// reports an invalid cell. `go` gates the build's kernels as an update's rebuild flag does.
template <typename T>
__global__ void store_grid_kernel(index_t* dims, T* widths, const T* cell, T radius, int nx,
                                  int ny, int nz, index_t* go, index_t* status)
{
    const int n[3] = {nx, ny, nz};
    bool narrow = false;
    for (int a = 0; a < 3; ++a)
    {
        dims[a] = n[a];
        widths[a] = cell[a] / n[a];
        narrow = narrow || !(widths[a] >= radius);
    }
    go[0] = 1;
    status[0] = narrow ? kInvalidCell : 0;
    status[1] = 0;
}

// The array's device address on the current device, looked up once per device; concurrent
// first calls from several host threads store the same address.
int no_alloc_scratch_address(unsigned char** address)
{
    constexpr int kMaxDevices = 64;
    static std::atomic<unsigned char*> addresses[kMaxDevices] = {};
    int device = 0;
    ND_CUDA_TRY(cudaGetDevice(&device));
    ND_REQUIRE(device >= 0 && device < kMaxDevices, "the device index is out of range");
    unsigned char* known = addresses[device].load(std::memory_order_acquire);
    if (known == nullptr)
    {
        void* found = nullptr;
        ND_CUDA_TRY(cudaGetSymbolAddress(&found, no_alloc_scratch));
        known = static_cast<unsigned char*>(found);
        addresses[device].store(known, std::memory_order_release);
    }
    *address = known;
    return ND_OK;
}

template <typename T>
int build_no_alloc(const void* positions, const void* cell, std::int64_t n, double radius,
                   const std::int32_t* dims, std::int32_t* pairs, std::int64_t capacity,
                   std::int32_t* pair_total, std::int32_t* status, cudaStream_t stream)
{
    unsigned char* base = nullptr;
    const int found = no_alloc_scratch_address(&base);
    if (found != ND_OK)
    {
        return found;
    }
    const std::int64_t bins = static_cast<std::int64_t>(dims[0]) * dims[1] * dims[2];
    const bool all_pairs = dims[0] <= 3 && dims[1] <= 3 && dims[2] <= 3;
    nd_neighbor_buffers b{};
    b.dims = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::dims);
    b.widths = base + NoAllocLayout::widths;
    b.atom_bin = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::atom_bin);
    b.bin_counts = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::bin_counts);
    b.bin_offsets = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::bin_offsets);
    b.num_bin_slots = bins + 1;
    b.unordered_ids = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::unordered_ids);
    b.sorted_ids = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::sorted_ids);
    b.sorted_positions = base + NoAllocLayout::sorted_positions;
    b.scan_temp = base + NoAllocLayout::scan_temp;
    b.scan_temp_bytes = NoAllocLayout::bits - NoAllocLayout::scan_temp;
    b.pair_counts = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::pair_counts);
    b.pair_offsets = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::pair_offsets);
    b.pair_total = pair_total;
    b.status = status;
    b.pairs = pairs;
    b.capacity = capacity;
    b.bits = all_pairs ? reinterpret_cast<std::int32_t*>(base + NoAllocLayout::bits) : nullptr;
    b.bits_numel = all_pairs ? n * bit_words(n) : 0;
    // What must start at zero: the bin counts (a build returns them to zero, but an earlier
    // call may have stopped short) and the total; the grid kernel sets the status and the gate.
    auto* go = reinterpret_cast<std::int32_t*>(base + NoAllocLayout::go);
    ND_CUDA_TRY(cudaMemsetAsync(b.bin_counts, 0, sizeof(std::int32_t) * (bins + 1), stream));
    ND_CUDA_TRY(cudaMemsetAsync(pair_total, 0, sizeof(std::int32_t), stream));
    store_grid_kernel<T><<<1, 1, 0, stream>>>(b.dims, static_cast<T*>(b.widths),
                                              static_cast<const T*>(cell),
                                              static_cast<T>(radius), dims[0], dims[1], dims[2],
                                              go, status);
    ND_LAUNCH_CHECK();
    const List list{&b, go};
    const auto* x = static_cast<const T*>(positions);
    const auto* box = static_cast<const T*>(cell);
    int rc = ND_OK;
    if (!all_pairs && (rc = launch_grid<T>(x, n, list, stream)) != ND_OK)
    {
        return rc;
    }
    if ((rc = launch_count<T>(x, box, n, radius, list, stream)) != ND_OK)
    {
        return rc;
    }
    return launch_fill<T>(box, n, radius, list, Commit<T>{}, stream);
}

}  // namespace nd

extern "C" int nd_neighbors_build_no_alloc(int dtype, const void* positions, const void* cell,
                                           int64_t num_atoms, double radius,
                                           const int32_t* dims, const double* widths,
                                           int32_t* pairs, int64_t capacity,
                                           int32_t* pair_total, int32_t* status,
                                           nd_stream_t stream)
{
    ND_REQUIRE(dtype == ND_FLOAT32 || dtype == ND_FLOAT64, "positions must be float32 or float64");
    ND_REQUIRE(positions && cell && dims && widths && pairs && pair_total && status,
               "a required pointer is null");
    ND_REQUIRE(num_atoms >= 1 && num_atoms <= nd::kNoAllocMaxAtoms,
               "nd_neighbors_build_no_alloc takes at most 16384 atoms");
    ND_REQUIRE(std::isfinite(radius) && radius > 0, "the radius must be positive and finite");
    ND_REQUIRE(dims[0] >= 1 && dims[1] >= 1 && dims[2] >= 1, "dims must be positive");
    for (int a = 0; a < 3; ++a)
    {
        ND_REQUIRE(std::isfinite(widths[a]) && widths[a] > 0,
                   "widths must be positive and finite");
        ND_REQUIRE(widths[a] >= radius, "a bin must be at least the radius wide");
    }
    const std::int64_t bins = static_cast<std::int64_t>(dims[0]) * dims[1] * dims[2];
    ND_REQUIRE(bins <= nd::kNoAllocMaxBins, "nd_neighbors_build_no_alloc takes at most 16384 bins");
    const bool all_pairs = dims[0] <= 3 && dims[1] <= 3 && dims[2] <= 3;
    ND_REQUIRE(!all_pairs || num_atoms <= nd::kNoAllocMaxAllPairsAtoms,
               "with at most three bins per axis nd_neighbors_build_no_alloc takes at most 2048 "
               "atoms");
    ND_REQUIRE(capacity >= 1 && capacity <= INT32_MAX, "pairs must be [2, C] with int32 C");
    auto s = static_cast<cudaStream_t>(stream);
    return dtype == ND_FLOAT32
               ? nd::build_no_alloc<float>(positions, cell, num_atoms, radius, dims, pairs,
                                           capacity, pair_total, status, s)
               : nd::build_no_alloc<double>(positions, cell, num_atoms, radius, dims, pairs,
                                            capacity, pair_total, status, s);
}
