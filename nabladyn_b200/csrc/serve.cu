// The replica server: many independent Lennard-Jones NVT replicas (tens to thousands of atoms
// each) resident in one pool, advanced by a persistent kernel in which a CTA, or a cluster of
// up to eight while the GPU has SMs to spare, owns one replica and runs a whole budget of
// steps: the chain half steps, the drift, the on-GPU reuse check, the rebuild, the forces and
// the second half kick, separated by block or cluster barriers only. No per-step launch, no
// grid-wide synchronisation: replicas never wait on each other, and every sum over a replica's
// atoms is taken per 32 list rows and then in row order, whoever computed the rows, so a
// replica's result does not depend, bit for bit, on its batch-mates or on the CTAs it was given.
//
// It serves the same step as the MD engine (src/nabladyn/md/_ensembles/_nvt.py:88-129,
// _nve.py:39-58, _chain.py:36-83, the reuse rule of src/nabladyn/neighbors/csrc/update/
// update.cuh:21-116) for systems too small to fill a GPU one at a time. Positions stay unwrapped
// between rebuilds and every pair takes its minimum image. The neighbor list is the engine's
// chunked full list of uint16 replica-local indices; a rebuild sorts the replica into cells
// (deterministically, by atom index within a cell) in the CTA, or tests all pairs when an axis
// has fewer than three cells.

#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <cstdint>

#include "common.cuh"
#include "geometry.cuh"
#include "md_common.cuh"

namespace nd {

constexpr int kServeThreads = 512;
constexpr int kServeWarps = kServeThreads / kWarp;
constexpr int kServeMaxCells = 4096;
constexpr int kServeTeam = 8;          // CTAs a replica gets at most (a portable cluster)
constexpr int kServeTeamAtoms = 1024;  // atoms for each of them: two rows per thread

struct ServePool
{
    nd_replica* replicas;
    Pos4<float>* pos;
    float* vel;
    float* force;
    float* mass;
    float* inv_mass;
    long long* images;
    Pos4<float>* ref_pos;
    std::uint16_t* nbr;
    index_t* nbr_count;
    index_t* sorted;
    index_t* scratch;
    index_t* cell_start;
    Pos4<float>* ordered;
};

// The scalar fields of one replica, in shared memory for the CTA.
struct ReplicaScalars
{
    int n;
    int width;
    int dims[3];
    int cells;
    float cell[3];
    float widths[3];
    float cutoff_squared;
    float radius_squared;
    float threshold_squared;
    float dt;
    float half_dt;
    PairParams<float> lj;
    int status;
    int rebuild_count;
    int steps_left;
};

// The CTAs that advance one replica: list rows (and atoms) go to them 512 at a time in turn.
// A team of one, whatever the launch's cluster, keeps to block barriers.
struct Team
{
    int rank;
    int size;

    __device__ int first() const { return rank * kServeThreads + static_cast<int>(threadIdx.x); }
    __device__ int stride() const { return size * kServeThreads; }

    // A barrier over the team; what each CTA wrote to global or its peers' shared memory before
    // it, every CTA reads after it.
    __device__ void sync() const
    {
        if (size == 1)
        {
            __syncthreads();
        }
        else
        {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;\n"
                         "barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }

    // Stores `value` in slot `rank` of every CTA's `slots`, by one warp's lanes.
    __device__ void tell(int* slots, int value) const
    {
        if (static_cast<int>(threadIdx.x) < size)
        {
            int* remote;
            asm volatile("mapa.u64 %0, %1, %2;"
                         : "=l"(remote)
                         : "l"(slots), "r"(static_cast<unsigned>(threadIdx.x)));
            remote[rank] = value;
        }
    }
};

// Block sum of one double per thread, in a fixed order; every thread gets the total.
__device__ double block_sum(double value, double* warp_sums)
{
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    value = warp_sum(value);
    if (lane == 0)
    {
        warp_sums[warp] = value;
    }
    __syncthreads();
    double total = 0;
    for (int w = 0; w < kServeWarps; ++w)
    {
        total += warp_sums[w];
    }
    __syncthreads();
    return total;
}

// Exclusive scan of counts[0, cells) in place (counts[cells] gets the total), kServeMaxCells at
// most: each thread owns 8 consecutive counts, the 512 thread sums are scanned by warps.
__device__ void block_scan_cells(int* counts, int cells, int* warp_totals)
{
    constexpr int kPer = kServeMaxCells / kServeThreads;
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
    const int base = threadIdx.x * kPer;
    int local[kPer];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k)
    {
        local[k] = base + k < cells ? counts[base + k] : 0;
        sum += local[k];
    }
    int inclusive = sum;
#pragma unroll
    for (int offset = 1; offset < kWarp; offset *= 2)
    {
        const int up = __shfl_up_sync(kFullMask, inclusive, offset);
        inclusive += lane >= offset ? up : 0;
    }
    if (lane == kWarp - 1)
    {
        warp_totals[warp] = inclusive;
    }
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w)
    {
        before += warp_totals[w];
    }
    int running = before + inclusive - sum;
#pragma unroll
    for (int k = 0; k < kPer; ++k)
    {
        if (base + k < cells)
        {
            counts[base + k] = running;
        }
        running += local[k];
    }
    if (threadIdx.x == kServeThreads - 1)
    {
        counts[cells] = running;
    }
    __syncthreads();
}

// The image of one stencil cell along an axis: the cell index h + d wrapped into [0, dims),
// and which side of the displacement takes the period. Past the upper face the center moves
// (center - L), past the lower face the candidate does (candidate - L): the two forms the
// minimum image rounds (min_image), so every candidate within the radius gets the bits the
// per-candidate minimum image gives it (the radius is below half the period: on a grid every
// axis has at least three cells at least one radius wide, and a displacement under the radius
// along an axis has one image within half the period).
struct AxisImage
{
    int cell;
    float center_shift;
    float candidate_shift;
};

__device__ __forceinline__ AxisImage axis_image(int h, int d, int dims, float length)
{
    AxisImage a{h + d, 0.0f, 0.0f};
    if (a.cell < 0)
    {
        a.cell += dims;
        a.candidate_shift = length;
    }
    else if (a.cell >= dims)
    {
        a.cell -= dims;
        a.center_shift = length;
    }
    return a;
}

// A row's chunks (see ListWriter), staged in a ring of 16 entries per lane in shared memory:
// a hit is one predicated 2-byte store, without a branch, and after every eight candidates one
// drain moves a full chunk to global memory. Entry e of a warp's lane lies at [e % 16][lane].
struct RingListWriter
{
    uint4* chunks;
    std::uint16_t* ring;  // this lane's entry 0
    int width;
    int row;
    int count;
    int drained;  // entries in global memory, or dropped beyond the width: a multiple of 8

    __device__ __forceinline__ RingListWriter(std::uint16_t* list, std::uint16_t* ring_,
                                              int width_, int row_)
        : chunks(reinterpret_cast<uint4*>(list)), ring(ring_), width(width_), row(row_), count(0),
          drained(0)
    {
    }

    __device__ __forceinline__ void add(bool hit, int index)
    {
        if (hit)
        {
            ring[(count & 15) * kWarp] = static_cast<std::uint16_t>(index);
            ++count;
        }
    }

    // After at most eight adds.
    __device__ __forceinline__ void drain()
    {
        if (count - drained >= kChunk)
        {
            store();
        }
    }

    __device__ __forceinline__ void store()
    {
        if (drained < width)
        {
            const std::uint16_t* from = ring + (drained & 15) * kWarp;
            unsigned packed[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                packed[k] = from[2 * k * kWarp] |
                            static_cast<unsigned>(from[(2 * k + 1) * kWarp]) << 16;
            }
            chunks[chunk_index(row, drained / kChunk, width)] =
                make_uint4(packed[0], packed[1], packed[2], packed[3]);
        }
        drained += kChunk;
    }

    // Stores a partial last chunk, its unused slots set to `pad`.
    __device__ __forceinline__ void finish(unsigned pad)
    {
        if (count > drained)
        {
            for (int e = count; e < drained + kChunk; ++e)
            {
                ring[(e & 15) * kWarp] = static_cast<std::uint16_t>(pad);
            }
            store();
        }
    }
};

// Adds to `list` the candidates k = begin .. end - 1 of the cell-ordered copy (x, y, z, and the
// atom's index in w) that lie closer than the list radius to the center (cell-order row
// `self`), in k order: one 16-B load per candidate, no index lookup and no per-candidate image
// choice. With kImaged the center and the candidates are moved by the cell's image (center at
// cx, candidates by -sx). Eight candidates at a time, all loaded before any is tested.
// Issue and the hits' divergence bound the scan. An append loop over each group's hit bits ran as
// often as the warp's fullest lane had hits (4-5 times for 1.1 hits on average) and fetched every
// index from memory: 148 replicas of 12,000 atoms, 60 steps with 7.5 rebuilds, 62.8 -> 55.4 ms.
template <bool kImaged>
__device__ __forceinline__ void scan_run(const ReplicaScalars& r, float cx, float cy, float cz,
                                         float sx, float sy, float sz, int self,
                                         const Pos4<float>* ordered, int begin, int end,
                                         RingListWriter& list)
{
    constexpr int kGroup = kChunk;
    for (int k = begin; k < end; k += kGroup)
    {
        Pos4<float> p[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
        {
            p[u] = ordered[min(k + u, end - 1)];
        }
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
        {
            const float d2 = kImaged ? squared_norm(cx - (p[u].x - sx), cy - (p[u].y - sy),
                                                    cz - (p[u].z - sz))
                                     : squared_norm(cx - p[u].x, cy - p[u].y, cz - p[u].z);
            list.add(k + u < end && k + u != self && d2 < r.radius_squared,
                     __float_as_int(p[u].w));
        }
        list.drain();
    }
}

// Adds to `list` the atoms k < n closer to `me` (atom `self`) than the list radius under the
// minimum image, in k order: the path of a replica with fewer than three cells along an axis
// (592 replicas of 500 atoms, 60 steps with 4.7 rebuilds: 7.8 -> 6.4 ms with the ring in place
// of chunks packed in registers by a branch per hit).
__device__ __forceinline__ void scan_all(const ReplicaScalars& r, const Pos4<float>& me, int self,
                                         const Pos4<float>* pos, RingListWriter& list)
{
    constexpr int kGroup = kChunk;
    for (int k = 0; k < r.n; k += kGroup)
    {
        Pos4<float> p[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
        {
            p[u] = pos[min(k + u, r.n - 1)];
        }
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
        {
            const float d2 = squared_norm(min_image(me.x, p[u].x, r.cell[0]),
                                          min_image(me.y, p[u].y, r.cell[1]),
                                          min_image(me.z, p[u].z, r.cell[2]));
            list.add(k + u < r.n && k + u != self && d2 < r.radius_squared, k + u);
        }
        list.drain();
    }
}

// Wraps the positions (counting crossings into the images), stores the reference frame and
// rebuilds the list. Called by the whole team; the cell sort, 3 % of a rebuild, is its first
// CTA's. On a grid, `ordered` receives the wrapped positions in cell order with each atom's
// index in w, which the candidate scan reads.
__device__ void rebuild_replica(const Team& team, const ReplicaScalars& r, Pos4<float>* pos,
                                Pos4<float>* ref, long long* images, std::uint16_t* nbr,
                                index_t* nbr_count, index_t* sorted, index_t* scratch,
                                index_t* cell_start, Pos4<float>* ordered, int* counts,
                                int* warp_totals, int* status_flags)
{
    const int n = r.n;
    for (int i = team.first(); i < n; i += team.stride())
    {
        Pos4<float> p = pos[i];
        long long c[3];
        p.x = wrap_axis(p.x, r.cell[0], c[0]);
        p.y = wrap_axis(p.y, r.cell[1], c[1]);
        p.z = wrap_axis(p.z, r.cell[2], c[2]);
        if (c[0] | c[1] | c[2])
        {
            images[3LL * i] += c[0];
            images[3LL * i + 1] += c[1];
            images[3LL * i + 2] += c[2];
        }
        pos[i] = p;
        ref[i] = p;
    }
    const bool grid = r.dims[0] >= 3 && r.dims[1] >= 3 && r.dims[2] >= 3;
    if (team.size > 1)
    {
        team.sync();
    }
    if (grid && team.rank == 0)
    {
        // Counting sort by cell (the slot parked in nbr_count, rewritten by the list below),
        // then each cell's range ordered by atom index, so the order is deterministic.
        for (int c = threadIdx.x; c <= r.cells; c += kServeThreads)
        {
            counts[c] = 0;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += kServeThreads)
        {
            const Pos4<float> p = pos[i];
            const int c = axis_bin(p.x, r.widths[0], r.dims[0]) +
                          r.dims[0] * (axis_bin(p.y, r.widths[1], r.dims[1]) +
                                       r.dims[1] * axis_bin(p.z, r.widths[2], r.dims[2]));
            scratch[i] = c;
            nbr_count[i] = atomicAdd(counts + c, 1);
        }
        __syncthreads();
        block_scan_cells(counts, r.cells, warp_totals);
        for (int c = threadIdx.x; c <= r.cells; c += kServeThreads)
        {
            cell_start[c] = counts[c];
        }
        for (int i = threadIdx.x; i < n; i += kServeThreads)
        {
            sorted[counts[scratch[i]] + nbr_count[i]] = i;
        }
        __syncthreads();
        for (int c = threadIdx.x; c < r.cells; c += kServeThreads)
        {
            const int begin = counts[c], end = counts[c + 1];
            for (int k = begin + 1; k < end; ++k)
            {
                const int atom = sorted[k];
                int m = k - 1;
                while (m >= begin && sorted[m] > atom)
                {
                    sorted[m + 1] = sorted[m];
                    --m;
                }
                sorted[m + 1] = atom;
            }
        }
    }
    team.sync();
    if (grid)
    {
        if (team.rank != 0)
        {
            for (int c = threadIdx.x; c <= r.cells; c += kServeThreads)
            {
                counts[c] = cell_start[c];
            }
        }
        for (int row = team.first(); row < n; row += team.stride())
        {
            const int atom = sorted[row];
            Pos4<float> p = pos[atom];
            p.w = __int_as_float(atom);
            ordered[row] = p;
        }
        team.sync();
    }
    // The list: every neighbor j != i closer than the list radius, minimum image. Row `row`
    // holds the list of atom sorted[row] on a grid (the lanes of a warp take atoms of one or
    // two cells, whose candidates they share), of atom `row` otherwise. On a grid the stencil
    // is scanned in two passes, each in stencil order with candidates in cell order: first the
    // cells that need no image, whose entries (the "direct" ones) keep the plain difference as
    // their minimum image until the next rebuild, then the cells across a face. Each cell is
    // scanned with its image, so the entries are those of a scan of every candidate with its
    // own minimum image. nbr_count[row] holds the count in its low 16 bits and the direct
    // entries in its high 16 bits (a count is at most N - 1 < 2^16).
    // The three cells of a stencil row are adjacent in the cell order, so those without an image
    // along x are one run of candidates.
    __shared__ std::uint16_t rings[kServeWarps][2 * kChunk][kWarp];
    for (int row = team.first(); row < n; row += team.stride())
    {
        RingListWriter list(nbr, &rings[threadIdx.x / kWarp][0][threadIdx.x % kWarp], r.width,
                            row);
        int direct = 0;
        if (grid)
        {
            const Pos4<float> me = ordered[row];
            const int hx = axis_bin(me.x, r.widths[0], r.dims[0]);
            const int hy = axis_bin(me.y, r.widths[1], r.dims[1]);
            const int hz = axis_bin(me.z, r.widths[2], r.dims[2]);
            const int low = max(hx - 1, 0), high = min(hx + 1, r.dims[0] - 1);
            for (int pass = 0; pass < 2; ++pass)
            {
                for (int dz = -1; dz <= 1; ++dz)
                {
                    const AxisImage iz = axis_image(hz, dz, r.dims[2], r.cell[2]);
                    const float cz = me.z - iz.center_shift;
                    for (int dy = -1; dy <= 1; ++dy)
                    {
                        const AxisImage iy = axis_image(hy, dy, r.dims[1], r.cell[1]);
                        const float cy = me.y - iy.center_shift;
                        const bool imaged = hy + dy != iy.cell || hz + dz != iz.cell;
                        const int* first = counts + r.dims[0] * (iy.cell + r.dims[1] * iz.cell);
                        if (pass == 0)
                        {
                            if (!imaged)
                            {
                                scan_run<false>(r, me.x, cy, cz, 0.0f, 0.0f, 0.0f, row, ordered,
                                                first[low], first[high + 1], list);
                            }
                            continue;
                        }
                        // Past the lower face, between the faces, past the upper face.
                        for (int side = -1; side <= 1; ++side)
                        {
                            const bool there = side < 0    ? hx == 0
                                               : side == 0 ? imaged
                                                           : hx == r.dims[0] - 1;
                            if (there)
                            {
                                const int from = side < 0 ? r.dims[0] - 1 : side == 0 ? low : 0;
                                const int to = side < 0 ? r.dims[0] : side == 0 ? high + 1 : 1;
                                scan_run<true>(r, side > 0 ? me.x - r.cell[0] : me.x, cy, cz,
                                               side < 0 ? r.cell[0] : 0.0f, iy.candidate_shift,
                                               iz.candidate_shift, row, ordered, first[from],
                                               first[to], list);
                            }
                        }
                    }
                }
                if (pass == 0)
                {
                    direct = list.count;
                }
            }
        }
        else
        {
            scan_all(r, pos[row], row, pos, list);
        }
        list.finish(0xffffu);
        nbr_count[row] = list.count | (direct << 16);
        if (list.count > r.width)
        {
            atomicOr(status_flags, kOverflow);
        }
    }
    __syncthreads();
}

// One list entry's pair term, added to the center's sums (an exact zero outside the cutoff).
// With kImage the displacement takes the minimum image; without, it is the plain difference,
// which is what the minimum image gives a direct entry (see rebuild_replica): the entry was
// within the list radius with no image at the rebuild, neither atom has moved half the skin
// since, and the period is more than twice the radius plus the skin on a grid.
template <bool kEnergy, bool kImage>
__device__ __forceinline__ void serve_pair(const ReplicaScalars& r, const Pos4<float>& me,
                                           const Pos4<float>& p, float& fx, float& fy, float& fz,
                                           float& esum, float& inside_count)
{
    const float dx = kImage ? min_image(me.x, p.x, r.cell[0]) : me.x - p.x;
    const float dy = kImage ? min_image(me.y, p.y, r.cell[1]) : me.y - p.y;
    const float dz = kImage ? min_image(me.z, p.z, r.cell[2]) : me.z - p.z;
    const float r2 = squared_norm(dx, dy, dz);
    const float mask = r2 < r.cutoff_squared ? 1.0f : 0.0f;
    const float inv_r2 = fast_reciprocal(r2);
    const float q = r.lj.s2 * inv_r2;
    const float p6 = q * q * q;
    const float fs = mask * (inv_r2 * (p6 * fmaf(2.0f, p6, -1.0f)));
    if (kEnergy)
    {
        esum = fmaf(mask, fmaf(p6, p6, -p6), esum);
        inside_count += mask;
    }
    fx = fmaf(fs, dx, fx);
    fy = fmaf(fs, dy, fy);
    fz = fmaf(fs, dz, fz);
}

// The eight entries of one list word.
template <bool kEnergy, bool kImage>
__device__ __forceinline__ void serve_chunk(const ReplicaScalars& r, const Pos4<float>* pos,
                                            const Pos4<float>& me, const uint4& word, float& fx,
                                            float& fy, float& fz, float& esum,
                                            float& inside_count)
{
    const unsigned packed[4] = {word.x, word.y, word.z, word.w};
#pragma unroll
    for (int k = 0; k < kChunk; ++k)
    {
        const Pos4<float> p = pos[(packed[k / 2] >> (16 * (k % 2))) & 0xffffu];
        serve_pair<kEnergy, kImage>(r, me, p, fx, fy, fz, esum, inside_count);
    }
}

// Forces at the current positions; with `kKick`, also the second half kick, leaving K of every
// 32 rows in kinetic_sums[row / 32] (float64); with `kEnergy`, their E in energy_sums (a step
// needs E only when its energy is reported: the last step of a round). Whole chunks of the list
// go through without a bound check; only the last, partial chunk checks the count.
template <bool kKick, bool kEnergy>
__device__ void replica_forces(const Team& team, const ReplicaScalars& r, const Pos4<float>* pos,
                               float* vel, float* force, const float* mass, const float* inv_mass,
                               const std::uint16_t* nbr, const index_t* nbr_count,
                               const index_t* order, double* kinetic_sums, double* energy_sums)
{
    for (int row = team.first(); row - static_cast<int>(threadIdx.x) % kWarp < r.n;
         row += team.stride())
    {
        double kinetic = 0, energy = 0;  // of this row
        const unsigned active = __ballot_sync(kFullMask, row < r.n);
        if (row < r.n)
        {
            const int i = order != nullptr ? order[row] : row;  // the list row's atom
            const Pos4<float> me = pos[i];
            const int listed = nbr_count[row] & 0xffff;
            const int count = listed < r.width ? listed : r.width;
            const uint4* chunks =
                reinterpret_cast<const uint4*>(nbr) + chunk_index(row, 0, r.width);
            // The kick's inputs are loaded before the pairs, so their latency hides behind them.
            float v[3] = {0.0f, 0.0f, 0.0f}, w = 0.0f, m = 0.0f;
            if (kKick)
            {
                const float* vi = vel + 3LL * i;
                v[0] = vi[0];
                v[1] = vi[1];
                v[2] = vi[2];
                w = inv_mass[i];
                m = mass[i];
            }
            float fx = 0, fy = 0, fz = 0, esum = 0, inside_count = 0;
            const int full = count / kChunk;
            const int chunk_count = (count + kChunk - 1) / kChunk;
            // The whole words of direct entries come first; the word that holds the last direct
            // entry and every later one take the minimum image (which gives a direct entry the
            // same bits as the plain difference).
            const int direct_words = min((nbr_count[row] >> 16) / kChunk, full);
            // Each chunk's word is loaded one chunk ahead: a pool's lists are far larger than L2,
            // so a word comes from DRAM, and its latency now overlaps the previous chunk's pairs.
            uint4 next = chunk_count > 0 ? chunks[0] : make_uint4(0, 0, 0, 0);
            auto advance = [&](int chunk) {
                const uint4 word = next;
                if (chunk + 1 < chunk_count)
                {
                    next = chunks[static_cast<std::int64_t>(chunk + 1) * kWarp];
                }
                return word;
            };
            // One vote per word keeps the choice uniform over the warp, whose rows are the atoms of
            // one or two cells: the plain difference when every lane's word is direct.
            const int warp_full = __reduce_max_sync(active, full);
            for (int chunk = 0; chunk < warp_full; ++chunk)
            {
                const bool mine = chunk < full;
                const bool direct = __all_sync(active, !mine || chunk < direct_words);
                if (mine)
                {
                    const uint4 word = advance(chunk);
                    if (direct)
                    {
                        serve_chunk<kEnergy, false>(r, pos, me, word, fx, fy, fz, esum,
                                                    inside_count);
                    }
                    else
                    {
                        serve_chunk<kEnergy, true>(r, pos, me, word, fx, fy, fz, esum,
                                                   inside_count);
                    }
                }
            }
            if (full < chunk_count)
            {
                const unsigned packed[4] = {next.x, next.y, next.z, next.w};
#pragma unroll
                for (int k = 0; k < kChunk; ++k)
                {
                    if (full * kChunk + k < count)
                    {
                        const Pos4<float> p = pos[(packed[k / 2] >> (16 * (k % 2))) & 0xffffu];
                        serve_pair<kEnergy, true>(r, me, p, fx, fy, fz, esum, inside_count);
                    }
                }
            }
            fx *= r.lj.e24;
            fy *= r.lj.e24;
            fz *= r.lj.e24;
            if (kEnergy)
            {
                energy = 0.5 * (double(r.lj.e4) * esum - double(r.lj.shift) * inside_count);
            }
            float* f = force + 3LL * i;
            f[0] = fx;
            f[1] = fy;
            f[2] = fz;
            if (kKick)
            {
                const float kick = r.half_dt * w;
                const float vx = fmaf(kick, fx, v[0]);
                const float vy = fmaf(kick, fy, v[1]);
                const float vz = fmaf(kick, fz, v[2]);
                float* vi = vel + 3LL * i;
                vi[0] = vx;
                vi[1] = vy;
                vi[2] = vz;
                kinetic = 0.5 * double(m) * (double(vx) * vx + double(vy) * vy + double(vz) * vz);
            }
        }
        __syncwarp();
        if (kKick)
        {
            kinetic = warp_sum(kinetic);
        }
        if (kEnergy)
        {
            energy = warp_sum(energy);
        }
        if (threadIdx.x % kWarp == 0)
        {
            if (kKick)
            {
                kinetic_sums[row / kWarp] = kinetic;
            }
            if (kEnergy)
            {
                energy_sums[row / kWarp] = energy;
            }
        }
    }
}

// The sum of `units` values in an order that depends on their number only; every thread gets it.
__device__ double sum_units(const double* values, int units, double* warp_sums)
{
    double sum = 0;
    for (int u = threadIdx.x; u < units; u += kServeThreads)
    {
        sum += values[u];
    }
    return block_sum(sum, warp_sums);
}

// mode 0: wrap, rebuild and the first forces of newly admitted replicas. mode 1: run each
// listed replica for min(budget, steps left) NVT steps. One CTA per SM, up to 128 registers a
// thread: held to two CTAs (64 registers) the kernel spills, and measured slower.
//
// `team_ctas` CTAs (one cluster) per replica; those past a CTA per kServeTeamAtoms atoms leave
// at once. One 512-thread CTA takes 1.4 ms a step of a 16,384-atom replica, whatever else the
// GPU has to do, so the largest replicas of a batch outlast the rest on a nearly idle GPU; a
// team divides the rows of every phase but the cell sort. Every CTA keeps the chain's state and
// closes it from the same sums; a step costs two cluster barriers, a rebuild three more. Every
// branch around a barrier is decided from values that all CTAs read after the same barrier.
// 512 replicas of 64 to 16,384 atoms, 100 steps each: 192 ms on the GPU with one CTA each,
// 118 ms with the teams the server picks (98 ms with the candidate scan as it is now).
__global__ void __launch_bounds__(kServeThreads, 1) serve_kernel(ServePool p, const int* slots,
                                                              const int* budgets, int mode,
                                                              int team_ctas)
{
    __shared__ ReplicaScalars r;
    __shared__ double thermo[kThermoSize];
    __shared__ __align__(16) int counts[kServeMaxCells + 4];
    __shared__ int moved_slots[kServeTeam];  // by rank: the last step that moved an atom too far
    __shared__ int bad_slots[kServeTeam];    // a coordinate is not finite
    __shared__ int flag_slots[kServeTeam];   // the rebuild's status bits
    __shared__ double warp_sums[kServeWarps];
    __shared__ float scales[2];
    __shared__ int flags;
    __shared__ int warp_totals[kServeWarps];
    const int entry = static_cast<int>(blockIdx.x) / team_ctas;
    nd_replica* replica = p.replicas + slots[entry];
    Team team;
    team.rank = static_cast<int>(blockIdx.x) % team_ctas;
    team.size = min(team_ctas, max(1, replica->num_atoms / kServeTeamAtoms));
    if (team.rank >= team.size)
    {
        return;
    }
    if (threadIdx.x < kServeTeam)
    {
        moved_slots[threadIdx.x] = bad_slots[threadIdx.x] = flag_slots[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0)
    {
        r.n = replica->num_atoms;
        r.width = replica->width;
        r.cells = 1;
        for (int a = 0; a < 3; ++a)
        {
            r.dims[a] = replica->dims[a];
            r.cells *= replica->dims[a];
            r.cell[a] = replica->cell[a];
            r.widths[a] = replica->widths[a];
        }
        r.cutoff_squared = replica->cutoff * replica->cutoff;
        r.radius_squared = replica->radius * replica->radius;
        r.threshold_squared = replica->threshold_squared;
        r.dt = replica->timestep;
        r.half_dt = 0.5f * replica->timestep;
        r.lj = pair_params(replica->sigma, replica->epsilon, r.cutoff_squared);
        r.status = replica->status;
        r.rebuild_count = replica->rebuild_count;
        r.steps_left = replica->steps_left;
        flags = 0;
    }
    for (int k = threadIdx.x; k < kThermoSize; k += kServeThreads)
    {
        thermo[k] = replica->thermostat[k];
    }
    __syncthreads();
    const std::int64_t a0 = replica->atom_offset;
    Pos4<float>* pos = p.pos + a0;
    Pos4<float>* ref = p.ref_pos + a0;
    float* vel = p.vel + 3 * a0;
    float* force = p.force + 3 * a0;
    const float* mass = p.mass + a0;
    const float* inv_mass = p.inv_mass + a0;
    long long* images = p.images + 3 * a0;
    std::uint16_t* nbr = p.nbr + replica->list_offset;
    index_t* nbr_count = p.nbr_count + a0;
    index_t* sorted = p.sorted + a0;
    index_t* scratch = p.scratch + a0;
    index_t* cell_start = p.cell_start + replica->cell_offset;
    Pos4<float>* ordered = p.ordered + a0;
    // List rows follow the cell order on a grid (set by every rebuild), else the atoms.
    const bool grid = r.dims[0] >= 3 && r.dims[1] >= 3 && r.dims[2] >= 3;
    const index_t* order = grid ? sorted : nullptr;
    // The sums of every 32 rows: in the cell counts' shared memory when one CTA owns the replica
    // and they fit, else in the rebuild's scratch array (both idle outside a rebuild), from its
    // first 8-byte boundary on: a replica's room may begin at any atom.
    const int units = (r.n + kWarp - 1) / kWarp;
    const bool in_shared = team.size == 1 && 2 * units * sizeof(double) <= sizeof(counts);
    auto* aligned = reinterpret_cast<double*>(
        (reinterpret_cast<std::uintptr_t>(scratch) + 7u) & ~std::uintptr_t{7});
    double* kinetic_sums = in_shared ? reinterpret_cast<double*>(counts) : aligned;
    double* energy_sums = kinetic_sums + units;
    // The team's status bits from every CTA's slot.
    auto told = [&](const int* slots_by_rank) {
        int bits = 0;
        for (int k = 0; k < team.size; ++k)
        {
            bits |= slots_by_rank[k];
        }
        return bits;
    };
    if (team.size > 1)
    {
        team.sync();  // every CTA has read the replica and set its slots
    }

    if (mode == 0)
    {
        rebuild_replica(team, r, pos, ref, images, nbr, nbr_count, sorted, scratch, cell_start,
                        ordered, counts, warp_totals, &flags);
        team.tell(flag_slots, flags);
        replica_forces<false, true>(team, r, pos, vel, force, mass, inv_mass, nbr, nbr_count,
                                    order, kinetic_sums, energy_sums);
        team.sync();
        const double energy = sum_units(energy_sums, units, warp_sums);
        if (threadIdx.x == 0 && team.rank == 0)
        {
            replica->status = r.status | told(flag_slots);
            replica->rebuild_count = r.rebuild_count + 1;
            replica->energy = energy;
        }
        return;
    }
    const int budget = budgets[entry] < r.steps_left ? budgets[entry] : r.steps_left;
    int done = 0;
    double last_energy = replica->energy;  // thread 0's copy
    for (; done < budget; ++done)
    {
        if (r.status != 0)
        {
            break;
        }
        if (threadIdx.x == 0)
        {
            // The opening chain half step; the previous closing factor is still pending.
            double kinetic = thermo[kKineticA];
            double q[3], pc[3];
            for (int k = 0; k < 3; ++k)
            {
                q[k] = thermo[kChainA + k];
                pc[k] = thermo[kChainA + 3 + k];
            }
            const double factor = chain_half_step(kinetic, q, pc, thermo + kChainMass,
                                                  thermo[kDegrees], thermo[kThermalEnergy],
                                                  thermo[kTimestep]);
            scales[0] = static_cast<float>(thermo[kPendingScale]);
            scales[1] = static_cast<float>(factor);
            for (int k = 0; k < 3; ++k)
            {
                thermo[kChainB + k] = q[k];
                thermo[kChainB + 3 + k] = pc[k];
            }
        }
        __syncthreads();
        int moved = 0, bad = 0;
        for (int i = team.first(); i < r.n; i += team.stride())
        {
            float* v = vel + 3LL * i;
            const float* f = force + 3LL * i;
            const float kick = r.half_dt * inv_mass[i];
            const float vx = fmaf(kick, f[0], (v[0] * scales[0]) * scales[1]);
            const float vy = fmaf(kick, f[1], (v[1] * scales[0]) * scales[1]);
            const float vz = fmaf(kick, f[2], (v[2] * scales[0]) * scales[1]);
            v[0] = vx;
            v[1] = vy;
            v[2] = vz;
            Pos4<float> x = pos[i];
            x.x = fmaf(r.dt, vx, x.x);
            x.y = fmaf(r.dt, vy, x.y);
            x.z = fmaf(r.dt, vz, x.z);
            pos[i] = x;
            bad |= !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z));
            const Pos4<float> x0 = ref[i];
            moved |= squared_norm(x.x - x0.x, x.y - x0.y, x.z - x0.z) >= r.threshold_squared;
        }
        bad = __syncthreads_or(bad);
        moved = __syncthreads_or(moved);
        if (team.size > 1)
        {
            team.tell(bad_slots, bad);
            team.tell(moved_slots, moved ? done + 1 : 0);
            team.sync();
            bad = told(bad_slots);
            moved = 0;
            for (int k = 0; k < team.size; ++k)
            {
                moved |= moved_slots[k] == done + 1;
            }
        }
        if (bad)
        {
            if (threadIdx.x == 0)
            {
                r.status |= kNonFinite;
            }
            __syncthreads();
            break;
        }
        if (moved)
        {
            rebuild_replica(team, r, pos, ref, images, nbr, nbr_count, sorted, scratch,
                            cell_start, ordered, counts, warp_totals, &flags);
            team.tell(flag_slots, flags);
            if (threadIdx.x == 0)
            {
                ++r.rebuild_count;
            }
        }
        const bool reported = done + 1 == budget;  // the round's last step reports its energy
        if (reported)
        {
            replica_forces<true, true>(team, r, pos, vel, force, mass, inv_mass, nbr, nbr_count,
                                       order, kinetic_sums, energy_sums);
        }
        else
        {
            replica_forces<true, false>(team, r, pos, vel, force, mass, inv_mass, nbr, nbr_count,
                                        order, kinetic_sums, energy_sums);
        }
        team.sync();
        double kinetic = sum_units(kinetic_sums, units, warp_sums);
        const double energy = reported ? sum_units(energy_sums, units, warp_sums) : 0.0;
        if (threadIdx.x == 0)
        {
            r.status |= told(flag_slots);
            if (reported)
            {
                last_energy = energy;
            }
            // The closing chain half step against this step's K.
            double q[3], pc[3];
            for (int k = 0; k < 3; ++k)
            {
                q[k] = thermo[kChainB + k];
                pc[k] = thermo[kChainB + 3 + k];
            }
            const double factor = chain_half_step(kinetic, q, pc, thermo + kChainMass,
                                                  thermo[kDegrees], thermo[kThermalEnergy],
                                                  thermo[kTimestep]);
            for (int k = 0; k < 3; ++k)
            {
                thermo[kChainA + k] = q[k];
                thermo[kChainA + 3 + k] = pc[k];
            }
            thermo[kKineticA] = kinetic;
            thermo[kPendingScale] = factor;
        }
        __syncthreads();
    }
    if (team.rank != 0)
    {
        return;  // the first CTA's copy of the state is everyone's
    }
    for (int k = threadIdx.x; k < kThermoSize; k += kServeThreads)
    {
        replica->thermostat[k] = thermo[k];
    }
    if (threadIdx.x == 0)
    {
        replica->steps_left = r.steps_left - done;
        replica->status = r.status;
        replica->rebuild_count = r.rebuild_count;
        replica->energy = last_energy;
    }
}

// Frames of newly admitted replicas into the pool, a CTA per replica: float32 positions and
// masses, velocities with the center of mass taken out in float64 before the rounding, zero
// forces and images, and the slot's record with the kinetic energy of the rounded velocities.
// Bound by the 56 B read per atom (twice: the second pass hits L2). It replaces the conversion
// on the host, 95 ms of one core for 512 replicas (1.5 million atoms) before the first launch;
// the host now copies the arrays as they are, and this kernel takes 0.1 ms a batch.
__global__ void __launch_bounds__(kServeThreads)
    admit_kernel(ServePool p, const nd_replica* records, const int* slots,
                 const std::int64_t* starts, const double* positions, const double* velocities,
                 const double* masses)
{
    __shared__ double warp_sums[kServeWarps];
    const nd_replica* record = records + blockIdx.x;
    const int n = record->num_atoms;
    const std::int64_t a0 = record->atom_offset, first = starts[blockIdx.x];
    const double* x = positions + 3 * first;
    const double* v = velocities + 3 * first;
    const double* m = masses + first;
    double momentum[3] = {0, 0, 0}, total = 0;
    for (int i = threadIdx.x; i < n; i += kServeThreads)
    {
        const double mass = m[i];
        total += mass;
        for (int a = 0; a < 3; ++a)
        {
            momentum[a] += mass * v[3 * i + a];
        }
    }
    total = block_sum(total, warp_sums);
    for (int a = 0; a < 3; ++a)
    {
        momentum[a] = block_sum(momentum[a], warp_sums) / total;  // the center's velocity
    }
    double kinetic = 0;
    for (int i = threadIdx.x; i < n; i += kServeThreads)
    {
        const std::int64_t atom = a0 + i;
        Pos4<float> position;
        position.x = static_cast<float>(x[3 * i]);
        position.y = static_cast<float>(x[3 * i + 1]);
        position.z = static_cast<float>(x[3 * i + 2]);
        position.w = 0.0f;
        p.pos[atom] = position;
        double squared = 0;
        for (int a = 0; a < 3; ++a)
        {
            const float rounded = static_cast<float>(v[3 * i + a] - momentum[a]);
            squared += double(rounded) * rounded;
            p.vel[3 * atom + a] = rounded;
            p.force[3 * atom + a] = 0.0f;
            p.images[3 * atom + a] = 0;
        }
        kinetic += m[i] * squared;
        const float mass = static_cast<float>(m[i]);
        p.mass[atom] = mass;
        p.inv_mass[atom] = 1.0f / mass;
    }
    kinetic = 0.5 * block_sum(kinetic, warp_sums);
    constexpr int kWords = sizeof(nd_replica) / sizeof(std::uint64_t);
    constexpr int kKineticWord =
        offsetof(nd_replica, thermostat) / sizeof(std::uint64_t) + kKineticA;
    static_assert(sizeof(nd_replica) % sizeof(std::uint64_t) == 0 && kWords <= kServeThreads,
                  "a thread copies a word of the record");
    if (threadIdx.x < kWords)
    {
        const std::uint64_t word = reinterpret_cast<const std::uint64_t*>(record)[threadIdx.x];
        reinterpret_cast<std::uint64_t*>(p.replicas + slots[blockIdx.x])[threadIdx.x] =
            threadIdx.x == kKineticWord
                ? static_cast<std::uint64_t>(__double_as_longlong(kinetic))
                : word;
    }
}

// Frames of finished replicas, a CTA per replica, from row starts[k] on: the positions wrapped
// with every product rounded by itself (as wrap_separately), the images with those crossings,
// the velocities with the pending chain factor applied. One pass where about twenty elementwise
// launches read three uploaded per-atom arrays (harvests of 512 replicas: 70 -> 15 ms of the
// host's time).
__global__ void __launch_bounds__(kServeThreads)
    harvest_kernel(ServePool p, const nd_replica* records, const std::int64_t* starts,
                   float* positions, float* velocities, std::int64_t* images)
{
    const nd_replica* record = records + blockIdx.x;
    const int n = record->num_atoms;
    const std::int64_t a0 = record->atom_offset, first = starts[blockIdx.x];
    const float scale = static_cast<float>(record->thermostat[kPendingScale]);
    const float cell[3] = {record->cell[0], record->cell[1], record->cell[2]};
    for (int i = threadIdx.x; i < n; i += kServeThreads)
    {
        const Pos4<float> position = p.pos[a0 + i];
        const float x[3] = {position.x, position.y, position.z};
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            float crossings = floorf(x[a] / cell[a]);
            float wrapped = x[a] - __fmul_rn(crossings, cell[a]);
            if (wrapped < 0.0f)
            {
                wrapped += cell[a];
                crossings -= 1.0f;
            }
            if (wrapped >= cell[a])
            {
                wrapped -= cell[a];
                crossings += 1.0f;
            }
            const std::int64_t from = 3 * (a0 + i) + a, to = 3 * (first + i) + a;
            positions[to] = wrapped;
            velocities[to] = p.vel[from] * scale;
            images[to] = p.images[from] + static_cast<long long>(crossings);
        }
    }
}

bool pool_of(const nd_replica_pool* pool, ServePool& p)
{
    if (!(pool->replicas && pool->positions && pool->velocities && pool->forces &&
          pool->masses && pool->inverse_masses && pool->images && pool->reference_positions &&
          pool->neighbors && pool->neighbor_counts && pool->sorted && pool->scratch &&
          pool->cell_starts && pool->ordered_positions))
    {
        return false;
    }
    p.replicas = pool->replicas;
    p.pos = static_cast<Pos4<float>*>(pool->positions);
    p.vel = static_cast<float*>(pool->velocities);
    p.force = static_cast<float*>(pool->forces);
    p.mass = static_cast<float*>(pool->masses);
    p.inv_mass = static_cast<float*>(pool->inverse_masses);
    p.images = reinterpret_cast<long long*>(pool->images);
    p.ref_pos = static_cast<Pos4<float>*>(pool->reference_positions);
    p.nbr = pool->neighbors;
    p.nbr_count = pool->neighbor_counts;
    p.sorted = pool->sorted;
    p.scratch = pool->scratch;
    p.cell_start = pool->cell_starts;
    p.ordered = static_cast<Pos4<float>*>(pool->ordered_positions);
    return true;
}

}  // namespace nd

extern "C" int nd_serve_run(const nd_replica_pool* pool, const int32_t* slots,
                            const int32_t* budgets, int32_t count, int32_t mode,
                            nd_stream_t stream)
{
    return nd_serve_run_teams(pool, slots, budgets, count, mode, 1, stream);
}

extern "C" int nd_serve_run_teams(const nd_replica_pool* pool, const int32_t* slots,
                                  const int32_t* budgets, int32_t count, int32_t mode,
                                  int32_t team, nd_stream_t stream)
{
    ND_REQUIRE(team == 1 || team == 2 || team == 4 || team == nd::kServeTeam,
               "a team is 1, 2, 4 or 8 CTAs");
    ND_REQUIRE(pool != nullptr && slots != nullptr, "the pool or the slot list is null");
    ND_REQUIRE(mode == 0 || (mode == 1 && budgets != nullptr), "mode is 0 (admit) or 1 (run)");
    ND_REQUIRE(count >= 0 && count <= 1 << 20, "count out of range");
    nd::ServePool p;
    ND_REQUIRE(nd::pool_of(pool, p), "a pool buffer is null");
    if (count == 0)
    {
        return ND_OK;
    }
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(count) * static_cast<unsigned>(team));
    config.blockDim = dim3(nd::kServeThreads);
    config.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = static_cast<unsigned>(team);
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = team > 1 ? 1 : 0;
    ND_CUDA_TRY(cudaLaunchKernelEx(&config, nd::serve_kernel, p, slots, budgets,
                                   static_cast<int>(mode), static_cast<int>(team)));
    return ND_OK;
}

extern "C" int nd_serve_admit(const nd_replica_pool* pool, const nd_replica* records,
                              const int32_t* slots, const int64_t* starts,
                              const double* positions, const double* velocities,
                              const double* masses, int32_t count, nd_stream_t stream)
{
    ND_REQUIRE(pool != nullptr, "the pool is null");
    ND_REQUIRE(count >= 0 && count <= 1 << 20, "count out of range");
    nd::ServePool p;
    ND_REQUIRE(nd::pool_of(pool, p), "a pool buffer is null");
    if (count == 0)
    {
        return ND_OK;
    }
    ND_REQUIRE(records && slots && starts && positions && velocities && masses,
               "an admission buffer is null");
    nd::admit_kernel<<<count, nd::kServeThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        p, records, slots, starts, positions, velocities, masses);
    ND_CUDA_TRY(cudaGetLastError());
    return ND_OK;
}

extern "C" int nd_serve_harvest(const nd_replica_pool* pool, const nd_replica* records,
                                const int64_t* starts, int32_t count, float* positions,
                                float* velocities, int64_t* images, nd_stream_t stream)
{
    ND_REQUIRE(pool != nullptr, "the pool is null");
    ND_REQUIRE(count >= 0 && count <= 1 << 20, "count out of range");
    nd::ServePool p;
    ND_REQUIRE(nd::pool_of(pool, p), "a pool buffer is null");
    if (count == 0)
    {
        return ND_OK;
    }
    ND_REQUIRE(records && starts && positions && velocities && images,
               "a harvest buffer is null");
    nd::harvest_kernel<<<count, nd::kServeThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        p, records, starts, positions, velocities, images);
    ND_CUDA_TRY(cudaGetLastError());
    return ND_OK;
}
