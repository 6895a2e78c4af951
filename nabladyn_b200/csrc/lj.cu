// Lennard-Jones energy, forces, virial (and parameter gradients) over a [2, C] pair index,
// the NeighborPairs contract of src/nabladyn/neighbors/_pairs.py:8-22.
//
// It restates src/nabladyn/potential/_lennard_jones/_potential.py:209-234 with the
// derivatives written out instead of taken by torch.func (src/nabladyn/quantity.py:160-184):
// for a valid column (i != j, r^2 < r_c^2) with p6 = (sigma^2 / r^2)^3,
//     u   = 4 eps (p6^2 - p6) - u_c,                  u_c = u at r_c, unshifted,
//     f_s = 24 eps (2 p6^2 - p6) / r^2,               F_i += f_s d, F_j -= f_s d,
//     W  += f_s d (x) d,                               (W = -dE/dstrain at zero strain)
//     dE/deps   += 4 (p6^2 - p6) - 4 (pc6^2 - pc6),
//     dE/dsigma += 24 eps / sigma (2 p6^2 - p6 - 2 pc6^2 + pc6),
// with d the minimum-image vector x_i - x_j of src/nabladyn/space.py:11-19. Under a strain
// eps_s (src/nabladyn/space.py:51-64) every vector is deformed first, d' = (I + eps_s) d; then
// F_i = f_s (I + eps_s)^T d' and W_ab = f_s d'_a d_b, the derivatives of the strained energy.
//
// One pass computes everything; pair arithmetic runs in the positions' dtype and the totals
// (E, W, parameter gradients) are reduced in float64: per-thread partials, warp shuffles,
// one float64 atomic per block.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "geometry.cuh"

namespace nd {

constexpr int kLJThreads = 256;
constexpr int kMaxRows = 36;  // T(T+1)/2 rows for up to 8 atom types

// The minimum-image vector left - right for coordinates in [0, L): the far coordinate moves
// by L first (src/nabladyn/space.py:11-19).
template <typename T>
__device__ __forceinline__ T displacement(T left, T right, T length)
{
    const T raw = left - right;
    const T half = T(0.5) * length;
    const T left_shift = raw > half ? length : T(0);
    const T right_shift = raw < -half ? length : T(0);
    return (left - left_shift) - (right - right_shift);
}

// Positions [F, N, 3] wrapped into [0, L) by their frame's cell, in one pass instead of the
// dozen elementwise ones of space.wrap.
template <typename T>
__global__ void __launch_bounds__(kThreads) wrap_kernel(
    const T* __restrict__ positions, const T* __restrict__ cells, std::int64_t num_atoms,
    std::int64_t values, T* __restrict__ wrapped)
{
    const std::int64_t k = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < values)
    {
        wrapped[k] = wrap_separately(positions[k], cells[k / (3 * num_atoms) * 3 + k % 3]);
    }
}

__device__ __forceinline__ int pair_row(int a, int b, int num_types)
{
    const int low = a < b ? a : b;
    const int high = a < b ? b : a;
    return low * (2 * num_types - low - 1) / 2 + high;
}

template <typename T>
struct LJAccumulators
{
    T energy = 0;
    T w[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // row-major W
};

// Block sums of `count` per-thread values in float64, one atomic per block into out[k].
template <int kCount>
__device__ __forceinline__ void add_block_sums(double (&values)[kCount], double* const (&out)[kCount])
{
    __shared__ double partial[kCount][kLJThreads / kWarp];
    const int lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
#pragma unroll
    for (int k = 0; k < kCount; ++k)
    {
        values[k] = warp_sum(values[k]);
        if (lane == 0)
        {
            partial[k][warp] = values[k];
        }
    }
    __syncthreads();
    if (warp == 0)
    {
#pragma unroll
        for (int k = 0; k < kCount; ++k)
        {
            double v = lane < kLJThreads / kWarp ? partial[k][lane] : 0.0;
            v = warp_sum(v);
            if (lane == 0)
            {
                atomicAdd(out[k], v);
            }
        }
    }
}

// One frame with a strain, or with the energy's parameter gradients (the model's own energy
// under autograd): one column per thread, scalar atomics. Calls without either run
// lj_frames_kernel below.
template <typename T, bool kParameterGrads, bool kStrained>
__global__ void __launch_bounds__(kLJThreads) lj_pairs_kernel(
    const T* __restrict__ positions,
    const T* __restrict__ cell,
    const index_t* __restrict__ pairs,
    std::int64_t capacity,
    index_t num_atoms,
    const index_t* __restrict__ atom_types,  // null: one type
    int num_types,
    const T* __restrict__ sigma,
    const T* __restrict__ epsilon,
    const T* __restrict__ strain,
    T cutoff_squared,
    double* __restrict__ energy,
    T* __restrict__ forces,
    double* __restrict__ virial,
    double* __restrict__ sigma_grad,
    double* __restrict__ epsilon_grad
)
{
    const int rows = num_types * (num_types + 1) / 2;
    __shared__ double row_grads[2 * kMaxRows];
    if (kParameterGrads)
    {
        for (int k = threadIdx.x; k < 2 * rows; k += blockDim.x)
        {
            row_grads[k] = 0.0;
        }
        __syncthreads();
    }
    const T lx = cell[0], ly = cell[1], lz = cell[2];
    T e[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (kStrained)
    {
#pragma unroll
        for (int k = 0; k < 9; ++k)
        {
            e[k] = strain[k];
        }
    }
    LJAccumulators<T> acc;
    const std::int64_t stride = static_cast<std::int64_t>(gridDim.x) * blockDim.x;
    for (std::int64_t column = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
         column < capacity; column += stride)
    {
        const index_t i = pairs[column];
        const index_t j = pairs[capacity + column];
        // Self-pairs are padding; an index outside [0, N) is skipped, never read.
        if (i == j || static_cast<unsigned>(i) >= static_cast<unsigned>(num_atoms) ||
            static_cast<unsigned>(j) >= static_cast<unsigned>(num_atoms))
        {
            continue;
        }
        const T ux = displacement(positions[3LL * i], positions[3LL * j], lx);
        const T uy = displacement(positions[3LL * i + 1], positions[3LL * j + 1], ly);
        const T uz = displacement(positions[3LL * i + 2], positions[3LL * j + 2], lz);
        T dx = ux, dy = uy, dz = uz;
        if (kStrained)
        {
            dx = ux + ux * e[0] + uy * e[1] + uz * e[2];
            dy = uy + ux * e[3] + uy * e[4] + uz * e[5];
            dz = uz + ux * e[6] + uy * e[7] + uz * e[8];
        }
        const T r2 = dx * dx + dy * dy + dz * dz;
        if (!(r2 < cutoff_squared))
        {
            continue;
        }
        const int row = atom_types == nullptr ? 0 : pair_row(atom_types[i], atom_types[j], num_types);
        const T s = sigma[row];
        const T eps = epsilon[row];
        const T s2 = s * s;
        const T inv_r2 = T(1) / r2;
        const T q = s2 * inv_r2;
        const T p6 = q * q * q;
        const T qc = s2 / cutoff_squared;
        const T pc6 = qc * qc * qc;
        const T shift = T(4) * eps * (pc6 * pc6 - pc6);
        acc.energy += T(4) * eps * (p6 * p6 - p6) - shift;
        const T fs = T(24) * eps * (T(2) * p6 * p6 - p6) * inv_r2;
        T fx = fs * dx, fy = fs * dy, fz = fs * dz;
        if (kStrained)
        {
            acc.w[0] += fx * ux;
            acc.w[1] += fx * uy;
            acc.w[2] += fx * uz;
            acc.w[3] += fy * ux;
            acc.w[4] += fy * uy;
            acc.w[5] += fy * uz;
            acc.w[6] += fz * ux;
            acc.w[7] += fz * uy;
            acc.w[8] += fz * uz;
            // The force on the undeformed positions: (I + eps_s)^T f.
            const T gx = fx + e[0] * fx + e[3] * fy + e[6] * fz;
            const T gy = fy + e[1] * fx + e[4] * fy + e[7] * fz;
            const T gz = fz + e[2] * fx + e[5] * fy + e[8] * fz;
            fx = gx;
            fy = gy;
            fz = gz;
        }
        else
        {
            acc.w[0] += fx * dx;
            acc.w[4] += fy * dy;
            acc.w[8] += fz * dz;
            acc.w[1] += fx * dy;
            acc.w[2] += fx * dz;
            acc.w[5] += fy * dz;
        }
        atomicAdd(forces + 3LL * i, fx);
        atomicAdd(forces + 3LL * i + 1, fy);
        atomicAdd(forces + 3LL * i + 2, fz);
        atomicAdd(forces + 3LL * j, -fx);
        atomicAdd(forces + 3LL * j + 1, -fy);
        atomicAdd(forces + 3LL * j + 2, -fz);
        if (kParameterGrads)
        {
            const double de = 4.0 * (double(p6) * p6 - p6) - 4.0 * (double(pc6) * pc6 - pc6);
            const double ds = 24.0 * double(eps) / double(s) *
                              (2.0 * double(p6) * p6 - p6 - 2.0 * double(pc6) * pc6 + pc6);
            atomicAdd(row_grads + row, ds);
            atomicAdd(row_grads + rows + row, de);
        }
    }
    // Block totals in float64: warp shuffles, then one warp over the per-warp sums. Without a
    // strain only the upper triangle was accumulated; the lower one mirrors it.
    if (!kStrained)
    {
        acc.w[3] = acc.w[1];
        acc.w[6] = acc.w[2];
        acc.w[7] = acc.w[5];
    }
    double values[10];
    values[0] = double(acc.energy);
#pragma unroll
    for (int k = 0; k < 9; ++k)
    {
        values[k + 1] = double(acc.w[k]);
    }
    double* const out[10] = {energy, virial, virial + 1, virial + 2, virial + 3, virial + 4,
                             virial + 5, virial + 6, virial + 7, virial + 8};
    add_block_sums(values, out);
    if (kParameterGrads)
    {
        __syncthreads();
        for (int k = threadIdx.x; k < rows; k += blockDim.x)
        {
            atomicAdd(sigma_grad + k, row_grads[k]);
            atomicAdd(epsilon_grad + k, row_grads[rows + k]);
        }
    }
}

// ---------------------------------------------------------------------------------------
// E, F and W of F frames of one system, without strain or parameter gradients: the path of
// quantity.energy_force_virial and of the training predictions.
//
// What bounds it is the force scatter and the position gathers through L2, not the index
// stream: one column costs two gathered atoms and two scattered forces, 48 B of L2 traffic
// each way against 8 B of index. So:
//   * atoms are gathered as packed (x, y, z, type) slots, one 16-B load each instead of three
//     scalar ones and a type load; the pass that packs them wraps them too;
//   * float32 forces are summed into packed [N, 4] slots, one 16-B vector atomic per atom
//     instead of three scalar ones, and unpacked by the closing pass (float64 has no vector
//     atomic and adds its three components in place);
//   * a warp takes 128 consecutive columns. The list groups its columns by first atom (about
//     60 columns each in a liquid), so the pair forces pass through shared memory into four
//     consecutive columns per lane, a lane sums its first atom's force in registers, the
//     lanes that end on the same first atom meet in a segmented warp sum, and a first atom
//     costs two or three atomics instead of one per column. An index in any other order gives
//     the same sums with more atomics.
// Measured, float32, the whole call: 1,048,576 atoms (64 million columns) 1,765 -> 428 us, 415 of it
// this kernel; step by step 587 with packing and wide atomics, 525 with a column per lane in the
// gathers and atomics, 432 with 16-byte reads of the staged forces and padding skipped. 27,000
// atoms of two types 165 -> 47 us; 512 atoms in float64 150 -> 47 us. At the largest the L1 pipe
// is busy 79 % of the time (gathers and atomics of lines that are random in memory), issue 67 %.

// Blocks an SM holds: the registers of four columns in flight, 80 (float32) or 124 (float64).
template <typename T>
constexpr int kFrameBlocksPerSM = sizeof(T) == 4 ? 3 : 2;

constexpr int kLaneColumns = 4;  // columns a lane has in flight
constexpr int kWarpColumns = kWarp * kLaneColumns;

// An atom as the kernels gather it; w holds the type's bits. 16-B aligned: float64 slots are
// two 16-B words.
template <typename T>
struct alignas(16) PackedAtom
{
    T x, y, z, w;
};

__device__ __forceinline__ float type_word(float, index_t type) { return __int_as_float(type); }
__device__ __forceinline__ double type_word(double, index_t type)
{
    return __longlong_as_double(static_cast<long long>(type));
}
__device__ __forceinline__ int word_type(float w) { return __float_as_int(w); }
__device__ __forceinline__ int word_type(double w)
{
    return static_cast<int>(__double_as_longlong(w));
}

constexpr int kFrameSums = 7;  // E, W xx yy zz xy xz yz
constexpr int kFrameSlots = 8;

// The workspace of a batch: float64 sums (per frame, or of the parameter rows), packed atoms,
// and packed forces (the forward's in float32, the loss's force gradients in the backward).
template <typename T>
struct FrameWorkspace
{
    std::int64_t sums, atoms, forces, total;

    FrameWorkspace(std::int64_t frames, std::int64_t num_atoms)
    {
        const std::int64_t bytes =
            (frames * num_atoms * static_cast<std::int64_t>(sizeof(PackedAtom<T>)) + 255) / 256 * 256;
        sums = 0;
        atoms = (std::max<std::int64_t>(frames * kFrameSlots, 2 * kMaxRows) * 8 + 255) / 256 * 256;
        forces = atoms + bytes;
        total = forces + bytes;
    }
};

template <typename T, bool kWrap>
__device__ __forceinline__ PackedAtom<T> packed_atom(const T* position, const T* cell,
                                                     const index_t* atom_types, index_t atom)
{
    PackedAtom<T> p{position[0], position[1], position[2],
                    type_word(T(0), atom_types == nullptr ? 0 : atom_types[atom])};
    if (kWrap)
    {
        p.x = wrap_separately(p.x, cell[0]);
        p.y = wrap_separately(p.y, cell[1]);
        p.z = wrap_separately(p.z, cell[2]);
    }
    return p;
}

// Packs the atoms (wrapped into the cell first when kWrap, in space.wrap's rounding) and sets
// the sums and the forces to zero. One thread per atom of the batch.
template <typename T, bool kWrap>
__global__ void __launch_bounds__(kThreads) pack_atoms_kernel(
    const T* __restrict__ positions, const T* __restrict__ cells,
    const index_t* __restrict__ atom_types, index_t num_atoms, std::int64_t slots,
    std::int64_t frames, PackedAtom<T>* __restrict__ atoms, float4* __restrict__ packed_forces,
    T* __restrict__ forces, double* __restrict__ sums)
{
    const std::int64_t slot = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (std::int64_t k = slot; k < frames * kFrameSlots;
         k += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
    {
        sums[k] = 0.0;
    }
    if (slot >= slots)
    {
        return;
    }
    const std::int64_t frame = slot / num_atoms;
    atoms[slot] = packed_atom<T, kWrap>(positions + 3 * slot, cells + 3 * frame, atom_types,
                                        static_cast<index_t>(slot - frame * num_atoms));
    if (packed_forces != nullptr)
    {
        packed_forces[slot] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    else
    {
        forces[3 * slot] = T(0);
        forces[3 * slot + 1] = T(0);
        forces[3 * slot + 2] = T(0);
    }
}

// Unpacks the forces (float32) and casts the sums: E [F] and W [F, 3, 3] in the frames' dtype.
template <typename T>
__global__ void __launch_bounds__(kThreads) unpack_frames_kernel(
    const float4* __restrict__ packed_forces, std::int64_t slots, std::int64_t frames,
    const double* __restrict__ sums, float* __restrict__ forces, T* __restrict__ energy,
    T* __restrict__ virial)
{
    const std::int64_t slot = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (std::int64_t k = slot; k < frames * 10;
         k += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
    {
        constexpr int place[10] = {0, 1, 4, 5, 4, 2, 6, 5, 6, 3};  // E, then W row-major
        const std::int64_t frame = k / 10;
        const int entry = static_cast<int>(k - 10 * frame);
        int from = 0;
#pragma unroll
        for (int e = 0; e < 10; ++e)
        {
            from = entry == e ? place[e] : from;
        }
        const double value = sums[kFrameSlots * frame + from];
        if (entry == 0)
        {
            energy[frame] = static_cast<T>(value);
        }
        else
        {
            virial[9 * frame + entry - 1] = static_cast<T>(value);
        }
    }
    if (packed_forces != nullptr && slot < slots)
    {
        const float4 f = packed_forces[slot];
        forces[3 * slot] = f.x;
        forces[3 * slot + 1] = f.y;
        forces[3 * slot + 2] = f.z;
    }
}

// A column counts when its atoms differ and both lie in [0, N): self-pairs are padding, an
// index outside is skipped and never read.
__device__ __forceinline__ bool counts(index_t i, index_t j, index_t num_atoms)
{
    return i != j && static_cast<unsigned>(i) < static_cast<unsigned>(num_atoms) &&
           static_cast<unsigned>(j) < static_cast<unsigned>(num_atoms);
}

// One type-pair row's constants, in the pair arithmetic's dtype.
template <typename T>
struct RowConstants
{
    T s2, eps4, eps24, shift;
};

// 1 / x. In float32 a hardware estimate and one Newton step: for normal results the bits of the
// rounded quotient (every mantissa, exponents 2^-125 to 2^125), in two operations after the
// estimate where the division takes about eight and a branch (1,048,576 atoms, the kernel: 414
// and 446 us). In float64 the division.
__device__ __forceinline__ float reciprocal(float x)
{
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(y, fmaf(-x, y, 1.0f), y);
}
__device__ __forceinline__ double reciprocal(double x) { return 1.0 / x; }

// A warp's 128 pair forces and first atoms (-1: no pair), written a column per lane and read
// four consecutive columns per lane.
template <typename T>
struct alignas(16) PairStage
{
    T x[kWarpColumns], y[kWarpColumns], z[kWarpColumns];
    index_t key[kWarpColumns];
};

// Four consecutive staged values, read 16 bytes at a time (scalar reads 16 bytes apart would
// meet in the same banks four at a time).
template <typename T>
struct alignas(16) Four
{
    T v[4];
};

template <typename T>
__device__ __forceinline__ Four<T> load4(const T* staged)
{
    return *reinterpret_cast<const Four<T>*>(staged);
}

template <typename T>
struct FramesPass
{
    const PackedAtom<T>* atoms;   // packed, or null: positions and types below
    const T* positions;
    const index_t* atom_types;    // null: one type
    const T* cells;
    const index_t* pairs;
    std::int64_t capacity;
    index_t num_atoms;
    int num_types;
    const T* sigma;
    const T* epsilon;
    T cutoff_squared;
    float4* packed_forces;        // float32 with a workspace; else the forces below
    T* forces;
    double* sums;                 // packed: [F][8]; else null and the two below
    double* energy;
    double* virial;
};

template <typename T, bool kPacked>
__device__ __forceinline__ void add_force(const FramesPass<T>& a, index_t atom, T x, T y, T z)
{
    if constexpr (kPacked && sizeof(T) == 4)
    {
        atomicAdd(a.packed_forces + atom, make_float4(x, y, z, 0.f));
    }
    else
    {
        T* f = a.forces + 3LL * atom;
        atomicAdd(f, x);
        atomicAdd(f + 1, y);
        atomicAdd(f + 2, z);
    }
}

template <typename T, bool kPacked>
__device__ __forceinline__ PackedAtom<T> gather(const FramesPass<T>& a, index_t atom)
{
    if constexpr (kPacked)
    {
        return a.atoms[atom];
    }
    else
    {
        const T* p = a.positions + 3LL * atom;
        return {p[0], p[1], p[2],
                type_word(T(0), a.atom_types == nullptr ? 0 : a.atom_types[atom])};
    }
}

// Frame blockIdx.y; its warps take runs of 128 columns in turn.
template <typename T, bool kPacked, bool kTypes>
__global__ void __launch_bounds__(kLJThreads, kFrameBlocksPerSM<T>)
lj_frames_kernel(FramesPass<T> a)
{
    const std::int64_t frame = blockIdx.y;
    if (kPacked)
    {
        a.atoms += frame * a.num_atoms;
        a.packed_forces += sizeof(T) == 4 ? frame * a.num_atoms : 0;
    }
    else
    {
        a.positions += 3 * frame * a.num_atoms;
    }
    if (!(kPacked && sizeof(T) == 4))
    {
        a.forces += 3 * frame * a.num_atoms;
    }
    a.cells += 3 * frame;
    a.pairs += 2 * frame * a.capacity;
    __shared__ RowConstants<T> rows[kTypes ? kMaxRows : 1];
    const int row_count = kTypes ? a.num_types * (a.num_types + 1) / 2 : 1;
    if (threadIdx.x < row_count)
    {
        const T s = a.sigma[threadIdx.x], eps = a.epsilon[threadIdx.x];
        const T qc = s * s / a.cutoff_squared;
        const T pc6 = qc * qc * qc;
        rows[threadIdx.x] = {s * s, T(4) * eps, T(24) * eps, T(4) * eps * (pc6 * pc6 - pc6)};
    }
    __syncthreads();
    const T lx = a.cells[0], ly = a.cells[1], lz = a.cells[2];
    const T hx = T(0.5) * lx, hy = T(0.5) * ly, hz = T(0.5) * lz;
    const int lane = threadIdx.x % kWarp;
    __shared__ PairStage<T> stages[kLJThreads / kWarp];
    PairStage<T>& stage = stages[threadIdx.x / kWarp];
    T energy = 0, wxx = 0, wyy = 0, wzz = 0, wxy = 0, wxz = 0, wyz = 0;
    // Columns are below 2^31 and the grid below 2^20 columns, so 32 bits hold every step.
    const auto capacity = static_cast<unsigned>(a.capacity);
    const index_t* firsts = a.pairs;
    const index_t* seconds = a.pairs + a.capacity;
    const unsigned stride = gridDim.x * (kLJThreads / kWarp) * kWarpColumns;
    unsigned base = (blockIdx.x * (kLJThreads / kWarp) + threadIdx.x / kWarp) * kWarpColumns;
    index_t i[kLaneColumns], j[kLaneColumns];
    auto load_columns = [&](unsigned from) {
#pragma unroll
        for (int k = 0; k < kLaneColumns; ++k)
        {
            const unsigned column = from + kWarp * k + lane;
            i[k] = column < capacity ? firsts[column] : -1;
            j[k] = column < capacity ? seconds[column] : -1;
        }
    };
    load_columns(base);
    while (base < capacity)
    {
        // All gathers of the four columns before any is used.
        PackedAtom<T> left[kLaneColumns], right[kLaneColumns];
        index_t first[kLaneColumns], second[kLaneColumns];
        bool any = false;
#pragma unroll
        for (int k = 0; k < kLaneColumns; ++k)
        {
            const bool live = counts(i[k], j[k], a.num_atoms);
            any = any || live;
            first[k] = live ? i[k] : -1;
            second[k] = live ? j[k] : 0;
        }
        const bool padding = !__any_sync(kFullMask, any);  // a fifth of a list's columns
        if (!padding)
        {
#pragma unroll
            for (int k = 0; k < kLaneColumns; ++k)
            {
                left[k] = gather<T, kPacked>(a, first[k] < 0 ? 0 : first[k]);
                right[k] = gather<T, kPacked>(a, second[k]);
            }
        }
        // The next run's columns, loaded behind this run's arithmetic.
        base += stride;
        load_columns(base);
        if (padding)
        {
            continue;
        }
        // E and W of the four columns, summed by themselves: the running sums then take a quarter
        // of the terms.
        T four_e = 0, four_xx = 0, four_yy = 0, four_zz = 0, four_xy = 0, four_xz = 0, four_yz = 0;
#pragma unroll
        for (int k = 0; k < kLaneColumns; ++k)
        {
            T dx = left[k].x - right[k].x;
            T dy = left[k].y - right[k].y;
            T dz = left[k].z - right[k].z;
            // Few pairs cross a face: a warp without one takes the plain differences.
            if (fabs(dx) > hx || fabs(dy) > hy || fabs(dz) > hz)
            {
                dx = displacement(left[k].x, right[k].x, lx);
                dy = displacement(left[k].y, right[k].y, ly);
                dz = displacement(left[k].z, right[k].z, lz);
            }
            const T r2 = dx * dx + dy * dy + dz * dz;
            const bool hit = first[k] >= 0 && r2 < a.cutoff_squared;
            T px = 0, py = 0, pz = 0;
            if (hit)
            {
                const RowConstants<T> c =
                    rows[kTypes ? pair_row(word_type(left[k].w), word_type(right[k].w),
                                           a.num_types)
                                : 0];
                const T inv_r2 = reciprocal(r2);
                const T q = c.s2 * inv_r2;
                const T p6 = q * q * q;
                four_e += c.eps4 * (p6 * p6 - p6) - c.shift;
                const T fs = c.eps24 * (T(2) * p6 * p6 - p6) * inv_r2;
                px = fs * dx;
                py = fs * dy;
                pz = fs * dz;
                four_xx += px * dx;
                four_yy += py * dy;
                four_zz += pz * dz;
                four_xy += px * dy;
                four_xz += px * dz;
                four_yz += py * dz;
                add_force<T, kPacked>(a, second[k], -px, -py, -pz);
            }
            const int at = kWarp * k + lane;
            stage.x[at] = px;
            stage.y[at] = py;
            stage.z[at] = pz;
            stage.key[at] = hit ? first[k] : -1;
        }
        energy += four_e;
        wxx += four_xx;
        wyy += four_yy;
        wzz += four_zz;
        wxy += four_xy;
        wxz += four_xz;
        wyz += four_yz;
        __syncwarp();
        // The first atoms' side: the lane's four consecutive columns, summed while the atom
        // stays the same.
        index_t key = -1;
        T fx = 0, fy = 0, fz = 0;
        const Four<T> sx = load4(stage.x + kLaneColumns * lane);
        const Four<T> sy = load4(stage.y + kLaneColumns * lane);
        const Four<T> sz = load4(stage.z + kLaneColumns * lane);
        const Four<index_t> keys = load4(stage.key + kLaneColumns * lane);
#pragma unroll
        for (int k = 0; k < kLaneColumns; ++k)
        {
            const index_t atom = keys.v[k];
            if (atom >= 0 && atom != key)
            {
                if (key >= 0)
                {
                    add_force<T, kPacked>(a, key, fx, fy, fz);
                }
                key = atom;
                fx = fy = fz = T(0);
            }
            fx += sx.v[k];
            fy += sy.v[k];
            fz += sz.v[k];
        }
        __syncwarp();
        // Lanes in a row that end on the same first atom sum into their first lane.
        const index_t before = __shfl_up_sync(kFullMask, key, 1);
        const bool head = lane == 0 || before != key;
        const unsigned heads = __ballot_sync(kFullMask, head);
        const unsigned later = lane == kWarp - 1 ? 0u : heads >> (lane + 1);
        const int reach = later == 0 ? kWarp - 1 - lane : __ffs(later) - 1;  // lanes after mine
#pragma unroll
        for (int offset = 1; offset < kWarp; offset *= 2)
        {
            const T ox = __shfl_down_sync(kFullMask, fx, offset);
            const T oy = __shfl_down_sync(kFullMask, fy, offset);
            const T oz = __shfl_down_sync(kFullMask, fz, offset);
            if (offset <= reach)
            {
                fx += ox;
                fy += oy;
                fz += oz;
            }
        }
        if (head && key >= 0)
        {
            add_force<T, kPacked>(a, key, fx, fy, fz);
        }
    }
    double values[kFrameSums] = {double(energy), double(wxx), double(wyy), double(wzz),
                                 double(wxy), double(wxz), double(wyz)};
    if (kPacked)
    {
        double* s = a.sums + kFrameSlots * frame;
        double* const out[kFrameSums] = {s, s + 1, s + 2, s + 3, s + 4, s + 5, s + 6};
        add_block_sums(values, out);
    }
    else
    {
        double all[10] = {values[0], values[1], values[4], values[5], values[4], values[2],
                          values[6], values[5], values[6], values[3]};
        double* w = a.virial + 9 * frame;
        double* const out[10] = {a.energy + frame, w, w + 1, w + 2, w + 3, w + 4, w + 5, w + 6,
                                 w + 7, w + 8};
        add_block_sums(all, out);
    }
}

// Blocks per frame, each taking kColumns columns at a time: as many as the columns fill, up to
// `per_sm` blocks per SM over all frames, then several turns per block.
template <int kColumns>
int frame_blocks(std::int64_t capacity, std::int64_t frames, int per_sm, unsigned* blocks)
{
    int sms = 148;
    ND_CUDA_TRY(multiprocessors(&sms));
    const std::int64_t wanted = (capacity + kColumns - 1) / kColumns;
    const std::int64_t most = std::max<std::int64_t>(1, static_cast<std::int64_t>(sms) * per_sm /
                                                            std::max<std::int64_t>(1, frames));
    *blocks = static_cast<unsigned>(std::max<std::int64_t>(1, std::min(wanted, most)));
    return ND_OK;
}

template <typename T, bool kPacked>
int launch_frames(const FramesPass<T>& pass, std::int64_t frames, cudaStream_t stream)
{
    unsigned blocks = 1;
    const int rc = frame_blocks<kLJThreads * kLaneColumns>(
        pass.capacity, frames, frames == 1 ? kFrameBlocksPerSM<T> : 4 * kFrameBlocksPerSM<T>,
        &blocks);
    if (rc != ND_OK)
    {
        return rc;
    }
    const dim3 grid(blocks, static_cast<unsigned>(frames));
    if (pass.num_types > 1)
    {
        lj_frames_kernel<T, kPacked, true><<<grid, kLJThreads, 0, stream>>>(pass);
    }
    else
    {
        lj_frames_kernel<T, kPacked, false><<<grid, kLJThreads, 0, stream>>>(pass);
    }
    ND_LAUNCH_CHECK();
    return ND_OK;
}

// The frames with a workspace: pack (and wrap), pairs, unpack.
template <typename T>
int lj_frames(const nd_lj_batch_args* a, bool wrap, void* workspace, cudaStream_t stream)
{
    const std::int64_t n = a->num_atoms, frames = a->frames, slots = n * frames;
    const FrameWorkspace<T> ws(frames, n);
    auto* base = static_cast<unsigned char*>(workspace);
    auto* sums = reinterpret_cast<double*>(base + ws.sums);
    auto* atoms = reinterpret_cast<PackedAtom<T>*>(base + ws.atoms);
    auto* packed = sizeof(T) == 4 ? reinterpret_cast<float4*>(base + ws.forces) : nullptr;
    const auto* types = a->num_types > 1 ? a->atom_types : nullptr;
    auto* forces = static_cast<T*>(a->forces);
    const auto* positions = static_cast<const T*>(a->positions);
    const auto* cells = static_cast<const T*>(a->cells);
    const auto atoms_n = static_cast<index_t>(n);
    if (wrap)
    {
        pack_atoms_kernel<T, true><<<blocks_for(slots), kThreads, 0, stream>>>(
            positions, cells, types, atoms_n, slots, frames, atoms, packed, forces, sums);
    }
    else
    {
        pack_atoms_kernel<T, false><<<blocks_for(slots), kThreads, 0, stream>>>(
            positions, cells, types, atoms_n, slots, frames, atoms, packed, forces, sums);
    }
    ND_LAUNCH_CHECK();
    const T rc = static_cast<T>(a->cutoff);
    FramesPass<T> pass{};
    pass.atoms = atoms;
    pass.cells = cells;
    pass.pairs = a->pairs;
    pass.capacity = a->capacity;
    pass.num_atoms = atoms_n;
    pass.num_types = a->num_types;
    pass.sigma = static_cast<const T*>(a->sigma);
    pass.epsilon = static_cast<const T*>(a->epsilon);
    pass.cutoff_squared = rc * rc;
    pass.packed_forces = packed;
    pass.forces = forces;
    pass.sums = sums;
    const int launched = launch_frames<T, true>(pass, frames, stream);
    if (launched != ND_OK)
    {
        return launched;
    }
    const std::int64_t items = sizeof(T) == 4 ? slots : frames * 10;
    unpack_frames_kernel<T><<<blocks_for(items), kThreads, 0, stream>>>(
        packed, slots, frames, sums, sizeof(T) == 4 ? reinterpret_cast<float*>(forces) : nullptr,
        reinterpret_cast<T*>(a->energy), reinterpret_cast<T*>(a->virial));
    ND_LAUNCH_CHECK();
    return ND_OK;
}

// The frames without a workspace: float64 sums and scalar force atomics in place.
template <typename T>
int lj_frames_in_place(std::int64_t frames, const nd_lj_batch_args* a, cudaStream_t stream)
{
    const std::int64_t n = a->num_atoms;
    ND_CUDA_TRY(cudaMemsetAsync(a->forces, 0, sizeof(T) * 3 * n * frames, stream));
    ND_CUDA_TRY(cudaMemsetAsync(a->energy, 0, sizeof(double) * frames, stream));
    ND_CUDA_TRY(cudaMemsetAsync(a->virial, 0, sizeof(double) * 9 * frames, stream));
    const T rc = static_cast<T>(a->cutoff);
    FramesPass<T> pass{};
    pass.positions = static_cast<const T*>(a->positions);
    pass.atom_types = a->num_types > 1 ? a->atom_types : nullptr;
    pass.cells = static_cast<const T*>(a->cells);
    pass.pairs = a->pairs;
    pass.capacity = a->capacity;
    pass.num_atoms = static_cast<index_t>(n);
    pass.num_types = a->num_types;
    pass.sigma = static_cast<const T*>(a->sigma);
    pass.epsilon = static_cast<const T*>(a->epsilon);
    pass.cutoff_squared = rc * rc;
    pass.forces = static_cast<T*>(a->forces);
    pass.energy = a->energy;
    pass.virial = a->virial;
    return launch_frames<T, false>(pass, frames, stream);
}

template <typename T>
int lj_pairs(const nd_lj_pairs_args* a, cudaStream_t stream)
{
    const bool grads = a->sigma_grad != nullptr;
    if (!grads && a->strain == nullptr)
    {
        nd_lj_batch_args frame{};
        frame.frames = 1;
        frame.positions = a->positions;
        frame.cells = a->cell;
        frame.num_atoms = a->num_atoms;
        frame.pairs = a->pairs;
        frame.capacity = a->capacity;
        frame.atom_types = a->atom_types;
        frame.num_types = a->num_types;
        frame.sigma = a->sigma;
        frame.epsilon = a->epsilon;
        frame.cutoff = a->cutoff;
        frame.energy = a->energy;
        frame.forces = a->forces;
        frame.virial = a->virial;
        return lj_frames_in_place<T>(1, &frame, stream);
    }
    const std::int64_t n = a->num_atoms;
    ND_CUDA_TRY(cudaMemsetAsync(a->forces, 0, sizeof(T) * 3 * n, stream));
    ND_CUDA_TRY(cudaMemsetAsync(a->energy, 0, sizeof(double), stream));
    ND_CUDA_TRY(cudaMemsetAsync(a->virial, 0, sizeof(double) * 9, stream));
    const int rows = a->num_types * (a->num_types + 1) / 2;
    if (grads)
    {
        ND_CUDA_TRY(cudaMemsetAsync(a->sigma_grad, 0, sizeof(double) * rows, stream));
        ND_CUDA_TRY(cudaMemsetAsync(a->epsilon_grad, 0, sizeof(double) * rows, stream));
    }
    unsigned blocks = 1;
    const int counted = frame_blocks<kLJThreads>(a->capacity, 1, 8, &blocks);
    if (counted != ND_OK)
    {
        return counted;
    }
    const T rc = static_cast<T>(a->cutoff);
    const auto* types = a->num_types > 1 ? a->atom_types : nullptr;
    const auto* strain = static_cast<const T*>(a->strain);
    auto launch = [&](auto kernel) {
        kernel<<<blocks, kLJThreads, 0, stream>>>(
            static_cast<const T*>(a->positions), static_cast<const T*>(a->cell), a->pairs,
            a->capacity, static_cast<index_t>(a->num_atoms), types, a->num_types,
            static_cast<const T*>(a->sigma), static_cast<const T*>(a->epsilon), strain, rc * rc,
            a->energy, static_cast<T*>(a->forces), a->virial, a->sigma_grad, a->epsilon_grad);
    };
    if (grads && strain)
    {
        launch(lj_pairs_kernel<T, true, true>);
    }
    else if (grads)
    {
        launch(lj_pairs_kernel<T, true, false>);
    }
    else
    {
        launch(lj_pairs_kernel<T, false, true>);
    }
    ND_LAUNCH_CHECK();
    return ND_OK;
}

// ---------------------------------------------------------------------------------------
// The parameter backward of a batch: given the loss's gradients with respect to each frame's
// energy, forces and virial, accumulates dLoss/dsigma and dLoss/depsilon per type-pair row.
// For a valid column with d = x_i - x_j and f_s = 24 eps (2 p6^2 - p6) / r^2 (so F_i = f_s d,
// F_j = -f_s d, W = f_s d (x) d), the pair adds
//     g_E du/dtheta + (d . (g_F[i] - g_F[j]) + d^T g_W d) df_s/dtheta,
// with du/deps = 4 (p6^2 - p6) - 4 (pc6^2 - pc6), du/dsigma = 24 eps / sigma (2 p6^2 - p6 -
// 2 pc6^2 + pc6), df_s/deps = f_s / eps and df_s/dsigma = 144 eps p6 (4 p6 - 1) / (sigma r^2).
// This is the double backward the reference takes through torch.func
// (src/nabladyn/training/_fit.py:245-271), written out. Per-row sums are float64.
//
// A column gathers two atoms and two force gradients and scatters nothing, so with packed
// slots it is bound by the float64 arithmetic: the row's constants are worked out once per
// block, and a thread keeps its rows' sums to itself (in registers for one row, else in its own
// column of shared memory), since float64 atomics on a few shared words serialise the block
// (64 frames of 4,096 atoms, two types, float32: 778 -> 98 us; gathering the force gradients before
// the cutoff test, or six blocks per SM at 40 registers, gave 100).

// One type-pair row's float64 constants.
struct RowGradients
{
    double s2, eps24_s, eps144_s, pc_deps, pc_dsigma;
};

template <typename T>
struct BackwardPass
{
    FramesPass<T> frames;             // atoms, cells, pairs, parameters
    const PackedAtom<T>* force_slots; // packed force gradients, or null:
    const T* force_grads;             // [F, N, 3]
    const T* energy_grad;             // packed: [F] and [F, 9] in the frames' dtype
    const T* virial_grad;
    const double* energy_grad64;      // else float64
    const double* virial_grad64;
    double* row_sums;                 // sigma rows, then epsilon rows
    double* epsilon_sums;
};

template <typename T, bool kPacked>
__device__ __forceinline__ PackedAtom<T> gather_gradient(const BackwardPass<T>& a, index_t atom)
{
    if constexpr (kPacked)
    {
        return a.force_slots[atom];
    }
    else
    {
        const T* g = a.force_grads + 3LL * atom;
        return {g[0], g[1], g[2], T(0)};
    }
}

template <typename T, bool kPacked, bool kTypes>
__global__ void __launch_bounds__(kLJThreads) lj_parameter_backward_kernel(BackwardPass<T> a)
{
    extern __shared__ double own_sums[];  // [2 rows][kLJThreads] with several types
    const std::int64_t frame = blockIdx.y;
    FramesPass<T>& f = a.frames;
    if (kPacked)
    {
        f.atoms += frame * f.num_atoms;
        a.force_slots += frame * f.num_atoms;
    }
    else
    {
        f.positions += 3 * frame * f.num_atoms;
        a.force_grads += 3 * frame * f.num_atoms;
    }
    f.cells += 3 * frame;
    f.pairs += 2 * frame * f.capacity;
    const double ge = kPacked ? static_cast<double>(a.energy_grad[frame]) : a.energy_grad64[frame];
    double gw[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
    {
        gw[k] = kPacked ? static_cast<double>(a.virial_grad[9 * frame + k])
                        : a.virial_grad64[9 * frame + k];
    }
    // d^T g_W d takes the sums of mirrored entries.
    const double gxy = gw[1] + gw[3], gxz = gw[2] + gw[6], gyz = gw[5] + gw[7];
    __shared__ RowGradients rows[kTypes ? kMaxRows : 1];
    const int row_count = kTypes ? f.num_types * (f.num_types + 1) / 2 : 1;
    if (threadIdx.x < row_count)
    {
        const double s = f.sigma[threadIdx.x], eps = f.epsilon[threadIdx.x];
        const double qc = s * s / static_cast<double>(f.cutoff_squared);
        const double pc6 = qc * qc * qc;
        rows[threadIdx.x] = {s * s, 24.0 * eps / s, 144.0 * eps / s, 4.0 * (pc6 * pc6 - pc6),
                             2.0 * pc6 * pc6 - pc6};
    }
    if (kTypes)
    {
        for (int r = 0; r < 2 * row_count; ++r)
        {
            own_sums[r * kLJThreads + threadIdx.x] = 0.0;
        }
    }
    __syncthreads();
    double sigma_sum = 0.0, epsilon_sum = 0.0;  // one type
    const T lx = f.cells[0], ly = f.cells[1], lz = f.cells[2];
    const auto capacity = static_cast<unsigned>(f.capacity);
    const index_t* firsts = f.pairs;
    const index_t* seconds = f.pairs + f.capacity;
    const unsigned stride = gridDim.x * kLJThreads;
    // A column's atoms are read one column ahead: its gathers then wait for one load, not two.
    unsigned column = blockIdx.x * kLJThreads + threadIdx.x;
    index_t next_i = column < capacity ? firsts[column] : 0;
    index_t next_j = column < capacity ? seconds[column] : 0;
    while (column < capacity)
    {
        const index_t i = next_i, j = next_j;
        column += stride;
        if (column < capacity)
        {
            next_i = firsts[column];
            next_j = seconds[column];
        }
        if (!counts(i, j, f.num_atoms))
        {
            continue;
        }
        const PackedAtom<T> left = gather<T, kPacked>(f, i), right = gather<T, kPacked>(f, j);
        const T tx = displacement(left.x, right.x, lx);
        const T ty = displacement(left.y, right.y, ly);
        const T tz = displacement(left.z, right.z, lz);
        const T r2 = tx * tx + ty * ty + tz * tz;
        if (!(r2 < f.cutoff_squared))
        {
            continue;
        }
        const PackedAtom<T> gi = gather_gradient<T, kPacked>(a, i);
        const PackedAtom<T> gj = gather_gradient<T, kPacked>(a, j);
        const int row =
            kTypes ? pair_row(word_type(left.w), word_type(right.w), f.num_types) : 0;
        const RowGradients c = rows[row];
        const double inv_r2 = 1.0 / static_cast<double>(r2);
        const double q = c.s2 * inv_r2;
        const double p6 = q * q * q;
        const double x = tx, y = ty, z = tz;
        const double dgx = static_cast<double>(gi.x) - static_cast<double>(gj.x);
        const double dgy = static_cast<double>(gi.y) - static_cast<double>(gj.y);
        const double dgz = static_cast<double>(gi.z) - static_cast<double>(gj.z);
        const double g = x * (dgx + gw[0] * x + gxy * y + gxz * z) +
                         y * (dgy + gw[4] * y + gyz * z) + z * (dgz + gw[8] * z);
        const double slope = p6 * (2.0 * p6 - 1.0);  // 2 p6^2 - p6
        const double pull = g * inv_r2;
        const double dsigma = c.eps24_s * (ge * (slope - c.pc_dsigma)) +
                              c.eps144_s * (pull * (p6 * (4.0 * p6 - 1.0)));
        const double depsilon = ge * (4.0 * (p6 * (p6 - 1.0)) - c.pc_deps) + 24.0 * (pull * slope);
        if (kTypes)
        {
            own_sums[row * kLJThreads + threadIdx.x] += dsigma;
            own_sums[(row_count + row) * kLJThreads + threadIdx.x] += depsilon;
        }
        else
        {
            sigma_sum += dsigma;
            epsilon_sum += depsilon;
        }
    }
    if (!kTypes)
    {
        double values[2] = {sigma_sum, epsilon_sum};
        double* const out[2] = {a.row_sums, a.epsilon_sums};
        add_block_sums(values, out);
        return;
    }
    __syncthreads();
    const int lane = threadIdx.x % kWarp;
    for (int r = threadIdx.x / kWarp; r < 2 * row_count; r += kLJThreads / kWarp)
    {
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < kLJThreads; k += kWarp)
        {
            sum += own_sums[r * kLJThreads + k + lane];
        }
        sum = warp_sum(sum);
        if (lane == 0)
        {
            atomicAdd(r < row_count ? a.row_sums + r : a.epsilon_sums + (r - row_count), sum);
        }
    }
}

// As many blocks as the GPU holds at once: with eight per SM, of which five fit, the second wave
// left two SMs in five idle (64 frames of 4,096 atoms: 118 us, in one wave 99).
template <typename T, bool kPacked>
int launch_backward(const BackwardPass<T>& pass, std::int64_t frames, cudaStream_t stream)
{
    const bool types = pass.frames.num_types > 1;
    const int rows = pass.frames.num_types * (pass.frames.num_types + 1) / 2;
    const std::size_t bytes = types ? 2 * rows * kLJThreads * sizeof(double) : 0;
    auto* kernel = types ? lj_parameter_backward_kernel<T, kPacked, true>
                         : lj_parameter_backward_kernel<T, kPacked, false>;
    if (types)
    {
        static DeviceGrant grant;
        ND_CUDA_TRY(grant.allow(lj_parameter_backward_kernel<T, kPacked, true>, bytes));
    }
    int resident = 1;
    ND_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kLJThreads, bytes));
    unsigned blocks = 1;
    const int counted =
        frame_blocks<kLJThreads>(pass.frames.capacity, frames, std::max(1, resident), &blocks);
    if (counted != ND_OK)
    {
        return counted;
    }
    kernel<<<dim3(blocks, static_cast<unsigned>(frames)), kLJThreads, bytes, stream>>>(pass);
    ND_LAUNCH_CHECK();
    return ND_OK;
}

template <typename T>
FramesPass<T> backward_frames(const nd_lj_batch_args* a)
{
    const T rc = static_cast<T>(a->cutoff);
    FramesPass<T> frames{};
    frames.positions = static_cast<const T*>(a->positions);
    frames.atom_types = a->num_types > 1 ? a->atom_types : nullptr;
    frames.cells = static_cast<const T*>(a->cells);
    frames.pairs = a->pairs;
    frames.capacity = a->capacity;
    frames.num_atoms = static_cast<index_t>(a->num_atoms);
    frames.num_types = a->num_types;
    frames.sigma = static_cast<const T*>(a->sigma);
    frames.epsilon = static_cast<const T*>(a->epsilon);
    frames.cutoff_squared = rc * rc;
    return frames;
}

// Without a workspace: the caller's arrays as they are.
template <typename T>
int lj_batch_parameter_backward(const nd_lj_batch_args* a, cudaStream_t stream)
{
    const int rows = a->num_types * (a->num_types + 1) / 2;
    ND_CUDA_TRY(cudaMemsetAsync(a->sigma_grad, 0, sizeof(double) * rows, stream));
    ND_CUDA_TRY(cudaMemsetAsync(a->epsilon_grad, 0, sizeof(double) * rows, stream));
    BackwardPass<T> pass{};
    pass.frames = backward_frames<T>(a);
    pass.force_grads = static_cast<const T*>(a->forces_grad);
    pass.energy_grad64 = a->energy_grad;
    pass.virial_grad64 = a->virial_grad;
    pass.row_sums = a->sigma_grad;
    pass.epsilon_sums = a->epsilon_grad;
    return launch_backward<T, false>(pass, a->frames, stream);
}

// Packs the force gradients and sets the row sums to zero.
template <typename T>
__global__ void __launch_bounds__(kThreads) pack_gradients_kernel(
    const T* __restrict__ force_grads, std::int64_t slots, PackedAtom<T>* __restrict__ gradients,
    double* __restrict__ sums)
{
    const std::int64_t slot = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x < 2 * kMaxRows)
    {
        sums[threadIdx.x] = 0.0;
    }
    if (slot < slots)
    {
        const T* g = force_grads + 3 * slot;
        gradients[slot] = {g[0], g[1], g[2], T(0)};
    }
}

// The row sums in the parameters' dtype.
template <typename T>
__global__ void cast_rows_kernel(const double* __restrict__ sums, int rows,
                                 T* __restrict__ sigma_grad, T* __restrict__ epsilon_grad)
{
    if (threadIdx.x < rows)
    {
        sigma_grad[threadIdx.x] = static_cast<T>(sums[threadIdx.x]);
        epsilon_grad[threadIdx.x] = static_cast<T>(sums[kMaxRows + threadIdx.x]);
    }
}

template <typename T>
int lj_frames_parameter_backward(const nd_lj_batch_args* a, void* workspace, cudaStream_t stream)
{
    const std::int64_t n = a->num_atoms, slots = n * a->frames;
    const FrameWorkspace<T> ws(a->frames, n);
    auto* base = static_cast<unsigned char*>(workspace);
    auto* sums = reinterpret_cast<double*>(base + ws.sums);
    auto* gradients = reinterpret_cast<PackedAtom<T>*>(base + ws.forces);
    pack_gradients_kernel<T><<<blocks_for(slots), kThreads, 0, stream>>>(
        static_cast<const T*>(a->forces_grad), slots, gradients, sums);
    ND_LAUNCH_CHECK();
    BackwardPass<T> pass{};
    pass.frames = backward_frames<T>(a);
    pass.frames.atoms = reinterpret_cast<const PackedAtom<T>*>(
        static_cast<const unsigned char*>(a->positions) + ws.atoms);
    pass.force_slots = gradients;
    pass.energy_grad = reinterpret_cast<const T*>(a->energy_grad);
    pass.virial_grad = reinterpret_cast<const T*>(a->virial_grad);
    pass.row_sums = sums;
    pass.epsilon_sums = sums + kMaxRows;
    const int launched = launch_backward<T, true>(pass, a->frames, stream);
    if (launched != ND_OK)
    {
        return launched;
    }
    cast_rows_kernel<T><<<1, 64, 0, stream>>>(
        sums, a->num_types * (a->num_types + 1) / 2, reinterpret_cast<T*>(a->sigma_grad),
        reinterpret_cast<T*>(a->epsilon_grad));
    ND_LAUNCH_CHECK();
    return ND_OK;
}

int check_batch(const nd_lj_batch_args* a, bool backward)
{
    ND_REQUIRE(a != nullptr, "the arguments are null");
    ND_REQUIRE(a->dtype == ND_FLOAT32 || a->dtype == ND_FLOAT64, "positions must be float32 or float64");
    ND_REQUIRE(a->frames >= 1 && a->frames <= 65535, "1 to 65535 frames per batch");
    ND_REQUIRE(a->num_atoms >= 1 && a->num_atoms <= INT32_MAX, "N must be in [1, 2**31)");
    ND_REQUIRE(a->capacity >= 1 && a->capacity <= INT32_MAX, "pairs must be [F, 2, C]");
    ND_REQUIRE(a->num_types >= 1 && a->num_types <= 8, "1 to 8 atom types are supported");
    ND_REQUIRE(a->num_types == 1 || a->atom_types != nullptr, "atom_types is null");
    ND_REQUIRE(a->cutoff > 0, "the cutoff must be positive");
    ND_REQUIRE(a->positions && a->cells && a->pairs && a->sigma && a->epsilon,
               "a required pointer is null");
    if (backward)
    {
        ND_REQUIRE(a->energy_grad && a->forces_grad && a->virial_grad && a->sigma_grad &&
                       a->epsilon_grad,
                   "a gradient pointer is null");
    }
    else
    {
        ND_REQUIRE(a->energy && a->forces && a->virial, "an output pointer is null");
    }
    return ND_OK;
}

}  // namespace nd

extern "C" int nd_lj_batch_forward(const nd_lj_batch_args* args, nd_stream_t stream)
{
    const int rc = nd::check_batch(args, false);
    if (rc != ND_OK)
    {
        return rc;
    }
    auto s = static_cast<cudaStream_t>(stream);
    return args->dtype == ND_FLOAT32 ? nd::lj_frames_in_place<float>(args->frames, args, s)
                                     : nd::lj_frames_in_place<double>(args->frames, args, s);
}

extern "C" int64_t nd_lj_workspace_bytes(int dtype, int64_t frames, int64_t num_atoms)
{
    if ((dtype != ND_FLOAT32 && dtype != ND_FLOAT64) || frames < 1 || num_atoms < 1)
    {
        return -1;
    }
    return dtype == ND_FLOAT32 ? nd::FrameWorkspace<float>(frames, num_atoms).total
                               : nd::FrameWorkspace<double>(frames, num_atoms).total;
}

extern "C" int nd_lj_frames(const nd_lj_batch_args* args, int32_t wrap, void* workspace,
                            nd_stream_t stream)
{
    const int rc = nd::check_batch(args, false);
    if (rc != ND_OK)
    {
        return rc;
    }
    ND_REQUIRE(workspace != nullptr, "the workspace is null");
    ND_REQUIRE(reinterpret_cast<std::uintptr_t>(workspace) % 256 == 0,
               "the workspace must be 256-byte aligned");
    auto s = static_cast<cudaStream_t>(stream);
    return args->dtype == ND_FLOAT32 ? nd::lj_frames<float>(args, wrap != 0, workspace, s)
                                     : nd::lj_frames<double>(args, wrap != 0, workspace, s);
}

extern "C" int nd_lj_frames_parameter_backward(const nd_lj_batch_args* args, void* workspace,
                                               nd_stream_t stream)
{
    const int rc = nd::check_batch(args, true);
    if (rc != ND_OK)
    {
        return rc;
    }
    ND_REQUIRE(workspace != nullptr, "the workspace is null");
    ND_REQUIRE(reinterpret_cast<std::uintptr_t>(workspace) % 256 == 0 &&
                   reinterpret_cast<std::uintptr_t>(args->positions) % 256 == 0,
               "the workspaces must be 256-byte aligned");
    auto s = static_cast<cudaStream_t>(stream);
    return args->dtype == ND_FLOAT32
               ? nd::lj_frames_parameter_backward<float>(args, workspace, s)
               : nd::lj_frames_parameter_backward<double>(args, workspace, s);
}

extern "C" int nd_wrap(int dtype, const void* positions, const void* cells, int64_t frames,
                       int64_t num_atoms, void* wrapped, nd_stream_t stream)
{
    ND_REQUIRE(dtype == ND_FLOAT32 || dtype == ND_FLOAT64, "positions must be float32 or float64");
    ND_REQUIRE(frames >= 0 && num_atoms >= 0 && frames <= INT32_MAX && num_atoms <= INT32_MAX &&
                   frames * num_atoms <= INT64_C(1) << 38,
               "too many atoms");
    if (frames * num_atoms == 0)
    {
        return ND_OK;
    }
    ND_REQUIRE(positions && cells && wrapped, "a required pointer is null");
    auto s = static_cast<cudaStream_t>(stream);
    const int64_t values = 3 * frames * num_atoms;
    if (dtype == ND_FLOAT32)
    {
        nd::wrap_kernel<float><<<nd::blocks_for(values), nd::kThreads, 0, s>>>(
            static_cast<const float*>(positions), static_cast<const float*>(cells), num_atoms,
            values, static_cast<float*>(wrapped));
    }
    else
    {
        nd::wrap_kernel<double><<<nd::blocks_for(values), nd::kThreads, 0, s>>>(
            static_cast<const double*>(positions), static_cast<const double*>(cells), num_atoms,
            values, static_cast<double*>(wrapped));
    }
    ND_LAUNCH_CHECK();
    return ND_OK;
}

extern "C" int nd_lj_batch_parameter_backward(const nd_lj_batch_args* args, nd_stream_t stream)
{
    const int rc = nd::check_batch(args, true);
    if (rc != ND_OK)
    {
        return rc;
    }
    auto s = static_cast<cudaStream_t>(stream);
    return args->dtype == ND_FLOAT32 ? nd::lj_batch_parameter_backward<float>(args, s)
                                     : nd::lj_batch_parameter_backward<double>(args, s);
}

extern "C" int nd_lj_energy_force_virial(const nd_lj_pairs_args* args, nd_stream_t stream)
{
    ND_REQUIRE(args != nullptr, "the arguments are null");
    ND_REQUIRE(args->dtype == ND_FLOAT32 || args->dtype == ND_FLOAT64,
               "positions must be float32 or float64");
    ND_REQUIRE(args->num_atoms >= 1 && args->num_atoms <= INT32_MAX, "N must be in [1, 2**31)");
    ND_REQUIRE(args->capacity >= 1 && args->capacity <= INT32_MAX, "pairs must be [2, C]");
    ND_REQUIRE(args->num_types >= 1 && args->num_types <= 8, "1 to 8 atom types are supported");
    ND_REQUIRE(args->num_types == 1 || args->atom_types != nullptr, "atom_types is null");
    ND_REQUIRE(args->cutoff > 0, "the cutoff must be positive");
    ND_REQUIRE(args->positions && args->cell && args->pairs && args->sigma && args->epsilon &&
                   args->energy && args->forces && args->virial,
               "a required pointer is null");
    ND_REQUIRE((args->sigma_grad == nullptr) == (args->epsilon_grad == nullptr),
               "sigma_grad and epsilon_grad come together");
    auto s = static_cast<cudaStream_t>(stream);
    return args->dtype == ND_FLOAT32 ? nd::lj_pairs<float>(args, s) : nd::lj_pairs<double>(args, s);
}
