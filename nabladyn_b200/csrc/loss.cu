// The training loss of a batch and its gradient in the predictions.
//
//     L = sum_c w_c t_c,  t_c = sum_f k_f mean_i ((X_fi - Y_fi) / s_c)^2,
//
// over up to three channels (energy [F], forces [F, N, 3], virial [F, 3, 3]), with the frames'
// coefficients k_f (1/F when none are given); src/nabladyn/training/_loss.py:105-125. As
// elementwise operations a loss and its backward take some forty launches of a few microseconds
// each, which bound a fit of ordinary frames; here each direction is one pass: the forward
// reads predictions and labels once and, when a gradient will be wanted, also writes the terms'
// slopes, which the backward scales (64 frames of 4,096 atoms, energy, forces and virial: the
// whole training update 680 -> 378 us). Squares are taken in the predictions' dtype and summed in
// float64.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace nd {
namespace {

constexpr int kChannels = 3;
constexpr std::int64_t kLossItems = 8;  // elements per thread the grid aims at
constexpr int kLossBlocks = 148 * 8;    // per channel, at most
static_assert(ND_LOSS_PARTIALS >= kChannels * kLossBlocks + 1, "a sum per block and the count");

template <typename T>
struct LossPass
{
    const T* predicted[kChannels];
    const T* labels[kChannels];
    std::int64_t size[kChannels];  // components per frame
    T scale[kChannels];
    double weight[kChannels];
    std::int64_t frames;
    const T* coefficients;         // null: 1/F
    int channels;
    double* partials;              // forward: [channels][blocks], then the count of finished blocks
    T* total;
    T* terms[kChannels];
    const T* total_grad;           // backward: null means zero
    const T* term_grad[kChannels];
    T* gradients[kChannels];       // forward: dt_c/dX; backward: dL/dX; null: not wanted
};

template <typename T>
__global__ void __launch_bounds__(kThreads) loss_forward_kernel(LossPass<T> a)
{
    const int c = blockIdx.y;
    const std::int64_t size = a.size[c], items = size * a.frames;
    const T scale = a.scale[c];
    T* const slopes = a.gradients[c];
    const double share = 2.0 / static_cast<double>(size) /
                         (a.coefficients != nullptr ? 1.0 : static_cast<double>(a.frames));
    double sum = 0.0;
    const std::int64_t stride = static_cast<std::int64_t>(gridDim.x) * blockDim.x;
    for (std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
         i < items; i += stride)
    {
        const T error = (a.predicted[c][i] - a.labels[c][i]) / scale;
        const double frame =
            a.coefficients != nullptr ? static_cast<double>(a.coefficients[i / size]) : 1.0;
        sum += static_cast<double>(error * error) * frame;
        if (slopes != nullptr)
        {
            slopes[i] = static_cast<T>(share * frame) * error / scale;  // 2 k (X - Y) / (s^2 n)
        }
    }
    __shared__ double warp_sums[kThreads / kWarp];
    __shared__ bool last;
    // One block sum per block, in a fixed order; thread 0 gets it.
    auto block_sum = [&](double value) {
        value = warp_sum(value);
        if (threadIdx.x % kWarp == 0)
        {
            warp_sums[threadIdx.x / kWarp] = value;
        }
        __syncthreads();
        double all = 0.0;
        for (int w = 0; w < kThreads / kWarp && threadIdx.x == 0; ++w)
        {
            all += warp_sums[w];
        }
        __syncthreads();
        return all;
    };
    sum = block_sum(sum);
    if (threadIdx.x == 0)
    {
        a.partials[c * gridDim.x + blockIdx.x] = sum;
        __threadfence();
        auto* finished = reinterpret_cast<unsigned*>(a.partials + a.channels * gridDim.x);
        last = atomicAdd(finished, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!last)
    {
        return;
    }
    // The last block to finish: every block's sum is there. They are added in the blocks' order,
    // whichever block this is, so a loss has the same bits each time.
    __threadfence();
    double total = 0.0;
    for (int k = 0; k < a.channels; ++k)
    {
        double part = 0.0;
        for (unsigned i = threadIdx.x; i < gridDim.x; i += kThreads)
        {
            part += *reinterpret_cast<volatile double*>(a.partials + k * gridDim.x + i);
        }
        part = block_sum(part);
        if (threadIdx.x == 0)
        {
            const double term = part / static_cast<double>(a.size[k]) /
                                (a.coefficients != nullptr ? 1.0 : static_cast<double>(a.frames));
            *a.terms[k] = static_cast<T>(term);
            total += a.weight[k] * term;
        }
    }
    if (threadIdx.x == 0)
    {
        *a.total = static_cast<T>(total);
    }
}

// dL/dX = (w_c dL + dt_c) slope, the slopes in `predicted`.
template <typename T>
__global__ void __launch_bounds__(kThreads) loss_backward_kernel(LossPass<T> a)
{
    const int c = blockIdx.y;
    if (a.gradients[c] == nullptr)
    {
        return;
    }
    const std::int64_t items = a.size[c] * a.frames;
    const T factor =
        (a.total_grad != nullptr ? static_cast<T>(a.weight[c]) * *a.total_grad : T(0)) +
        (a.term_grad[c] != nullptr ? *a.term_grad[c] : T(0));
    const std::int64_t stride = static_cast<std::int64_t>(gridDim.x) * blockDim.x;
    for (std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
         i < items; i += stride)
    {
        a.gradients[c][i] = factor * a.predicted[c][i];
    }
}

template <typename T>
LossPass<T> loss_pass(const nd_loss_args& s)
{
    LossPass<T> a{};
    for (int c = 0; c < s.channels; ++c)
    {
        a.predicted[c] = static_cast<const T*>(s.predicted[c]);
        a.labels[c] = static_cast<const T*>(s.labels[c]);
        a.size[c] = s.sizes[c];
        a.scale[c] = static_cast<T>(s.scales[c]);
        a.weight[c] = s.weights[c];
        a.terms[c] = static_cast<T*>(s.terms[c]);
        a.term_grad[c] = static_cast<const T*>(s.term_grads[c]);
        a.gradients[c] = static_cast<T*>(s.gradients[c]);
    }
    a.frames = s.frames;
    a.coefficients = static_cast<const T*>(s.coefficients);
    a.channels = s.channels;
    a.partials = s.partials;
    a.total = static_cast<T*>(s.total);
    a.total_grad = static_cast<const T*>(s.total_grad);
    return a;
}

int check_loss(const nd_loss_args* s, bool forward)
{
    ND_REQUIRE(s != nullptr, "the arguments are null");
    ND_REQUIRE(s->dtype == ND_FLOAT32 || s->dtype == ND_FLOAT64,
               "predictions must be float32 or float64");
    ND_REQUIRE(s->channels >= 1 && s->channels <= kChannels, "one to three channels");
    ND_REQUIRE(s->frames >= 1, "at least one frame");
    for (int c = 0; c < s->channels; ++c)
    {
        ND_REQUIRE(forward ? s->predicted[c] && s->labels[c]
                           : s->predicted[c] || !s->gradients[c],
                   "a channel is null");
        ND_REQUIRE(s->sizes[c] >= 1 && s->sizes[c] <= INT64_MAX / s->frames,
                   "a channel's size is out of range");
    }
    return ND_OK;
}

dim3 loss_grid(const nd_loss_args& s)
{
    std::int64_t most = 1;
    for (int c = 0; c < s.channels; ++c)
    {
        most = std::max(most, s.sizes[c] * s.frames);
    }
    const std::int64_t blocks = (most + kThreads * kLossItems - 1) / (kThreads * kLossItems);
    return dim3(static_cast<unsigned>(std::min<std::int64_t>(blocks, kLossBlocks)),
                static_cast<unsigned>(s.channels));
}

}  // namespace
}  // namespace nd

extern "C" {

int nd_loss_forward(const nd_loss_args* args, nd_stream_t stream_handle)
{
    using namespace nd;
    const int rc = check_loss(args, true);
    if (rc != ND_OK)
    {
        return rc;
    }
    ND_REQUIRE(args->total && args->partials, "an output is null");
    for (int c = 0; c < args->channels; ++c)
    {
        ND_REQUIRE(args->terms[c], "an output is null");
    }
    auto stream = static_cast<cudaStream_t>(stream_handle);
    const dim3 grid = loss_grid(*args);
    ND_CUDA_TRY(cudaMemsetAsync(args->partials + static_cast<std::int64_t>(grid.x) * grid.y, 0,
                                sizeof(double), stream));
    if (args->dtype == ND_FLOAT32)
    {
        loss_forward_kernel<float><<<grid, kThreads, 0, stream>>>(loss_pass<float>(*args));
    }
    else
    {
        loss_forward_kernel<double><<<grid, kThreads, 0, stream>>>(loss_pass<double>(*args));
    }
    ND_LAUNCH_CHECK();
    return ND_OK;
}

int nd_loss_backward(const nd_loss_args* args, nd_stream_t stream_handle)
{
    using namespace nd;
    const int rc = check_loss(args, false);
    if (rc != ND_OK)
    {
        return rc;
    }
    auto stream = static_cast<cudaStream_t>(stream_handle);
    if (args->dtype == ND_FLOAT32)
    {
        loss_backward_kernel<float><<<loss_grid(*args), kThreads, 0, stream>>>(loss_pass<float>(*args));
    }
    else
    {
        loss_backward_kernel<double><<<loss_grid(*args), kThreads, 0, stream>>>(loss_pass<double>(*args));
    }
    ND_LAUNCH_CHECK();
    return ND_OK;
}

}  // extern "C"
