// Propagation of small batches: a warp per track (core/group.cuh).
//
// Kernel:
//   propagate_group_kernel  one warp, one CTA per track: the propagation loop
//                           in every lane, the candidate searches divided
//                           among the lanes
#include <cuda_runtime.h>

#include "api_common.cuh"
#include "track_io.cuh"

using namespace dprop;

namespace {

// Bound by the latency of one track's chain of operations, so the register
// budget is the largest that keeps every track of the batch resident at once
// (MinBlocks CTAs of one warp per SM: 16 -> 128 registers, 20 -> 96, 32 ->
// 64).  Against one thread per track in 40 registers (B200, toy detector, 2 T,
// tracks 1 / 1 000 / 3 000 / 5 000): 158 / 519 / 830 / 1 265 us against 426 /
// 1 990 / 2 080 / 2 070 us.  Budgets above 128 registers gain another 5 % but
// are compiled with other fused multiply-adds than the other kernels.
template <typename In, bool W, int MinBlocks>
__global__ void __launch_bounds__(32, MinBlocks)
    propagate_group_kernel(const __grid_constant__ detector_view<float, W> det,
                           const __grid_constant__ field_view<float> field,
                           const __grid_constant__ prop_cfg<float> cfg,
                           const __grid_constant__ api::io_ptrs<In> io,
                           uint64_t n) {
    api::run_group<In>(blockIdx.x, n, det, field, cfg, io,
                       lane_group<32>::make(threadIdx.x));
}

template <int MinBlocks, typename In>
void launch_group(cudaStream_t st, const dprop_detector* det,
                  const dprop_field* field, const prop_cfg<float>& cfg,
                  const api::io_ptrs<In>& io, uint64_t n) {
    const unsigned int grid = static_cast<unsigned int>(n);
    if (det->wires) {
        propagate_group_kernel<In, true, MinBlocks><<<grid, 32, 0, st>>>(
            det->view_as<true>(), field->view, cfg, io, n);
    } else {
        propagate_group_kernel<In, false, MinBlocks><<<grid, 32, 0, st>>>(
            det->view_as<false>(), field->view, cfg, io, n);
    }
}

}  // namespace

namespace dprop::api {

dprop_status load_group_forms() {
    cudaFuncAttributes a{};
    const auto load = [&a](auto kernel) {
        return cudaFuncGetAttributes(&a, kernel);
    };
    DPROP_CUDA(load(propagate_group_kernel<float, true, 16>));
    DPROP_CUDA(load(propagate_group_kernel<float, true, 20>));
    DPROP_CUDA(load(propagate_group_kernel<float, true, 32>));
    DPROP_CUDA(load(propagate_group_kernel<float, false, 16>));
    DPROP_CUDA(load(propagate_group_kernel<float, false, 20>));
    DPROP_CUDA(load(propagate_group_kernel<float, false, 32>));
    return DPROP_OK;
}

launch_request::launch_request(const dprop_launch* lc) : given_(lc != nullptr) {
    if (!lc) {
        return;
    }
    shape_ = *lc;
    if (shape_.by_size == 1u) {
        shape_.block_size = shape_.ctas_per_sm = shape_.steps_per_round = 0u;
        shape_.rounds = shape_.yield_lanes = shape_.sort_interval = 0u;
        shape_.tail_tracks = shape_.by_size = 0u;
    }
}

bool open_shape(const dprop_launch* lc) {
    return !lc || (lc->block_size | lc->ctas_per_sm | lc->steps_per_round |
                   lc->rounds | lc->yield_lanes | lc->sort_interval |
                   lc->tail_tracks) == 0u;
}

bool use_group(const dprop_launch* lc, const dprop_detector* det,
               const dprop_config& cfg, uint64_t n) {
    // a launch shape that is spelled out is launched as it is
    return open_shape(lc) && cfg.use_field_gradient == 0 &&
           n <= group_limit(det->traits, cfg.search_window);
}

template <typename In>
dprop_status enqueue_group(const dprop_detector* det, const dprop_field* field,
                           const prop_cfg<float>& cfg, const io_ptrs<In>& io,
                           uint64_t n, cudaStream_t st) {
    int dev = 0, sms = 0;
    DPROP_CUDA(cudaGetDevice(&dev));
    DPROP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint64_t per_sm = (n + static_cast<uint64_t>(sms) - 1u) /
                            static_cast<uint64_t>(sms);
    if (per_sm <= 16u) {
        launch_group<16>(st, det, field, cfg, io, n);
    } else if (per_sm <= 20u) {
        launch_group<20>(st, det, field, cfg, io, n);
    } else {
        launch_group<32>(st, det, field, cfg, io, n);
    }
    DPROP_CUDA(cudaGetLastError());
    return DPROP_OK;
}

template dprop_status enqueue_group<float>(const dprop_detector*,
                                           const dprop_field*,
                                           const prop_cfg<float>&,
                                           const io_ptrs<float>&, uint64_t,
                                           cudaStream_t);
template dprop_status enqueue_group<double>(const dprop_detector*,
                                            const dprop_field*,
                                            const prop_cfg<float>&,
                                            const io_ptrs<double>&, uint64_t,
                                            cudaStream_t);

}  // namespace dprop::api
