// fp64 propagation: the propagation core instantiated in double precision
// (the reference's full-fp64 build, DETRAY_CUSTOM_SCALARTYPE=double), for
// dprop_propagate with dprop_launch.precision = 8.  Track arrays, arithmetic
// and results are double; the field map nodes stay float4 (the reference's
// covfie field stores floats) and are interpolated in double.
//
// Kernels:
//   propagate_fp64_kernel<MB>  one thread per track, the whole propagation,
//                              register budget MB resident CTAs of 128
//                              threads per SM
//   propagate_fp64_group_kernel  small batches: a warp per track
//   the round-based phase kernels of rounds.cuh in double
//                              (dprop_launch.method = DPROP_METHOD_PERSISTENT)
#include <cuda_runtime.h>

#include <type_traits>

#include "api_common.cuh"
#include "core/config.hpp"
#include "track_io.cuh"

using namespace dprop;
using dprop::api::fail;

namespace {

constexpr int k_f64_block = 128;

template <int MinBlocks, bool W, bool Grad = false>
__global__ void __launch_bounds__(k_f64_block, MinBlocks)
    propagate_fp64_kernel(const __grid_constant__ detector_view<double, W> det,
                          const __grid_constant__ field_view<double> field,
                          const __grid_constant__ prop_cfg<double> cfg,
                          const __grid_constant__ api::io_ptrs<double, double> io, uint64_t n,
                          const uint32_t* __restrict__ order) {
    const uint64_t i =
        static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    const uint64_t t = order ? static_cast<uint64_t>(order[i]) : i;
    api::run_one<double, false, double, W, Grad>(t, n, det, field, cfg, io);
}

// A warp per track, as propagate_group_kernel (group_api.cu); 255 registers
// while that keeps the batch resident (8 warps per SM), else 128.
template <int MinBlocks, bool W>
__global__ void __launch_bounds__(32, MinBlocks)
    propagate_fp64_group_kernel(
        const __grid_constant__ detector_view<double, W> det,
        const __grid_constant__ field_view<double> field,
        const __grid_constant__ prop_cfg<double> cfg,
        const __grid_constant__ api::io_ptrs<double, double> io, uint64_t n) {
    api::run_group<double>(blockIdx.x, n, det, field, cfg, io,
                           lane_group<32>::make(threadIdx.x));
}

// kept between fp64 calls: the direction sort's scratch, and the persistent
// method's slots and queues; a call takes the sort's first
api::kept_scratch g_f64_sort{api::staging_area()};
api::kept_scratch g_f64_rounds{api::staging_area()};

}  // namespace

namespace dprop::api {

dprop_status propagate_fp64(const dprop_config& c, const dprop_launch* lc,
                            const dprop_detector* det, const dprop_field* field,
                            const dprop_tracks& tracks,
                            const dprop_results& results, uint64_t n,
                            cudaStream_t stream) {
    if (n > 0x7fffffffull * k_f64_block) {
        return fail(DPROP_E_INVALID, "propagate fp64: too many tracks");
    }
    const io_ptrs<double, double> io = make_io<double, double>(tracks, results);
    const prop_cfg<double> pc = make_prop_cfg<double>(c);
    int dev = 0, sms = 0;
    DPROP_CUDA(cudaGetDevice(&dev));
    DPROP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint64_t per_sm = n / static_cast<uint64_t>(sms);
    const bool open = open_shape(lc) && c.use_field_gradient == 0;
    if (open && n <= group_limit_fp64(det->traits, c.search_window)) {
        auto go = [&](auto view) {
            constexpr bool W =
                std::is_same<decltype(view), detector_view<double, true>>::value;
            const unsigned int grid = static_cast<unsigned int>(n);
            if (per_sm < 8u) {
                propagate_fp64_group_kernel<8, W><<<grid, 32, 0, stream>>>(
                    view, field->view_d, pc, io, n);
            } else {
                propagate_fp64_group_kernel<16, W><<<grid, 32, 0, stream>>>(
                    view, field->view_d, pc, io, n);
            }
        };
        if (det->wires) {
            go(det->view_d_as<true>());
        } else {
            go(det->view_d_as<false>());
        }
        DPROP_CUDA(cudaGetLastError());
        return DPROP_OK;
    }
    kept_scratch::use sort_use, rounds_use;
    const uint32_t* order = nullptr;
    if (lc && lc->sort_tracks) {
        const size_t need = sort_scratch_bytes(n);
        DPROP_CUDA(g_f64_sort.take(need, stream, &sort_use));
        const dprop_status s = enqueue_direction_sort(
            io.trk[4], io.trk[5], io.trk[6], io.trk[7], n, sort_use.buf, need,
            stream, &order);
        if (s != DPROP_OK) {
            return s;
        }
    }
    if (lc && lc->method == DPROP_METHOD_PERSISTENT &&
        !(open && n < rounds_from_fp64(det->traits))) {
        const size_t need = rounds_scratch_bytes_fp64(
            n, det->wires, staged_capacity(pc, io));
        DPROP_CUDA(g_f64_rounds.take(need, stream, &rounds_use));
        return enqueue_rounds_fp64(lc, det, field, pc, io, n, order,
                                   rounds_use.buf, need, stream);
    }
    const unsigned int grid =
        static_cast<unsigned int>((n + k_f64_block - 1) / k_f64_block);
    // the register budget (CTAs of 128 threads per SM: 2 -> 255 registers, 4
    // -> 128, 8 -> 64): the largest that keeps the batch resident, unless it
    // is spelled out (8 or 12).  Toy in the map, 30 000 sorted tracks: 2 932 us
    // against 3 966 in 64 and 4 753 in 40 registers.
    int mb = occupancy_of(lc) >= 12 ? 12 : 8;
    if (!(lc && lc->ctas_per_sm)) {
        mb = per_sm < 256u ? 2 : (per_sm < 512u ? 4 : 8);
    }
    auto go = [&](auto view) {
        constexpr bool W =
            std::is_same<decltype(view), detector_view<double, true>>::value;
        if (c.use_field_gradient) {
            propagate_fp64_kernel<8, W, true><<<grid, k_f64_block, 0, stream>>>(
                view, field->view_d, pc, io, n, order);
        } else if (mb == 2) {
            propagate_fp64_kernel<2, W><<<grid, k_f64_block, 0, stream>>>(
                view, field->view_d, pc, io, n, order);
        } else if (mb == 4) {
            propagate_fp64_kernel<4, W><<<grid, k_f64_block, 0, stream>>>(
                view, field->view_d, pc, io, n, order);
        } else if (mb == 12) {
            propagate_fp64_kernel<12, W><<<grid, k_f64_block, 0, stream>>>(
                view, field->view_d, pc, io, n, order);
        } else {
            propagate_fp64_kernel<8, W><<<grid, k_f64_block, 0, stream>>>(
                view, field->view_d, pc, io, n, order);
        }
    };
    if (det->wires) {
        go(det->view_d_as<true>());
    } else {
        go(det->view_d_as<false>());
    }
    DPROP_CUDA(cudaGetLastError());
    return DPROP_OK;
}

void release_fp64_scratch() {
    g_f64_sort.release();
    g_f64_rounds.release();
}

}  // namespace dprop::api
