// Pieces of the C ABI implementation shared by its translation units
// (dprop_api.cu: propagation; adjoint_api.cu: adjoint mode and the reverse
// sweep): error reporting, the detector and field handles, the direction
// sort of the inputs and the register-budget choice of a launch.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "core/launch_rules.hpp"
#include "core/propagate.cuh"
#include "detray_b200/dprop.h"

namespace dprop::api {

// Record msg as dprop_last_error() of this thread and return s.
dprop_status fail(dprop_status s, const std::string& msg);
dprop_status cuda_fail(cudaError_t e, const char* what);

// The launch, with its shape left open if by_size says so.
struct launch_request {
    explicit launch_request(const dprop_launch* lc);
    const dprop_launch* get() const { return given_ ? &shape_ : nullptr; }

private:
    dprop_launch shape_{};
    bool given_;
};

// Register budget a launch spells out: resident CTAs of 128 threads per SM, one
// of 8 (64 registers), 12 (40) or 16 (32).
int occupancy_of(const dprop_launch* lc);

// Device memory the library keeps between calls: one grow-only buffer per
// device, shared by all callers.  A call holds it (use) from take() until its
// work is enqueued, so that calls of several host threads do not interleave,
// and its work starts after that of the call before it, on whichever stream
// that was: calls on several streams that need the same buffer run one after
// the other, they do not overwrite each other.
class kept_scratch {
    struct slot {
        void* buf{nullptr};
        size_t bytes{0};
        cudaEvent_t last{nullptr};  // the last call's work on the buffer
        bool captured{false};       // a stream capture holds its address
    };

public:
    // spare: given back when an allocation here finds no memory
    explicit kept_scratch(kept_scratch* spare = nullptr) : spare_(spare) {}

    class use {
    public:
        use() = default;
        use(const use&) = delete;
        use& operator=(const use&) = delete;
        ~use();
        void* buf{nullptr};

    private:
        friend class kept_scratch;
        std::unique_lock<std::mutex> lock_;
        cudaEvent_t last_{nullptr};  // recorded at the end (not in a capture)
        cudaStream_t stream_{nullptr};
    };

    // At least `bytes` on the current device for work on `stream`.  Inside a
    // stream capture the captured work is not ordered against other calls
    // (an event from outside a capture cannot be waited for in it).
    cudaError_t take(size_t bytes, cudaStream_t stream, use* u);
    // Frees the buffers of all devices.
    void release();
    // Frees the current device's buffer; whether there was one.
    bool give_back();

private:
    kept_scratch* spare_;
    std::mutex mutex_;
    std::vector<slot> slots_;      // by device
    std::vector<void*> retired_;   // outgrown, but in a captured graph
};

// The staging area of sorted plain propagations.
kept_scratch* staging_area();

// cudaMalloc; without room for it the staging area of sorted propagations, an
// option that is kept between calls, is given back first.
cudaError_t alloc_device(void** p, size_t bytes);

// Number of a new detector or field handle, never given twice: a cached
// CUDA graph is matched by it, since the address of a destroyed handle may be
// the next one's.
uint64_t next_handle_id();

// Device scratch bytes of enqueue_direction_sort for n tracks.
size_t sort_scratch_bytes(uint64_t n);

// Enqueue the sort of n tracks by direction, charge and pT (20-bit key,
// CUB radix sort) on stream; *order receives the device array of sorted track
// indices, which lives in scratch.  No allocation, no synchronisation.
dprop_status enqueue_direction_sort(const float* dx, const float* dy,
                                    const float* dz, const float* dq,
                                    uint64_t n, void* scratch,
                                    size_t scratch_bytes, cudaStream_t stream,
                                    const uint32_t** order);
dprop_status enqueue_direction_sort(const double* dx, const double* dy,
                                    const double* dz, const double* dq,
                                    uint64_t n, void* scratch,
                                    size_t scratch_bytes, cudaStream_t stream,
                                    const uint32_t** order);

}  // namespace dprop::api

#define DPROP_CUDA(call)                                      \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess) {                              \
            return ::dprop::api::cuda_fail(e_, #call);        \
        }                                                     \
    } while (0)

struct dprop_detector {
    int device{0};
    uint64_t id{dprop::api::next_handle_id()};
    dprop::dev_volume* volumes{nullptr};
    dprop::dev_surface* surfaces{nullptr};
    dprop::dev_nav_surface<float>* nav_surfaces{nullptr};
    dprop::dev_nav_surface<double>* nav_surfaces_d{nullptr};
    dprop::dev_mask<float>* masks{nullptr};
    dprop::dev_transform<float>* transforms{nullptr};
    dprop::dev_slab<float>* slabs{nullptr};
    uint32_t* bf_surfaces{nullptr};
    dprop::dev_grid<float>* grids{nullptr};
    uint32_t* grid_bins{nullptr};
    uint32_t* vol_material{nullptr};  // NULL: no volume carries material
    dprop::scan_bound* scan_bounds{nullptr};  // [n_surfaces]
    // double-precision copies of the floating-point tables (fp64 launches)
    dprop::dev_mask<double>* masks_d{nullptr};
    dprop::dev_transform<double>* transforms_d{nullptr};
    dprop::dev_slab<double>* slabs_d{nullptr};
    dprop::dev_grid<double>* grids_d{nullptr};
    uint32_t n_volumes{0}, n_surfaces{0};
    // the detector holds line surfaces, material rods, multi-entry grid bins,
    // material maps or volume material: launches use the kernels that
    // include the code for them
    bool wires{false};
    dprop::launch_traits traits;
    uint32_t n_unbounded{0};  // surfaces the truth scan searches for any track
    dprop::detector_view<double> view_d() const { return view_d_as<true>(); }
    template <bool W>
    dprop::detector_view<double, W> view_d_as() const {
        dprop::detector_view<double, W> v;
        v.volumes = volumes;
        v.surfaces = surfaces;
        v.nav_surfaces = nav_surfaces_d;
        v.masks = masks_d;
        v.transforms = transforms_d;
        v.slabs = slabs_d;
        v.bf_surfaces = bf_surfaces;
        v.grids = grids_d;
        v.grid_bins = grid_bins;
        v.vol_material = vol_material;
        v.n_volumes = n_volumes;
        v.n_surfaces = n_surfaces;
        return v;
    }
    dprop::detector_view<float> view() const { return view_as<true>(); }
    template <bool W>
    dprop::detector_view<float, W> view_as() const {
        dprop::detector_view<float, W> v;
        v.volumes = volumes;
        v.surfaces = surfaces;
        v.nav_surfaces = nav_surfaces;
        v.masks = masks;
        v.transforms = transforms;
        v.slabs = slabs;
        v.bf_surfaces = bf_surfaces;
        v.grids = grids;
        v.grid_bins = grid_bins;
        v.vol_material = vol_material;
        v.n_volumes = n_volumes;
        v.n_surfaces = n_surfaces;
        return v;
    }
};

struct dprop_field {
    int device{0};
    uint64_t id{dprop::api::next_handle_id()};
    float4* nodes{nullptr};
    dprop::field_view<float> view{};
    dprop::field_view<double> view_d{};  // same nodes, double arithmetic
};

namespace dprop::api {

// fp64 propagation (dprop_launch.precision == 8): double inputs, arithmetic
// and results; the forms of group_limit_fp64 and rounds_from_fp64
// (core/launch_rules.hpp), optional direction sort.
dprop_status propagate_fp64(const dprop_config& cfg, const dprop_launch* lc,
                            const dprop_detector* det, const dprop_field* field,
                            const dprop_tracks& tracks,
                            const dprop_results& results, uint64_t n,
                            cudaStream_t stream);

// Frees the grow-only scratch of fp64 launches (dprop_release_cache).
void release_fp64_scratch();

}  // namespace dprop::api
