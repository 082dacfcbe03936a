// TEST-ONLY: the batch sizes at which an open launch shape changes its form.
#include "core/convert.hpp"
#include "core/launch_rules.hpp"

using namespace dprop;

// extra_code: as the library finds it (line surfaces, rods, multi-entry bins,
// material maps, volume material)
extern "C" int plain_budget_of(const dprop_detector_desc* d, int extra_code,
                               const uint32_t* window, int field_map,
                               uint64_t tracks_per_sm) {
    return plain_budget(launch_traits_of(d, extra_code != 0), window,
                        field_map != 0, tracks_per_sm);
}

extern "C" uint32_t tail_of(uint64_t n) { return default_tail_tracks(n); }

extern "C" uint64_t host_scratch(uint64_t n, uint64_t max_records) {
    return host_scratch_bytes(n, max_records);
}

extern "C" int scan_clusters(const dprop_detector_desc* d, uint64_t n) {
    uint32_t unbounded = 0u;
    for (const scan_bound& b : scan_bounds(d)) {
        unbounded += b.radius < 0.f ? 1u : 0u;
    }
    return scan_in_clusters(unbounded, n) ? 1 : 0;
}

extern "C" int drops_order(const dprop_detector_desc* d, int staged,
                           uint64_t n) {
    return order_is_a_loss(launch_traits_of(d, false), staged != 0, n) ? 1 : 0;
}

extern "C" int launch_rules(const dprop_detector_desc* d, int extra_code,
                            const uint32_t* window, int field_map,
                            uint64_t* out) {
    if (!validate_desc(d).empty()) {
        return 1;
    }
    const launch_traits t = launch_traits_of(d, extra_code != 0);
    out[0] = group_limit(t, window);
    out[1] = group_limit_fp64(t, window);
    out[2] = group_limit_adjoint(t, window, false);
    out[3] = group_limit_adjoint(t, window, true);
    out[4] = rounds_from(t, field_map != 0);
    out[5] = rounds_from_fp64(t);
    return 0;
}
