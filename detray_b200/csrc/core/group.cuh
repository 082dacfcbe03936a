// A track in several lanes of a warp.
//
// One thread per track leaves most of the GPU idle when a batch is small, and
// the time of the batch is then the serial latency of its slowest track: a
// volume switch alone walks some 50 grid bins one after the other, each a
// chain of dependent loads.  With a group of L lanes per track every lane
// carries the track's whole state and executes the same operations on it
// (so they need no exchange), and the lanes divide the candidate searches
// among them.  The candidates enter the cache in the order a single thread
// finds them in, so a track's results do not depend on the form.
#pragma once

#include "navigator.cuh"

namespace dprop {

// The L lanes of a warp that run one track.  All lanes of a group call every
// member together.  The kernels use whole warps: 8 and 16 lanes per track were
// never clearly faster at any batch size.
template <int L>
struct lane_group {
    static_assert(L == 32, "a warp per track");
    static constexpr int lanes = L;
    static constexpr bool packed = false;
    uint32_t mask;   // the group's lanes in the warp
    int rank;        // lane in the group

    DPROP_D static lane_group make(uint32_t lane) {
        lane_group g;
        g.rank = static_cast<int>(lane % static_cast<uint32_t>(L));
        const uint32_t all = L == 32 ? 0xffffffffu : (1u << (L % 32)) - 1u;
        g.mask = all << (lane - static_cast<uint32_t>(g.rank));
        return g;
    }
    DPROP_D bool leader() const { return rank == 0; }
    // one bit per lane of the group
    DPROP_D uint32_t ballot(bool p) const {
        const uint32_t b = __ballot_sync(mask, p) & mask;
        return b >> (__ffs(mask) - 1);
    }
    DPROP_D uint32_t count(bool p) const {
        return static_cast<uint32_t>(__popc(__ballot_sync(mask, p) & mask));
    }
    DPROP_D int first(uint32_t bits) const { return __ffs(bits) - 1; }
    template <typename T>
    DPROP_D T bcast(T v, int src) const {
        return __shfl_sync(mask, v, src, L);
    }
    template <typename S>
    DPROP_D candidate<S> bcast(const candidate<S>& c, int src) const {
        const uint32_t info = static_cast<uint32_t>(c.volume_link) |
                              (static_cast<uint32_t>(c.status) << 16) |
                              (static_cast<uint32_t>(c.flags) << 24);
        const uint32_t r = bcast(info, src);
        candidate<S> o;
        o.path = bcast(c.path, src);
        o.sf = bcast(c.sf, src);
        o.volume_link = static_cast<uint16_t>(r & 0xffffu);
        o.status = static_cast<uint8_t>((r >> 16) & 0xffu);
        o.flags = static_cast<uint8_t>(r >> 24);
        return o;
    }
    // inclusive sum over the group
    DPROP_D uint32_t scan(uint32_t v) const {
        for (int o = 1; o < L; o *= 2) {
            const uint32_t u = __shfl_up_sync(mask, v, o, L);
            v += rank >= o ? u : 0u;
        }
        return v;
    }
    // first lane whose inclusive sum exceeds f (the last one if none does)
    DPROP_D int owner(uint32_t end, uint32_t f) const {
        int lo = 0;
        for (int step = L / 2; step > 0; step /= 2) {
            const uint32_t e = bcast(end, lo + step - 1);
            lo += e <= f ? step : 0;
        }
        return lo;
    }
};

// The caching navigator run by a group (caching_navigation for one lane).
template <typename G>
struct group_navigation {
    static constexpr bool fixed_rounding = true;
    G g;
    template <typename S, bool W>
    DPROP_D bool update(nav_state<S>& nav, const detector_view<S, W>& det,
                        const track_view<S>& trk, const nav_cfg<S>& cfg,
                        bool first) {
        return navigator_update(nav, det, trk, cfg, first, g);
    }
};

}  // namespace dprop
