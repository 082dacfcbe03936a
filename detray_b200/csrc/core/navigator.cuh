// Navigation: the candidate cache, its trust-level update and the volume
// search, one track per thread.
//
// Follows the reference's caching navigator step for step so that the
// sequence of surfaces a track crosses is the same:
//   cache state         navigation/navigation_state.hpp:67-668
//   insert              navigation/caching_navigator.hpp:149-229
//   update_impl         navigation/caching_navigator.hpp:250-369
//   init / update       navigation/navigator_base.hpp:56-154
//   candidate_search    navigation/detail/navigation_functions.hpp:26-81
//   update_candidate    navigation/detail/navigation_functions.hpp:99-129
//   update_status       navigation/detail/navigation_functions.hpp:147-177
//   local_navigation    navigation/detail/navigation_functions.hpp:193-246
//   volume_switch       navigation/detail/navigation_functions.hpp:264-288
//   init_loose_cfg      navigation/detail/navigation_functions.hpp:304-331
//   intersection kernel navigation/detail/intersection_kernel.hpp:24-272
//   grid search         navigation/accelerators/spatial_grid.hpp:100-201,
//                       utils/grid/detail/axis_binning.hpp, axis_bounds.hpp,
//                       utils/grid/detail/bin_view.hpp (axis 0 outer loop)
#pragma once

#include <type_traits>

#include "geometry.cuh"

namespace dprop {

constexpr int k_cache = 8;  // navigation::default_cache_size

enum nav_status : int8_t {
    e_nav_abort = -3,
    e_nav_exit = -2,
    e_nav_unknown = -1,
    e_towards_object = 0,
    e_on_object = 1,
    e_on_portal = 2,
};

enum trust_level : uint8_t {
    e_no_trust = 0,
    e_fair_trust = 1,
    e_high_trust = 3,
    e_full_trust = 4,
};

enum abort_reason : uint8_t {
    e_reason_none = 0,
    e_reason_path_limit = 1,
    e_reason_stalled = 2,
    e_reason_no_surface = 3,
    e_reason_nonfinite = 4,
};

template <typename S>
struct nav_cfg {
    isect_cfg<S> isect;
    uint32_t win0, win1;
};

// Navigation state without the candidate cache.
template <typename S>
struct nav_meta {
    int8_t next;
    int8_t last;
    int8_t status;
    uint8_t trust;
    uint32_t volume;
    S external_tol;
    S direction;  // +1 forward, -1 backward
    uint8_t reason;
    uint32_t n_isect;  // ray-surface intersections evaluated

    DPROP_HD bool is_alive() const { return status > e_nav_unknown; }
    DPROP_HD bool finished() const { return status == e_nav_exit; }
    DPROP_HD bool is_on_surface() const {
        return status == e_on_object || status == e_on_portal;
    }
    DPROP_HD bool is_on_portal() const { return status == e_on_portal; }
    DPROP_HD int n_candidates() const { return last - next + 1; }
    DPROP_HD bool cache_exhausted() const { return n_candidates() == 0; }
    DPROP_HD int begin_index() const {
        return (is_on_surface() && next >= 1) ? next - 1 : next;
    }
    DPROP_HD int end_index() const { return last + 1; }
    DPROP_HD void set_no_trust() { trust = e_no_trust; }
    DPROP_HD void set_high_trust() {
        trust = trust < e_high_trust ? trust : e_high_trust;
    }
    DPROP_HD void set_fair_trust() {
        trust = trust < e_fair_trust ? trust : e_fair_trust;
    }
    DPROP_HD void set_volume(uint32_t v) {
        if (v != volume) {
            set_no_trust();
        }
        volume = v;
    }
    DPROP_HD void abort(uint8_t why) {
        status = e_nav_abort;
        reason = why;
    }
};

template <typename S>
struct nav_state : nav_meta<S> {
    static constexpr bool packed = false;
    // k_cache candidates plus one sentinel slot: when the last cached
    // candidate is reached the next index points one past the cache, and a
    // read there (which the reference does on its fixed-size array) finds
    // an unreachable candidate instead of leaving the state.
    // The cache lives outside this struct, in an array of k_cache + 1
    // candidates the owner binds here (nav_cache): indexed with the
    // run-time cache index, an array inside the state would make the
    // compiler keep the whole per-track state in the thread's stack instead
    // of registers.
    candidate<S>* cand;

    DPROP_HD void reset(uint32_t vol) {
        for (int i = 0; i <= k_cache; ++i) {
            cand[i] = invalid_candidate<S>();
        }
        this->next = 0;
        this->last = -1;
        this->status = e_nav_unknown;
        this->trust = e_no_trust;
        this->volume = vol;
        this->external_tol = S(0);
        this->direction = S(1);
        this->reason = e_reason_none;
        this->n_isect = 0u;
    }
    DPROP_HD candidate<S>& current() { return cand[this->next - 1]; }
    DPROP_HD const candidate<S>& current() const {
        return cand[this->next - 1];
    }
    DPROP_HD candidate<S>& target() { return cand[this->next]; }
    DPROP_HD const candidate<S>& target() const { return cand[this->next]; }
    // the target was reached: the next candidate becomes the target
    DPROP_HD void reached() { ++this->next; }
    // distance to the next candidate along the navigation direction
    DPROP_HD S dist() const { return this->direction * target().path; }
    DPROP_HD void clear_cache() {
        for (int i = 0; i < k_cache; ++i) {
            cand[i].path = limits<S>::max();
        }
        this->next = 0;
        this->last = -1;
    }
};

// Storage of a candidate cache (k_cache candidates and the sentinel); bind
// it to a state with bind_cache before the state is used.
template <typename S>
struct nav_cache {
    candidate<S> c[k_cache + 1];
};

template <typename S>
DPROP_HD void bind_cache(nav_state<S>& nav, nav_cache<S>& cache) {
    nav.cand = cache.c;
}

// Track position and direction seen by the navigator
template <typename S>
struct track_view {
    vec3<S> pos;
    vec3<S> dir;
};

#if defined(DPROP_TRACE) && !defined(__CUDA_ARCH__)
}  // namespace dprop
#include <cstdio>
namespace dprop {
template <typename S>
void nav_trace(const nav_state<S>& nav, const char* msg, vec3<S> p) {
    std::printf("[%s] st=%d trust=%d vol=%u pos=(%.4f %.4f %.4f)\n", msg,
                (int)nav.status, (int)nav.trust, (unsigned)nav.volume,
                (double)p.x, (double)p.y, (double)p.z);
    for (int i = 0; i < k_cache; ++i) {
        const candidate<S>& c = nav.cand[i];
        std::printf("   c%d sf=%u path=%.6f st=%d vl=%u\n", i,
                    c.sf == k_invalid ? 9999999u : c.sf,
                    c.path > S(1e30) ? -1.0 : (double)c.path, (int)c.status,
                    (unsigned)c.volume_link);
    }
}
#define DPROP_NAV_TRACE(nav, msg, p) nav_trace(nav, msg, p)
#else
#define DPROP_NAV_TRACE(nav, msg, p)
#endif

// --------------------------------------------------------- cache insert
template <typename S>
DPROP_HD void nav_insert(nav_state<S>& nav, const candidate<S>& nc) {
    // upper_bound over [begin, end) with |path| ordering
    const int b = nav.begin_index();
    const int e = nav.end_index();
    int pos = e;
    const S apath = fabs(nc.path);
    DPROP_ROLLED
    for (int i = b; i < e; ++i) {
        if (apath < fabs(nav.cand[i].path)) {
            pos = i;
            break;
        }
    }
    if (pos == k_cache) {
        return;  // too far away to be cached
    }
    if (nav.n_candidates() == 0) {
        nav.cand[0] = nc;
        nav.last = static_cast<int8_t>(nav.last + 1);
        return;
    }
    const S um = S(unit::um);
    // the same surface (same index <=> same barcode) at an overlapping path
    // is not added twice
    if ((nav.cand[pos].sf == nc.sf &&
         fabs(nav.cand[pos].path - nc.path) <= um) ||
        (pos > 0 && nav.cand[pos - 1].sf == nc.sf &&
         fabs(nav.cand[pos - 1].path - nc.path) <= um)) {
        return;
    }
    const int shift_max = k_cache - 2;
    const int shift_begin = nav.last < shift_max ? nav.last : shift_max;
    // prefer sensitives over portals and direct over edge hits
    if (fabs(nav.cand[pos].path - nc.path) <= um &&
        (nc.is_edge() || nc.is_portal())) {
        ++pos;
        pos = pos > shift_begin ? shift_begin : pos;
    }
    DPROP_ROLLED
    for (int i = shift_begin; i >= pos; --i) {
        nav.cand[i + 1] = nav.cand[i];
    }
    nav.cand[pos] = nc;
    const int nl = nav.last + 1;
    nav.last = static_cast<int8_t>(nl < k_cache - 1 ? nl : k_cache - 1);
}

// How many lanes work on one track.  one_lane: a thread per track.  The
// device's lane_group (group.cuh) runs a track in several lanes of a warp:
// every lane holds the track's whole state and executes the same operations,
// only the candidate searches are divided among them.
// packed: surfaces are read as one record (dev_nav_surface), 20 registers
// loaded at once, instead of through the surface, transform and mask tables.
// It shortens the chain of dependent loads where that is what a kernel waits
// for: the phases of the round-based method (toy 1.5 M 27.5 -> 25.1 ms, in the
// map 33.5 -> 30.7 ms), the direct navigator (300 k 1.27 -> 1.20 ms) and double
// precision (200 k 11.6 -> 11.0 ms).  The fp32 kernels that run the whole loop
// wait for instructions and registers and lose by it (1 M 21.0 -> 22.0 ms).
struct one_lane {
    static constexpr int lanes = 1;
    static constexpr bool packed = false;
};
struct one_lane_packed {
    static constexpr int lanes = 1;
    static constexpr bool packed = true;
};
// whether kernels in S for detectors W read packed records with trait P
template <typename S, bool W, typename P>
constexpr bool use_packed() {
    return !W && (P::packed || sizeof(S) == 8);
}

// -------------------------------------------- intersection_initialize
// Intersection of the ray with a surface of the packed table (planar or
// concentric cylinder); false if there is none within reach.
template <typename S>
DPROP_HD bool nav_intersect(const dev_nav_surface<S>& sf, vec3<S> ro,
                            vec3<S> rd, S overstep, isect_point<S>& ip) {
    if (sf.shape() == e_concentric_cylinder) {
        ip = intersect_portal_cylinder(ro, rd, sf.v[0], overstep);
    } else {
        ip = intersect_plane_at(ro, rd, vec3<S>{sf.n[0], sf.n[1], sf.n[2]},
                                vec3<S>{sf.t[0], sf.t[1], sf.t[2]});
    }
    return ip_valid(ip.path);
}

// Candidate c from the intersection ip of surface sf_idx: the masks in turn
// until one accepts it (resolve_mask for each).  With Fresh every mask starts
// from an unset candidate (a search), else c keeps what a mask beyond the
// overstepping tolerance leaves untouched (an update).
template <bool Fresh, typename S, bool W>
DPROP_HD bool nav_resolve(candidate<S>& c, const isect_point<S>& ip,
                          uint32_t sf_idx, const dev_nav_surface<S>& sf,
                          const detector_view<S, W>& det,
                          const isect_cfg<S>& cfg, S external_tol) {
    const uint8_t shape = sf.shape();
    S l0 = S(0), l1 = S(0);
    if (shape != e_concentric_cylinder) {
        l0 = add_rn(dot_rn(vec3<S>{sf.ax[0], sf.ax[1], sf.ax[2]}, ip.glob),
                    sf.tx);
        l1 = add_rn(dot_rn(vec3<S>{sf.ay[0], sf.ay[1], sf.ay[2]}, ip.glob),
                    sf.ty);
    }
    dev_mask<S> m;
    m.v[0] = sf.v[0];
    m.v[1] = sf.v[1];
    m.v[2] = sf.v[2];
    m.v[3] = sf.v[3];
    m.volume_link = sf.info & 0xffffu;
    const uint32_t n_masks =
        sf.multi() ? static_cast<uint32_t>(det.surfaces[sf_idx].n_masks) : 1u;
    for (uint32_t i = 0;;) {
        if (Fresh) {
            c = invalid_candidate<S>();
        }
        c.status = e_outside;
        if (ip.path >= cfg.overstep_tol) {
            S base_tol = S(0);
            S ext_tol = S(0);
            if (sf.kind() != e_portal || cfg.min_tol_is_max) {
                ext_tol = external_tol;
                base_tol = max_(cfg.min_mask_tol,
                                min_(cfg.max_mask_tol,
                                     cfg.mask_tol_scalor * fabs(ip.path)));
            }
            mask_result<S> r;
            if (shape == e_rectangle) {
                r = check_rectangle(m, l0, l1, base_tol, ext_tol);
            } else if (shape == e_trapezoid) {
                r = check_trapezoid(m, l0, l1, base_tol, ext_tol);
            } else if (shape == e_ring) {
                r = check_ring(m, perp(vec3<S>{l0, l1, S(0)}), base_tol);
            } else {
                r = check_portal_z(m, ip.glob.z, base_tol);
            }
            if (r.edge) {
                c.status = e_edge;
            }
            if (r.inside) {
                c.status = e_inside;
            }
            c.path = ip.path;
            c.sf = sf_idx;
            c.flags = static_cast<uint8_t>((signbit(ip.path) ? 0u : 1u) |
                                           (sf.kind() == e_portal ? 2u : 0u));
            c.volume_link = static_cast<uint16_t>(m.volume_link);
        }
        if (c.is_probably_inside()) {
            return true;
        }
        if (++i >= n_masks) {
            return false;
        }
        m = det.masks[sf.mask_begin + i];
    }
}

// Intersection with a surface of any shape but the general cylinder and the
// resolution of its masks through the tables (Fresh as in nav_resolve).
template <bool Fresh, typename S, bool W>
DPROP_HD bool table_resolve(candidate<S>& c, const detector_view<S, W>& det,
                            uint32_t sf_idx, const dev_surface& sf,
                            vec3<S> ro, vec3<S> rd, const isect_cfg<S>& cfg,
                            S external_tol) {
    const dev_transform<S>& trf = det.transforms[sf.transform];
    const uint32_t m0 = sf.mask_begin;
    const uint32_t m1 = sf.mask_begin + sf.n_masks;
    isect_point<S> ip;
    if (sf.shape == e_concentric_cylinder) {
        ip = intersect_portal_cylinder(ro, rd, det.masks[m0].v[0],
                                       cfg.overstep_tol);
    } else if (W && sf.shape == e_line) {
        ip = intersect_line(ro, rd, trf);
    } else {
        ip = intersect_plane(ro, rd, trf);
    }
    if (!ip_valid(ip.path)) {
        return false;
    }
    for (uint32_t mi = m0; mi < m1; ++mi) {
        if (Fresh) {
            c = invalid_candidate<S>();
        }
        resolve_mask<W>(c, ip, sf_idx, sf, det.masks[mi], trf, cfg,
                        external_tol);
        if (c.is_probably_inside()) {
            return true;
        }
    }
    return false;
}

// General cylinder: both solutions of the first masks that accept them.
template <typename S, bool W>
DPROP_HD void cylinder_candidates(nav_state<S>& nav,
                                  const detector_view<S, W>& det,
                                  uint32_t sf_idx, const dev_surface& sf,
                                  vec3<S> ro, vec3<S> rd,
                                  const isect_cfg<S>& cfg) {
    const dev_transform<S>& trf = det.transforms[sf.transform];
    const uint32_t m0 = sf.mask_begin;
    const uint32_t m1 = sf.mask_begin + sf.n_masks;
    isect_point<S> ips[2];
    intersect_cylinder(ro, rd, trf, det.masks[m0].v[0], ips);
    if (!ip_valid(ips[0].path) && !ip_valid(ips[1].path)) {
        return;
    }
    for (uint32_t mi = m0; mi < m1; ++mi) {
        candidate<S> is = invalid_candidate<S>();
        int n_found = 0;
        for (int i = 0; i < 2; ++i) {
            resolve_mask<W>(is, ips[i], sf_idx, sf, det.masks[mi], trf, cfg,
                            nav.external_tol);
            if (is.is_probably_inside()) {
                nav_insert(nav, is);
                ++n_found;
            }
            if (n_found == 2) {
                return;
            }
        }
    }
}

// Intersect one surface with the tangential ray and insert the result(s).
template <typename P, typename S, bool W>
DPROP_HD_LEAF void candidate_search(nav_state<S>& nav, const detector_view<S, W>& det,
                               uint32_t sf_idx, vec3<S> ro, vec3<S> rd,
                               const isect_cfg<S>& cfg) {
    ++nav.n_isect;
    candidate<S> is;
    bool found;
    if constexpr (!use_packed<S, W, P>()) {
        const dev_surface sf = det.surfaces[sf_idx];
        if (sf.shape == e_cylinder) {
            cylinder_candidates(nav, det, sf_idx, sf, ro, rd, cfg);
            return;
        }
        found = table_resolve<true>(is, det, sf_idx, sf, ro, rd, cfg,
                                    nav.external_tol);
    } else {
        const dev_nav_surface<S> ns = det.nav_surfaces[sf_idx];
        if (ns.shape() == e_cylinder) {
            cylinder_candidates(nav, det, sf_idx, det.surfaces[sf_idx], ro, rd,
                                cfg);
            return;
        }
        isect_point<S> ip;
        found = nav_intersect(ns, ro, rd, cfg.overstep_tol, ip) &&
                nav_resolve<true>(is, ip, sf_idx, ns, det, cfg,
                                  nav.external_tol);
    }
    if (found) {
        nav_insert(nav, is);
    }
}

// One surface per lane of a group (k_invalid: none): the lanes intersect
// theirs, then the candidates go into the cache in lane order, which is the
// order a single thread visits the surfaces in.
template <typename S, bool W, typename G>
DPROP_HD void group_search(nav_state<S>& nav, const detector_view<S, W>& det,
                           uint32_t sf_idx, vec3<S> ro, vec3<S> rd,
                           const isect_cfg<S>& cfg, const G& g) {
    candidate<S> is = invalid_candidate<S>();
    bool found = false, cylinder = false;
    if (sf_idx != k_invalid) {
        if constexpr (!use_packed<S, W, G>()) {
            const dev_surface sf = det.surfaces[sf_idx];
            cylinder = sf.shape == e_cylinder;
            found = !cylinder &&
                    table_resolve<true>(is, det, sf_idx, sf, ro, rd, cfg,
                                        nav.external_tol);
        } else {
            const dev_nav_surface<S> ns = det.nav_surfaces[sf_idx];
            cylinder = ns.shape() == e_cylinder;
            isect_point<S> ip;
            found = !cylinder &&
                    nav_intersect(ns, ro, rd, cfg.overstep_tol, ip) &&
                    nav_resolve<true>(is, ip, sf_idx, ns, det, cfg,
                                      nav.external_tol);
        }
    }
    nav.n_isect += g.count(sf_idx != k_invalid);
    const uint32_t cylinders = g.ballot(cylinder);
    for (uint32_t m = g.ballot(found) | cylinders; m != 0u; m &= m - 1u) {
        const int src = g.first(m);
        if ((cylinders >> src) & 1u) {
            const uint32_t idx = g.bcast(sf_idx, src);
            cylinder_candidates(nav, det, idx, det.surfaces[idx], ro, rd, cfg);
        } else {
            nav_insert(nav, g.bcast(is, src));
        }
    }
}

// ------------------------------------------------- intersection_update
template <typename P, typename S, bool W>
DPROP_HD_LEAF bool update_candidate(candidate<S>& c, const detector_view<S, W>& det,
                               vec3<S> ro, vec3<S> rd, const isect_cfg<S>& cfg,
                               S external_tol, uint32_t& n_isect) {
    if (c.sf == k_invalid) {
        return false;
    }
    ++n_isect;
    const uint32_t sf_idx = c.sf;
    auto cylinder = [&](const dev_surface& sf) {
        const dev_transform<S>& trf = det.transforms[sf.transform];
        isect_point<S> ips[2];
        intersect_cylinder(ro, rd, trf, det.masks[sf.mask_begin].v[0], ips);
        if (!ip_valid(ips[0].path) && !ip_valid(ips[1].path)) {
            return false;
        }
        for (uint32_t mi = sf.mask_begin; mi < sf.mask_begin + sf.n_masks;
             ++mi) {
            resolve_mask<W>(c, ips[0], sf_idx, sf, det.masks[mi], trf, cfg,
                            external_tol);
            if (c.is_probably_inside()) {
                return true;
            }
        }
        return false;
    };
    if constexpr (!use_packed<S, W, P>()) {
        const dev_surface sf = det.surfaces[sf_idx];
        if (sf.shape == e_cylinder) {
            return cylinder(sf);
        }
        return table_resolve<false>(c, det, sf_idx, sf, ro, rd, cfg,
                                    external_tol);
    } else {
        const dev_nav_surface<S> ns = det.nav_surfaces[sf_idx];
        if (ns.shape() == e_cylinder) {
            return cylinder(det.surfaces[sf_idx]);
        }
        isect_point<S> ip;
        return nav_intersect(ns, ro, rd, cfg.overstep_tol, ip) &&
               nav_resolve<false>(c, ip, sf_idx, ns, det, cfg, external_tol);
    }
}

// ------------------------------------------------------- update_status
template <typename S, typename NS>
DPROP_HD void update_status(NS& nav, const nav_cfg<S>& cfg) {
    if (!nav.cache_exhausted() &&
        fabs(nav.target().path) < cfg.isect.path_tol) {
        nav.status = nav.target().is_portal() ? e_on_portal : e_on_object;
        nav.reached();
    } else {
        nav.status = e_towards_object;
    }
    nav.trust = (nav.cache_exhausted() || nav.is_on_portal()) ? e_no_trust
                                                              : e_full_trust;
}

// ------------------------------------------------------- grid search
// Regular axis binning: int((v - min) / width + 1) - 1
template <typename S>
DPROP_HD int axis_bin(S v, S lo, S hi, uint32_t n) {
    const S width = (hi - lo) / static_cast<S>(n);
    const S u = (v - lo) / width + S(1);
    // out-of-range values (a failed reference-surface intersection) are
    // saturated instead of overflowing the integer conversion, far enough
    // from its limits for a search window either side of them
    int b;
    if (!(u == u)) {
        b = 0;
    } else if (u >= S(1073741824)) {
        b = 1073741824;
    } else if (u <= S(-1073741824)) {
        b = -1073741824;
    } else {
        b = static_cast<int>(u);
    }
    return b - 1;
}

// Closed axis: clamp the bin window, returns [lo, hi)
DPROP_HD void closed_range(int lbin, int ubin, int bins, int& lo,
                                  int& hi) {
    int mn = lbin > 0 ? lbin : 0;
    mn = mn >= bins ? bins - 1 : mn;
    int mx = ubin >= bins ? bins - 1 : ubin;
    mx = mx < 0 ? 0 : mx;
    lo = mn;
    hi = mx + 1;
}

DPROP_HD int wrap_bin(int b, int bins) {
    // within one turn (every window of a few bins): no division
    const int c = b < 0 ? b + bins : (b < bins ? b : b - bins);
    if (c >= 0 && c < bins) {
        return c;
    }
    return (bins + (b % bins)) % bins;
}

// Bin window of a grid around the track: axis 0 bins [lo0, hi0), axis 1 bins
// [lo1, hi1), the circular axis unwrapped.
struct bin_window {
    int lo0, hi0, lo1, hi1;
};

template <typename S, bool W>
DPROP_HD bin_window grid_window(const detector_view<S, W>& det,
                                const dev_grid<S>& g, const track_view<S>& trk,
                                const nav_cfg<S>& cfg) {
    // local position of the track on the grid's reference surface,
    // searched along the track direction (spatial_grid.hpp:100-140, 169-201)
    S p0, p1;
    if (g.kind == 1u) {
        const isect_point<S> ip = intersect_portal_cylinder(
            trk.pos, trk.dir, g.radius, -limits<S>::max());
        const vec3<S> at = trk.pos + ip.path * trk.dir;
        p0 = phi_of(at);
        p1 = ip.glob.z;
    } else {
        const dev_transform<S>& trf = det.transforms[g.transform];
        const isect_point<S> ip = intersect_plane(trk.pos, trk.dir, trf);
        const vec3<S> l = trf.point_to_local(ip.glob);
        p0 = perp(l);
        p1 = phi_of(l);
    }
    const int n0 = static_cast<int>(g.n0);
    const int n1 = static_cast<int>(g.n1);
    const int w0 = static_cast<int>(cfg.win0);
    const int w1 = static_cast<int>(cfg.win1);
    const int b0 = axis_bin(p0, g.min0, g.max0, g.n0);
    const int b1 = axis_bin(p1, g.min1, g.max1, g.n1);
    bin_window w;
    if (g.kind == 1u) {
        // axis 0: phi circular, axis 1: z closed
        w.lo0 = b0 - w0;
        w.hi0 = b0 + w1 + 1;
        closed_range(b1 - w0, b1 + w1, n1, w.lo1, w.hi1);
    } else {
        // axis 0: r closed, axis 1: phi circular
        closed_range(b0 - w0, b0 + w1, n0, w.lo0, w.hi0);
        w.lo1 = b1 - w0;
        w.hi1 = b1 + w1 + 1;
    }
    return w;
}

// Index into grid_bins of bin (i0, i1) of a window.
template <typename S>
DPROP_HD uint32_t window_bin(const dev_grid<S>& g, int i0, int i1) {
    const int j0 = (g.kind == 1u) ? wrap_bin(i0, static_cast<int>(g.n0)) : i0;
    const int j1 = (g.kind == 1u) ? i1 : wrap_bin(i1, static_cast<int>(g.n1));
    return g.bin_offset + static_cast<uint32_t>(j0) +
           static_cast<uint32_t>(j1) * g.n0;
}

// The surfaces of a volume in the order the reference visits them: the
// brute-force list (portals and passives), then the bins of the grid window,
// axis 0 outermost, each with its entries.  One thread's walk: next() returns
// the surfaces one by one and k_invalid at the end, so that the search has a
// single copy of the intersection code and a warp's lanes meet at it, each
// with a surface, instead of idling on empty bins.
template <typename S>
struct surface_walk {
    const uint32_t* list;  // the entries [e, end) come from it
    uint32_t e, end;
    int c, n_bins;         // next bin of the window, bins in it
    int i0, i1, lo1, hi1;

    template <bool W>
    DPROP_HD void start(const detector_view<S, W>& det, const dev_volume& vol,
                        const bin_window& w) {
        list = det.bf_surfaces;
        e = vol.bf_begin;
        end = vol.bf_end;
        c = 0;
        n_bins = (w.hi0 - w.lo0) * (w.hi1 - w.lo1);
        i0 = w.lo0;
        i1 = w.lo1;
        lo1 = w.lo1;
        hi1 = w.hi1;
    }
    template <bool W>
    DPROP_HD uint32_t next(const detector_view<S, W>& det,
                           const dev_grid<S>* g) {
        while (e >= end) {
            if (c >= n_bins) {
                return k_invalid;
            }
            const uint32_t b = window_bin(*g, i0, i1);
            ++c;
            if (++i1 == hi1) {
                i1 = lo1;
                ++i0;
            }
            const uint32_t v = det.grid_bins[b];
            if constexpr (W) {
                if (g->multi) {
                    list = det.grid_bins;
                    e = v;
                    end = det.grid_bins[b + 1u];
                    continue;
                }
            }
            if (v != k_invalid) {
                return v;
            }
        }
        return list[e++];
    }
};

// --------------------------------------------------- local_navigation
// overstep: the overstepping tolerance of the search
template <typename S, bool W, typename G = one_lane>
DPROP_HD_COLD void local_navigation(nav_state<S>& nav, const detector_view<S, W>& det,
                               const track_view<S>& trk, const nav_cfg<S>& cfg,
                               S overstep, const G& g = G{}) {
    const dev_volume vol = det.volumes[nav.volume];
    nav.clear_cache();
    isect_cfg<S> icfg = cfg.isect;
    icfg.overstep_tol = overstep;
    const vec3<S> ro = trk.pos;
    const vec3<S> rd = nav.direction * trk.dir;
    const bool has_grid = vol.grid != k_invalid;
    const dev_grid<S>* const grid = has_grid ? det.grids + vol.grid : nullptr;
    bin_window w{0, 0, 0, 0};  // no bins without a grid
    if (has_grid) {
        w = grid_window(det, *grid, trk, cfg);
    }
    if constexpr (G::lanes == 1) {
        surface_walk<S> walk;
        walk.start(det, vol, w);
        DPROP_ROLLED
        for (uint32_t sf = walk.next(det, grid); sf != k_invalid;
             sf = walk.next(det, grid)) {
            candidate_search<G>(nav, det, sf, ro, rd, icfg);
        }
    } else {
        // a group: one list entry per lane and pass, in the same order
        const int span = w.hi1 - w.lo1;
        const int n_bins = (w.hi0 - w.lo0) * span;
        auto bin_of = [&](int c) {
            const int row = c / span;
            return window_bin(*grid, w.lo0 + row, w.lo1 + (c - row * span));
        };
        if constexpr (W) {
            // lists: 0 the brute-force list, 1 + c the bins; a list per
            // lane, whose entries are then dealt out in a row
            for (int l0 = 0; l0 < 1 + n_bins; l0 += G::lanes) {
                const int l = l0 + g.rank;
                uint32_t e0 = 0u, e1 = 0u;
                if (l == 0) {
                    e0 = vol.bf_begin;
                    e1 = vol.bf_end;
                } else if (l <= n_bins) {
                    const uint32_t b = bin_of(l - 1);
                    const uint32_t v = det.grid_bins[b];
                    e0 = grid->multi ? v : b;
                    e1 = grid->multi ? det.grid_bins[b + 1u]
                                    : (v != k_invalid ? b + 1u : b);
                }
                // entry f of the pass: in the lane whose scanned counts
                // enclose f
                const uint32_t last = g.scan(e1 > e0 ? e1 - e0 : 0u);
                const uint32_t total = g.bcast(last, G::lanes - 1);
                for (uint32_t f0 = 0u; f0 < total;
                     f0 += static_cast<uint32_t>(G::lanes)) {
                    const uint32_t f = f0 + static_cast<uint32_t>(g.rank);
                    const int owner = g.owner(last, f);
                    const uint32_t entry =
                        g.bcast(e1, owner) - (g.bcast(last, owner) - f);
                    uint32_t sf = k_invalid;
                    if (f < total) {
                        sf = (l0 + owner == 0) ? det.bf_surfaces[entry]
                                               : det.grid_bins[entry];
                    }
                    group_search(nav, det, sf, ro, rd, icfg, g);
                }
            }
        } else {
            const int n_bf = static_cast<int>(vol.bf_end - vol.bf_begin);
            for (int k0 = 0; k0 < n_bf + n_bins; k0 += G::lanes) {
                const int k = k0 + g.rank;
                uint32_t sf = k_invalid;
                if (k < n_bf) {
                    sf = det.bf_surfaces[vol.bf_begin + static_cast<uint32_t>(k)];
                } else if (k < n_bf + n_bins) {
                    sf = det.grid_bins[bin_of(k - n_bf)];
                }
                group_search(nav, det, sf, ro, rd, icfg, g);
            }
        }
    }
    update_status(nav, cfg);
    if (nav.trust != e_full_trust) {
        if (nav.is_on_portal()) {
            nav.trust = (nav.current().volume_link == k_invalid_link)
                            ? e_full_trust
                            : e_no_trust;
        }
    }
    DPROP_NAV_TRACE(nav, "Init complete: ", trk.pos);
}

// ------------------------------------------- navigator init / update
template <typename S, bool W, typename G = one_lane>
DPROP_HD void navigator_init(nav_state<S>& nav, const detector_view<S, W>& det,
                             const track_view<S>& trk, const nav_cfg<S>& cfg,
                             const G& g = G{}) {
    local_navigation(nav, det, trk, cfg, -cfg.isect.path_tol, g);
}

// caching_navigator::update_impl, high-trust branch: re-intersect only the
// target.  Returns true if the update is complete (update_impl returned
// there); false if trust dropped to fair and the cache must be re-evaluated.
// A sensitive surface reached by the first pass is followed by a pass over
// the next candidate (one copy of the intersection code).
template <typename S, bool W, typename NS>
DPROP_HD bool high_trust_update(NS& nav, const detector_view<S, W>& det,
                                const track_view<S>& trk,
                                const nav_cfg<S>& cfg) {
    const vec3<S> ro = trk.pos;
    const vec3<S> rd = nav.direction * trk.dir;
    for (int pass = 0;; ++pass) {
        const bool hit = update_candidate<NS>(
            nav.target(), det, ro, rd, cfg.isect, nav.external_tol,
            nav.n_isect);
        if (pass == 1) {
            if (hit) {
                return true;
            }
            break;
        }
        if (!hit) {
            nav.status = e_nav_unknown;
            break;
        }
        update_status(nav, cfg);
        DPROP_NAV_TRACE(nav, "Update complete: high trust: ", trk.pos);
        if (nav.status == e_towards_object || nav.is_on_portal()) {
            return true;
        }
        if (nav.trust != e_full_trust) {
            break;
        }
    }
    nav.set_fair_trust();
    return false;
}

// caching_navigator::update_impl, fair-trust branch: re-evaluate the whole
// cache.
template <typename S, bool W, typename G = one_lane>
DPROP_HD_COLD void fair_trust_update(nav_state<S>& nav,
                                     const detector_view<S, W>& det,
                                     const track_view<S>& trk,
                                     const nav_cfg<S>& cfg,
                                     const G& g = G{}) {
    const vec3<S> ro = trk.pos;
    const vec3<S> rd = nav.direction * trk.dir;
    const int b = nav.begin_index();
    const int e = nav.end_index();
    if constexpr (G::lanes == 1) {
        for (int i = b; i < e; ++i) {
            if (!update_candidate<G>(nav.cand[i], det, ro, rd, cfg.isect,
                                  nav.external_tol, nav.n_isect)) {
                nav.cand[i].path = limits<S>::max();
            }
        }
    } else {
        // a candidate per lane (a group has at least k_cache lanes)
        static_assert(G::lanes >= k_cache, "a lane per candidate");
        candidate<S> c = invalid_candidate<S>();
        uint32_t looked = 0u;
        if (b + g.rank < e) {
            c = nav.cand[b + g.rank];
            if (!update_candidate<G>(c, det, ro, rd, cfg.isect, nav.external_tol,
                                  looked)) {
                c.path = limits<S>::max();
            }
        }
        nav.n_isect += g.count(looked != 0u);
        for (int i = b; i < e; ++i) {
            nav.cand[i] = g.bcast(c, i - b);
        }
    }
    // stable insertion sort of [b, e) by |path|
    DPROP_ROLLED
    for (int i = b + 1; i < e; ++i) {
        const candidate<S> key = nav.cand[i];
        const S ak = fabs(key.path);
        int j = i - 1;
        while (j >= b && fabs(nav.cand[j].path) > ak) {
            nav.cand[j + 1] = nav.cand[j];
            --j;
        }
        nav.cand[j + 1] = key;
    }
    nav.next = static_cast<int8_t>(b);
    // first unreachable candidate bounds the cache
    int inv = k_cache;
    DPROP_ROLLED
    for (int i = 0; i < k_cache; ++i) {
        if (nav.cand[i].path == limits<S>::max()) {
            inv = i;
            break;
        }
    }
    nav.last = static_cast<int8_t>(inv - 1);
    update_status(nav, cfg);
    DPROP_NAV_TRACE(nav, "Update complete: fair trust: ", trk.pos);
    if (nav.cache_exhausted()) {
        nav.set_no_trust();
    }
}

// The volume-level part of navigator_base::init and update (navigator_base.hpp:
// 56-154): up to three searches of a volume, one after the other.
//  -1  propagation start: the start volume, no overstepping; nothing follows
//   0  no trust left: the current volume again (caching_navigator::
//      update_impl)
//   1  on a portal: volume_switch (navigation_functions.hpp:264-288), with
//      the reference's default resolve_overstepping = true (:281)
//   2  still without full trust or a candidate: init_loose_cfg (:304-331)
// They share one copy of the search, which is most of the navigation's code:
// inlined once per call (four times with the start's), it overflowed the
// instruction cache of the kernels that run the whole loop.  Starts at stage
// `stage`; returns whether the volume was (re-)initialised.
template <typename S, bool W, typename G = one_lane>
DPROP_HD_COLD bool volume_update(nav_state<S>& nav,
                                 const detector_view<S, W>& det,
                                 const track_view<S>& trk,
                                 const nav_cfg<S>& cfg, int stage,
                                 const G& g = G{}) {
    bool is_init = false;
    for (; stage < 3; ++stage) {
        S overstep = cfg.isect.overstep_tol;
        if (stage == -1) {
            overstep = -cfg.isect.path_tol;
        } else if (stage == 1) {
            if (!nav.is_on_portal()) {
                continue;
            }
            if (nav.current().volume_link == k_invalid_link) {
                nav.status = e_nav_exit;
                return false;
            }
            nav.set_volume(nav.current().volume_link);
        } else if (stage == 2) {
            if (nav.trust == e_full_trust && !nav.cache_exhausted()) {
                break;
            }
            const S a = S(100) * cfg.isect.overstep_tol;
            const S b = S(-10) * cfg.isect.max_mask_tol;
            overstep = a < b ? a : b;
        }
        local_navigation(nav, det, trk, cfg, overstep, g);
        is_init = true;
        if (stage == -1) {
            break;
        }
        if (stage == 1) {
            nav.trust = e_full_trust;
        } else if (stage == 2 &&
                   (nav.trust != e_full_trust || nav.cache_exhausted())) {
            nav.abort(e_reason_no_surface);
        }
    }
    return is_init;
}

// navigator_base::update after the high-trust branch: fair- and no-trust
// branches unless that branch was complete; returns the stage volume_update
// continues with.
template <typename S, bool W, typename G = one_lane>
DPROP_HD int update_without_high_trust(nav_state<S>& nav,
                                       const detector_view<S, W>& det,
                                       const track_view<S>& trk,
                                       const nav_cfg<S>& cfg, bool complete,
                                       const G& g = G{}) {
    if (!complete && nav.trust == e_fair_trust && !nav.cache_exhausted()) {
        fair_trust_update(nav, det, trk, cfg, g);
    }
    return (!complete && nav.trust == e_no_trust) ? 0 : 1;
}

// navigator_base::init (first) and update
template <typename S, bool W, typename G = one_lane>
DPROP_HD bool navigator_update(nav_state<S>& nav, const detector_view<S, W>& det,
                               const track_view<S>& trk, const nav_cfg<S>& cfg,
                               bool first, const G& g = G{}) {
    int stage = -1;
    if (!first) {
        if (nav.trust == e_full_trust) {
            return false;
        }
        const bool complete =
            nav.trust == e_high_trust && high_trust_update(nav, det, trk, cfg);
        stage = update_without_high_trust(nav, det, trk, cfg, complete, g);
    }
    return volume_update(nav, det, trk, cfg, stage, g);
}

}  // namespace dprop
