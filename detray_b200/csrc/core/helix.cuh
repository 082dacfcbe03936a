// Helix "truth" intersections: the exact helical trajectory of a track in a
// constant field intersected with every surface of the detector by
// Newton-Raphson root finding - the reference's navigation-validation
// scanner, run on the GPU.
//
// Reference:
//   helix trajectory     core/include/detray/tracks/helix.hpp:32-180
//   root finding         core/include/detray/utils/root_finding.hpp:38-360
//                        (expand_bracket, newton_raphson_safe: Newton steps
//                        safeguarded by bisection, Numerical Recipes rtsafe)
//   helix intersectors   navigation/intersection/helix_plane_intersector.hpp
//                        :62-118, helix_cylinder_intersector.hpp:65-170,
//                        helix_line_intersector.hpp:48-150
//   mask resolution      root_finding.hpp:374-430 (resolve_mask for helix
//                        intersection points)
//   scan                 tests/include/detray/test/validation/
//                        detector_scanner.hpp:52-140 (brute_force_scan over
//                        all surfaces, kept if along the track, sorted by
//                        |path|, cut after the first world exit)
#pragma once

#include "actors.cuh"

namespace dprop {

template <typename S>
struct helix {
    vec3<S> pos0;
    vec3<S> t0;   // unit direction at s = 0
    vec3<S> h0;   // unit field direction
    vec3<S> n0;   // unit h0 x t0
    S qop;
    S B;          // field magnitude
    S alpha;      // |h0 x t0|
    S delta;      // h0 . t0
    S K;          // -q/p * B
    bool straight;  // no transverse momentum: moves along the field axis

    DPROP_HD void init(vec3<S> p, vec3<S> dir, S q_over_p, vec3<S> bfield) {
        pos0 = p;
        t0 = dir;
        qop = q_over_p;
        B = norm(bfield);
        h0 = (S(1) / B) * bfield;
        const vec3<S> hxt = cross(h0, t0);
        alpha = norm(hxt);
        n0 = (S(1) / alpha) * hxt;
        delta = dot(h0, t0);
        K = -qop * B;
        const vec3<S> mom = (S(1) / fabs(qop)) * t0;
        const S pz = dot(mom, h0);
        const vec3<S> pt = mom - pz * h0;
        straight = norm(pt) < S(1e-6);
    }
    DPROP_HD vec3<S> pos(S s) const {
        if (straight) {
            return pos0 + s * h0;
        }
        const S ks = K * s;
        const sin_cos<S> sc = sincos_(ks);
        const S sn = sc.s;
        const S cs = sc.c;
        vec3<S> r = pos0;
        r = r + (delta / K * (ks - sn)) * h0;
        r = r + (sn / K) * t0;
        r = r + (alpha / K * (S(1) - cs)) * n0;
        return r;
    }
    DPROP_HD vec3<S> dir(S s) const {
        if (straight) {
            return t0;
        }
        const sin_cos<S> sc = sincos_(K * s);
        const S cs = sc.c;
        vec3<S> d{S(0), S(0), S(0)};
        d = d + (delta * (S(1) - cs)) * h0;
        d = d + cs * t0;
        d = d + (alpha * sc.s) * n0;
        return normalize(d);
    }
    // position and direction at s from one sine/cosine pair (the same
    // values as pos(s) and dir(s))
    DPROP_HD void eval(S s, vec3<S>& p, vec3<S>& d) const {
        if (straight) {
            p = pos0 + s * h0;
            d = t0;
            return;
        }
        const S ks = K * s;
        const sin_cos<S> sc = sincos_(ks);
        const S sn = sc.s;
        const S cs = sc.c;
        vec3<S> r = pos0;
        r = r + (delta / K * (ks - sn)) * h0;
        r = r + (sn / K) * t0;
        r = r + (alpha / K * (S(1) - cs)) * n0;
        p = r;
        vec3<S> v{S(0), S(0), S(0)};
        v = v + (delta * (S(1) - cs)) * h0;
        v = v + cs * t0;
        v = v + (alpha * sn) * n0;
        d = normalize(v);
    }
    DPROP_HD vec3<S> b_field() const { return B * h0; }
};

// Result of a root search: path to the root and the last step length;
// limits::max() for both when there is no root.
template <typename S>
struct root_result {
    S s;
    S ds;
};

template <typename S>
struct root_cfg {
    S tol;             // convergence: |f| or |step| below 1 um
    uint32_t max_tries;
    S max_path;        // 5 m search range
};

// Safeguarded Newton-Raphson on f(s) = 0 from the guess s: widen a bracket
// around s (towards the side with the smaller |f|) until f changes sign -
// given up after 1000 widenings or on non-finite values -, then take Newton
// steps, falling back to bisection when a step would leave the bracket or
// converge slower than bisecting.  fdf(x, f, df) evaluates the function and
// its derivative.
//
// Every evaluation is made at one place, by a loop that goes on with what the
// search needs next: inlined at each of the search's eight call sites, the
// evaluation overflowed the instruction cache, and the lanes of a warp, each
// somewhere else in its search, could not evaluate together.
template <typename S, typename FDF>
DPROP_HD root_result<S> newton_safe(const FDF& fdf, S s,
                                    const root_cfg<S>& cfg) {
    const S inv = limits<S>::max();
    const S eps = limits<S>::epsilon();
    const root_result<S> none{inv, inv};
    if (!(fabs(s) < inv)) {
        return none;
    }
    // initial bracket around s (the factors are single-precision constants
    // in every build, as in the reference)
    S a = (fabs(s) == S(0)) ? S(-0.2f) : S(0.8f) * s;
    S b = (fabs(s) == S(0)) ? S(0.2f) : S(1.2f) * s;
    S lo = a > b ? b : a;
    S hi = a > b ? a : b;
    S flo = S(0), fhi = S(0), s_prev = S(0);
    uint32_t n = 0u;
    bool bracketed = false;
    // what the evaluated point is: the bracket's ends, an end after a
    // widening, the start of the Newton steps, a step
    enum { k_first, k_second, k_low, k_high, k_start, k_step };
    int at = k_first;
    S x = lo;
    while (true) {
        S fx, dfx;
        fdf(x, fx, dfx);
        if (at <= k_high) {
            if (at == k_first || at == k_low) {
                flo = fx;
            } else {
                fhi = fx;
            }
            if (at == k_first) {
                x = hi;
                at = k_second;
                continue;
            }
            const bool broken = n == 1000u || !isfinite(flo) ||
                                !isfinite(fhi) || !isfinite(lo) ||
                                !isfinite(hi);
            if (!signbit(flo * fhi) && !broken) {
                const S w = hi - lo;
                if (fabs(flo) < fabs(fhi)) {
                    lo -= w;
                    x = lo;
                    at = k_low;
                } else {
                    hi += w;
                    x = hi;
                    at = k_high;
                }
                ++n;
                continue;
            }
            if (!broken) {
                bracketed = true;
                s = S(0.5) * (hi + lo);
                if (fabs(lo) >= inv || fabs(hi) >= inv) {
                    return none;
                }
                if (fabs(s) > cfg.max_path && fabs(lo) >= cfg.max_path &&
                    fabs(hi) >= cfg.max_path) {
                    return none;
                }
                // (the initial bracket ends are returned, as the reference
                // does)
                if (fabs(flo) < cfg.tol) {
                    return {a, eps};
                }
                if (fabs(fhi) < cfg.tol) {
                    return {b, eps};
                }
                // a: the end with the negative function value
                const bool lower_neg = signbit(flo);
                a = lower_neg ? lo : hi;
                b = lower_neg ? hi : lo;
            }
            x = s;
            at = k_start;
            continue;
        }
        if (at == k_start) {
            if (fabs(fx) < cfg.tol) {
                return {s, eps};
            }
            if (signbit(fx)) {
                a = s;
            } else {
                b = s;
            }
            n = 0u;
        } else {
            if (bracketed && signbit(fx)) {
                a = s;
            } else {
                b = s;
            }
            if (fabs(s) > cfg.max_path && fabs(s_prev) > cfg.max_path &&
                ((a < -cfg.max_path && b < -cfg.max_path) ||
                 (a > cfg.max_path && b > cfg.max_path))) {
                return none;
            }
            ++n;
            if (n >= cfg.max_tries) {
                return none;
            }
        }
        if (!(fabs(s - s_prev) > cfg.tol)) {
            return {s, fabs(s - s_prev)};
        }
        bool escapes = true;
        S s_newton = S(0);
        if (fabs(dfx) != S(0)) {
            s_newton = s - fx / dfx;
            escapes = signbit((s_newton - a) * (b - s_newton));
        }
        bool slow = true;
        const S ds_bisect = S(0.5) * (a + b) - s;
        if (bracketed && fabs(ds_bisect) < S(10) * S(unit::mm)) {
            slow = S(2) * fabs(fx) > fabs(dfx * ds_bisect + fx);
        }
        s_prev = s;
        if (bracketed && (escapes || slow || fabs(dfx) == S(0))) {
            s = S(0.5) * (a + b);
        } else {
            if (!bracketed && fabs(dfx) == S(0)) {
                return none;
            }
            s = s_newton;
        }
        x = s;
        at = k_step;
    }
}

// ------------------------------------------------------------ intersectors
// The function whose root is a helix's intersection with a surface:
//   plane (rectangle, trapezoid, ring)  f(s) = n . (h(s) - c)
//   cylinder of radius r around z       f(s) = |(h(s) - c) x z|^2 - r^2
//   line (wire along z)                 f(s) = t(s) . w(s), w the vector from
//                                       the closest wire point to the helix
// axis: n or z; centre: c.
template <typename S>
struct helix_function {
    enum kind_t { k_plane, k_cylinder, k_line };
    const helix<S>& h;
    kind_t kind;
    vec3<S> axis, centre;
    S r;

    DPROP_HD void operator()(S x, S& f, S& df) const {
        vec3<S> p, d;
        h.eval(x, p, d);
        if (kind == k_plane) {
            f = dot(axis, p - centre);
            df = dot(axis, d);
        } else if (kind == k_cylinder) {
            const vec3<S> crp = cross(p - centre, axis);
            f = dot(crp, crp) - r * r;
            df = S(2) * dot(crp, cross(d, axis));
        } else {
            const S A = dot(p - centre, axis);
            const vec3<S> w = p - (centre + A * axis);
            f = dot(d, w);
            const vec3<S> dtds = h.qop * cross(d, h.b_field());
            const vec3<S> dwds = d - dot(d, axis) * axis;
            df = dot(dtds, w) + dot(d, dwds);
        }
    }
};

// Starting guesses of the root search (at most two); none for a line almost
// parallel to the track.
template <typename S>
DPROP_HD int helix_guesses(const helix_function<S>& fn,
                           const dev_transform<S>& trf, S guess[2]) {
    const helix<S>& h = fn.h;
    if (fn.kind == helix_function<S>::k_plane) {
        const vec3<S> dist = fn.centre - h.pos0;
        const S denom = dot(fn.axis, h.dir(S(0.5) * norm(dist)));
        guess[0] =
            (denom == S(0)) ? norm(dist) : dot(fn.axis, dist) / denom;
        return 1;
    }
    if (fn.kind == helix_function<S>::k_cylinder) {
        // the ray intersections along the direction at half the radius
        const vec3<S> hd = h.dir(S(0.5) * fn.r);
        isect_point<S> ips[2];
        const int n_sol = intersect_cylinder(h.pos0, hd, trf, fn.r, ips);
        if (n_sol == 0) {
            guess[0] = fn.r;
            guess[1] = -fn.r;
            return 2;
        }
        guess[0] = ips[0].path;
        guess[1] = ips[1].path;
        return n_sol;
    }
    const vec3<S> t0 = h.dir(S(0));
    const vec3<S> r0 = h.pos(S(0));
    const S lt0 = dot(fn.axis, t0);
    const S denom = S(1) - lt0 * lt0;
    if (denom < S(1e-5)) {
        return 0;
    }
    const vec3<S> D = fn.centre - r0;
    const S P = dot(D, fn.axis);
    const S Q = dot(D, t0);
    guess[0] = S(1) / denom * (Q - P * lt0);
    return 1;
}

// One scanned intersection
template <typename S>
struct scan_hit {
    S path;
    S loc0, loc1;
    uint32_t sf;
    uint16_t volume_link;
};

// Mask check of a helix intersection (resolve_mask for helix points):
// inside with the given tolerance, 0 on portals.
template <bool W, typename S>
DPROP_HD bool helix_inside(const dev_surface& sf, const dev_mask<S>& m,
                           const dev_transform<S>& trf, vec3<S> glob,
                           S mask_tol) {
    const S tol = (sf.kind == e_portal) ? S(0) : mask_tol;
    const vec3<S> l = trf.point_to_local(glob);
    switch (sf.shape) {
        case e_rectangle:
            return check_rectangle(m, l.x, l.y, tol, S(0)).inside;
        case e_trapezoid:
            return check_trapezoid(m, l.x, l.y, tol, S(0)).inside;
        case e_ring:
            return check_ring(m, perp(l), tol).inside;
        case e_line:
            if (W) {
                return check_line(m, l, tol, S(0)).inside;
            }
            return false;
        case e_cylinder:
        case e_concentric_cylinder:
        default:
            return check_cylinder_z(m, l.z, tol, S(0)).inside;
    }
}

// The intersections of the helix with one surface that are inside a mask
// and along the track (intersection_initialize for a helix: per mask, the
// solutions that pass it; a single-solution surface stops at the first mask
// that accepts it, a cylinder when a mask accepted both).  emit(hit) is
// called for each; the local coordinates are the surface's bound local
// coordinates at the point.
template <bool W, typename S, typename Emit>
DPROP_HD void helix_surface_hits(const detector_view<S, W>& det,
                                 uint32_t sf_idx, const helix<S>& h,
                                 S mask_tol, const root_cfg<S>& cfg,
                                 Emit&& emit) {
    const dev_surface sf = det.surfaces[sf_idx];
    const dev_transform<S>& trf = det.transforms[sf.transform];
    using fn_t = helix_function<S>;
    if (!W && sf.shape == e_line) {
        return;
    }
    const bool portal = sf.shape == e_concentric_cylinder;
    const bool cylinder = portal || sf.shape == e_cylinder;
    const fn_t fn{h,
                  cylinder ? fn_t::k_cylinder
                           : ((W && sf.shape == e_line) ? fn_t::k_line
                                                        : fn_t::k_plane),
                  trf.z(), trf.translation(),
                  cylinder ? det.masks[sf.mask_begin].v[0] : S(0)};
    const S no_root = limits<S>::max();
    root_result<S> res[2] = {{no_root, no_root}, {no_root, no_root}};
    S guess[2];
    const int n_runs = helix_guesses(fn, trf, guess);
    for (int i = 0; i < n_runs; ++i) {
        const root_result<S> root = newton_safe(fn, guess[i], cfg);
        if (portal) {
            // one solution: the first, or the second if that lies behind
            res[0] = root;
            if (!signbit(root.s)) {
                break;
            }
            if (n_runs == 1) {
                res[0] = {no_root, no_root};
            }
        } else {
            res[i] = root;
        }
    }
    const int n_res = sf.shape == e_cylinder ? 2 : 1;
    // an intersection point is valid within 10 m
    bool any = false;
    for (int i = 0; i < n_res; ++i) {
        any = any || fabs(res[i].s) < S(10000) * S(unit::mm);
    }
    if (!any) {
        return;
    }
    const S inv = limits<S>::max();
    for (uint32_t mi = sf.mask_begin; mi < sf.mask_begin + sf.n_masks; ++mi) {
        const dev_mask<S> m = det.masks[mi];
        int n_found = 0;
        for (int i = 0; i < n_res; ++i) {
            const S s = res[i].s;
            if (s == inv || s == -inv) {
                continue;  // no root
            }
            const vec3<S> p = h.pos(s);
            if (!helix_inside<W>(sf, m, trf, p, mask_tol)) {
                continue;
            }
            ++n_found;
            if (!signbit(s)) {  // along the track
                const vec3<S> d = h.dir(s);
                S l0, l1;
                if (W && sf.shape == e_line) {
                    const local2<S> l = line_bound_local(trf, p, d);
                    l0 = l.l0;
                    l1 = l.l1;
                } else {
                    global_to_bound_local(sf.shape, trf, p, l0, l1);
                }
                emit(scan_hit<S>{s, l0, l1, sf_idx,
                                 static_cast<uint16_t>(m.volume_link)});
            }
            if (n_found == n_res) {
                return;
            }
        }
    }
}

// ------------------------------------------------------------------ culling
// A track's helix in single precision, for the bounding test of the scan.
struct scan_probe {
    vec3<float> pos;
    vec3<float> t;  // unit direction
    vec3<float> h;  // unit field direction
    vec3<float> n;  // h x t (length alpha)
    float K;
    float K_inv;
    float alpha;
    float delta;
    float slack;  // mm: rounding of single-precision helix points

    template <typename S>
    DPROP_HD void init(const helix<S>& hx) {
        auto f3 = [](vec3<S> v) {
            return vec3<float>{static_cast<float>(v.x),
                               static_cast<float>(v.y),
                               static_cast<float>(v.z)};
        };
        pos = f3(hx.pos0);
        t = f3(hx.t0);
        h = f3(hx.h0);
        n = cross(h, t);
        K = static_cast<float>(hx.K);
        K_inv = 1.f / K;
        alpha = norm(n);
        delta = dot(h, t);
        // sine and cosine are good to 1e-6 here, 1/K converts them to mm; for
        // a helix of no curvature, or one that moves along the field axis
        // (helix::straight), every sphere is near.  The test of a plane along
        // the field holds for it as well: a track along the axis keeps its
        // distance to the plane, and without curvature the terms are not
        // numbers.
        slack = hx.straight ? limits<float>::max()
                            : 1.f + 4e-6f * fabs(K_inv);
    }
    DPROP_HD static void sincos_of(float x, float& sn, float& cs) {
#if defined(__CUDA_ARCH__)
        if (fabs(x) < 3.f) {
            sn = __sinf(x);
            cs = __cosf(x);
            return;
        }
#endif
        const sin_cos<float> r = sincos_(x);
        sn = r.s;
        cs = r.c;
    }
    // position at s relative to the start, without its component along h
    DPROP_HD vec3<float> transverse(float s) const {
        float sn, cs;
        sincos_of(K * s, sn, cs);
        return (sn * K_inv) * (t - delta * h) + ((1.f - cs) * K_inv) * n;
    }
    DPROP_HD vec3<float> offset(float s) const {
        return transverse(s) + (delta * s) * h;
    }
    DPROP_HD vec3<float> dir(float s) const {
        float sn, cs;
        sincos_of(K * s, sn, cs);
        return (delta * (1.f - cs)) * h + cs * t + sn * n;
    }
};

// Whether helix_surface_hits can emit a hit on a surface with bound b: false
// only where it cannot.  A hit is a point of the helix at s >= 0 that a mask
// accepts, and the root search returns one of
//   - a point on the surface (to the search's 1 um, or 0.2 mm around s = 0):
//     then it lies within the bounding sphere;
//   - an end of the initial bracket, 0.8 or 1.2 times the starting guess g,
//     when an end of the widened bracket is a root (newton_safe returns the
//     initial end there, as the reference does);
//   - s = 0, when the widened bracket is centred there.
// The last two need not lie on the surface, and the mask is checked in the
// surface's plane only.
//   - A plane along the field that the helix's circle around the field axis
//     does not reach has no root and no bracket, so none of the three arises
//     (the search would widen and step to its limits there, 2 000 helix
//     evaluations).
//   - The sphere is tested against the circle, and against the point where
//     the helix passes the sphere's height along the axis.
// Away from the sphere:
//   - with a sign change between 0.8 g and 1.2 g nothing is widened;
//   - otherwise the bracket's ends are tested against the sphere's shadow
//     along the normal, and so is the start, if the bracket can become
//     centred on it: each widening doubles the bracket at the end with the
//     smaller function value, and [-X, X] comes only from [0.8 g, 1.6 g] and
//     then [0, 1.6 g], with no sign change up to there.
// Comparisons are written so that a value that is not a number keeps the
// surface.
DPROP_HD bool scan_may_hit(const scan_bound& b, const scan_probe& p,
                           float mask_tol) {
    if (!(b.radius >= 0.f)) {
        return true;
    }
    const vec3<float> w{b.cx - p.pos.x, b.cy - p.pos.y, b.cz - p.pos.z};
    const vec3<float> nrm{b.nx, b.ny, b.nz};
    // n . (p(s) - c) = circle part + height part; the circle's centre is at
    // n / K from the start
    const float f0 = -dot(nrm, w);
    if (dot(nrm, p.h) == 0.f) {
        const float centre = f0 + p.K_inv * dot(nrm, p.n);
        const float circle = p.alpha * fabs(p.K_inv);
        // single-precision rounding of the three terms here and of the
        // search's own function values is below 1e-6 of 1/K and of the
        // coordinates
        if (fabs(centre) - circle >
            0.05f + 2e-6f * fabs(p.K_inv) + 4e-6f * fabs(f0)) {
            return false;
        }
    }
    const float dist = norm(w);
    const float r =
        1.001f * (b.radius + b.grow * mask_tol) + p.slack + 4e-6f * dist;
    const float wz = dot(w, p.h);
    const vec3<float> wt = w - wz * p.h;
    // (distance to the axis)^2 - (circle radius)^2, times |K|
    const float aK = fabs(p.K);
    const float side = 2.f * dot(wt, p.n);
    const float off = fabs(aK * dot(wt, wt) - (p.K < 0.f ? -side : side));
    bool near = !(off > r * (2.f * p.alpha + r * aK));
    // the sphere's height is reached at s >= 0
    near = near && !(fabs(wz) > r && wz * p.delta <= 0.f);
    const float ad = fabs(p.delta);
    if (near && ad > 1e-3f) {
        const float reach = r + p.alpha * r / ad;
        const vec3<float> e = wt - p.transverse(wz / p.delta);
        near = !(dot(e, e) > reach * reach);
    }
    if (near) {
        return true;
    }
    // the search's starting guess (helix_plane)
    const float denom = dot(nrm, p.dir(0.5f * dist));
    if (!(fabs(denom) > 1e-3f)) {
        return true;
    }
    const float s = -f0 / denom;
    if (!(fabs(s) > 1.f)) {
        return true;
    }
    const vec3<float> qa = p.offset(0.8f * s) - w;
    const vec3<float> qb = p.offset(1.2f * s) - w;
    const float fa = dot(nrm, qa);
    const float fb = dot(nrm, qb);
    // rounding of the guess moves the points by this much
    const float blur =
        p.slack + (1e-5f * fabs(s) + 1e-6f * dist) / fabs(denom);
    if (fabs(fa) > blur && fabs(fb) > blur && ((fa < 0.f) != (fb < 0.f))) {
        return false;
    }
    const float shadow = (r + blur) * (r + blur);
    if (!(dot(qa, qa) - fa * fa > shadow) ||
        !(dot(qb, qb) - fb * fb > shadow)) {
        return true;
    }
    if (dot(w, w) - f0 * f0 > shadow) {
        return false;
    }
    const float fc = dot(nrm, p.offset(1.6f * s) - w);
    const bool centred = !(fabs(fb) > fabs(fa) + 2.f * blur) &&
                         !(fabs(fa) > fabs(fc) + 2.f * blur);
    return centred;
}

// --------------------------------------------------- navigation validation
// Compare the surfaces a propagation reached (its records with
// record_all_surfaces, in path order) with the helix truth of the same track
// (navigation validation, tests/include/detray/test/validation/
// navigation_validation_utils.hpp:379-800: holes and extra surfaces).
//   - a sensitive or passive truth surface is reached if a record of the
//     same surface lies within path_tol of its path;
//   - adjacent volumes share a boundary through two coinciding portals, of
//     which the navigator records the one it continues in: a truth portal is
//     reached if any portal record lies within path_tol, and the final
//     world-exit portal if the propagation ended by leaving the world;
//   - a record is extra if no truth surface matches it the same way.
// Ti / Tr: path types of the truth and of the records.
template <typename Ti, typename Tr>
DPROP_HD void compare_trace(const uint64_t* truth_bc, const Ti* truth_path,
                            const uint16_t* truth_vlink, uint32_t n_truth,
                            const uint64_t* rec_bc, const Tr* rec_path,
                            uint32_t n_rec, bool exited, uint64_t stride,
                            uint64_t t, double path_tol, uint32_t& missed,
                            uint32_t& extra) {
    auto is_portal = [](uint64_t bc) { return ((bc >> 48) & 0xfu) == 0u; };
    missed = 0u;
    extra = 0u;
    for (uint32_t i = 0; i < n_truth; ++i) {
        const uint64_t o = static_cast<uint64_t>(i) * stride + t;
        const uint64_t bc = truth_bc[o];
        const double p = static_cast<double>(truth_path[o]);
        bool found = false;
        if (is_portal(bc) && truth_vlink[o] == k_invalid_link && exited) {
            found = true;
        }
        for (uint32_t j = 0; j < n_rec && !found; ++j) {
            const uint64_t q = static_cast<uint64_t>(j) * stride + t;
            const bool same = is_portal(bc) ? is_portal(rec_bc[q])
                                            : rec_bc[q] == bc;
            found = same &&
                    fabs(static_cast<double>(rec_path[q]) - p) <= path_tol;
        }
        missed += found ? 0u : 1u;
    }
    for (uint32_t j = 0; j < n_rec; ++j) {
        const uint64_t q = static_cast<uint64_t>(j) * stride + t;
        const uint64_t bc = rec_bc[q];
        const double p = static_cast<double>(rec_path[q]);
        bool found = false;
        for (uint32_t i = 0; i < n_truth && !found; ++i) {
            const uint64_t o = static_cast<uint64_t>(i) * stride + t;
            const bool same = is_portal(bc) ? is_portal(truth_bc[o])
                                            : truth_bc[o] == bc;
            found = same && fabs(static_cast<double>(truth_path[o]) - p) <=
                                path_tol;
        }
        extra += found ? 0u : 1u;
    }
}

}  // namespace dprop
