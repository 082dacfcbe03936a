// Which form a call takes that leaves its launch shape open: the properties of
// a detector the rules look at, and the batch sizes where one form becomes
// the faster one.  Every line holds both sides as measured (B200, 148 SMs,
// microseconds, device time).
#pragma once

#include <cstdint>

#include "detray_b200/dprop.h"

namespace dprop {

// What of a detector decides the form: not whether its kernels carry the code
// for lines, rods, material maps and volume material (that is one flag for all
// of them), but what a track spends its time on.
struct launch_traits {
    bool lines{false};          // line surfaces or several surfaces per bin:
                                // long tracks, many candidates a volume
    bool surface_grids{false};  // volumes find their surfaces in grids
    bool long_lists{false};     // more than 32 surfaces in a volume's
                                // brute-force list
    bool extra_code{false};     // kernels with the code of all options (a
                                // lone warp waits longer for instructions)
};

inline launch_traits launch_traits_of(const dprop_detector_desc* d,
                                      bool extra_code) {
    launch_traits t;
    t.extra_code = extra_code;
    for (uint32_t i = 0; i < d->n_surfaces; ++i) {
        t.lines = t.lines || d->surfaces[i].shape == DPROP_SHAPE_LINE;
    }
    for (uint32_t i = 0; i < d->n_volumes; ++i) {
        t.long_lists = t.long_lists ||
                       d->volumes[i].bf_end - d->volumes[i].bf_begin > 32u;
        const uint32_t g = d->volumes[i].grid;
        if (g != DPROP_INVALID_INDEX) {
            t.surface_grids = true;
            t.lines = t.lines || d->grids[g].multi != 0u;
        }
    }
    return t;
}

// Bins of a grid that a search looks at, with the configuration's window.
inline uint64_t window_bins(const uint32_t window[2]) {
    const uint64_t side = uint64_t(window[0]) + window[1] + 1u;
    return side * side;
}

// Whether a search of that window is a small part of a track: the lanes of a
// warp have little to share, and more warps per SM little to hide.
inline bool narrow_search(const launch_traits& t, const uint32_t window[2]) {
    return t.surface_grids &&
           window_bins(window) < (t.extra_code ? 16u : 9u);
}

// Tracks up to which a warp per track is the faster form, fp32.  The lanes of a
// warp share only the searches, so beyond a full GPU one thread per track
// wins; how far beyond depends on how much of a track is search.  Warp per
// track / thread per track in input order / sorted:
//   toy 5 000: 1 025 / 1 882 / 1 356, 8 000: 1 566 / 1 910 / 1 381; in the map
//   5 000: 1 218 / 1 956 / 1 418
//   toy with material maps 4 000: 1 658 / 2 002 / 1 575, 5 000: 1 979 / 2 035 /
//   1 616, 10 000: 3 954 / 2 017 / 1 566
//   wire chamber, pT from 0.5 GeV, |eta| < 1, 5 000: 1 939 / 2 361 / 2 517,
//   8 000: 2 814 / 2 399 / 2 511; pT from 0.1 GeV, |eta| < 3, 8 000: 4 134 /
//   7 577 / 10 225
//   telescope (no grid, 11 surfaces) 2 300: 215 / 249 / 307, 3 000: 340 / 248 /
//   308; with volume material 1 400: 305 / 322 / 384, 1 800: 328 / 316 / 389,
//   10 000: 1 669 / 347 / 430
// all with windows of 3 bins either side.  With a window of one bin, half the
// limit, a warp / a thread per track:
//   toy 4 000: 588 / 581, 6 000: 874 / 581; with material maps 2 000: 778 / 757,
//   4 000: 1 198 / 757 (3 x 3 bins 2 000: 994 / 1 197); wire chamber in the map
//   5 000: 1 928 / 1 775, 8 000: 2 906 / 1 983
inline uint64_t group_limit(const launch_traits& t) {
    if (t.lines) {
        return 8192u;
    }
    if (t.surface_grids) {
        return t.extra_code ? 4096u : 6144u;
    }
    return t.extra_code ? 1536u : 2368u;
}
inline uint64_t group_limit(const launch_traits& t, const uint32_t window[2]) {
    return group_limit(t) / (narrow_search(t, window) ? 2u : 1u);
}

// The same in the adjoint propagation.  It pays for fewer tracks there: the
// Jacobians, which the lanes repeat, are a larger part of a track.  Warp per
// track / thread per track / sorted, with the field gradient:
//   toy in the map 1 400: 1 434 / 2 187 / 1 696, 1 800: 1 480 / 2 151 / 1 641;
//   with material maps 1 000: 1 648 / 2 409 / 1 927, 1 400: 2 289 / 2 455 /
//   1 940; wire chamber 2 300: 2 891 / 3 028 / 3 050, 3 000: 4 060 / 3 107 /
//   3 102; telescope 700: 492 / 519 / 572, 1 400: 655 / 525 / 584
// and without it:
//   toy 4 000: 1 368 / 2 067 / 1 585, 5 000: 1 659 / 2 125 / 1 585; with
//   material maps 2 300: 1 491 / 2 403 / 1 835, 3 000: 2 051 / 2 425 / 1 774;
//   wire chamber 5 000: 3 100 / 2 799 / 2 962 (pT from 0.1 GeV 3 843 / 8 274 /
//   8 223); telescope 1 400: 345 / 384 / 455, 3 000: 537 / 396 / 472
// The window matters to the form without the field gradient alone (one bin:
// toy 2 700: 716 / 780, 4 000: 961 / 780; with it the searches are a small part
// anyway), and a window of 3 x 3 bins only where there are lines (wire chamber
// in the map 5 400: 3 664 / 3 258).
inline uint64_t group_limit_adjoint(const launch_traits& t,
                                    const uint32_t window[2],
                                    bool field_gradient) {
    if (field_gradient) {
        return group_limit(t) / 4u;
    }
    const bool narrow = t.surface_grids &&
                        window_bins(window) < (t.lines ? 16u : 9u);
    return 2u * group_limit(t) / (narrow ? 6u : 3u);
}

// The same in double precision.  Warp per track / thread per track / sorted:
// toy 3 000: 1 255 / 1 763 / 1 307, 4 000: 1 575 / 1 729 / 1 347; with material
// maps 2 300: 1 761 / 2 455 / 1 827, 3 000: 2 406 / 2 440 / 1 775, 8 000: 6 426 /
// 2 501 / 1 889; wire chamber 4 000: 2 969 / 2 840 / 2 879, 5 000: 3 649 / 2 891 /
// 2 972 (pT from 0.1 GeV 4 640 / 8 960 / 8 862); telescope 1 000: 217 / 288 /
// 355, 1 800: 333 / 289 / 353; with volume material 1 000: 326 / 411 / 478,
// 1 400: 529 / 425 / 483, 8 000: 2 206 / 436 / 527.  With a window of one bin:
// toy 2 000: 584 / 665, 3 000: 862 / 665; with material maps 1 000: 814 / 966,
// 3 000: 1 884 / 966.
inline uint64_t group_limit_fp64(const launch_traits& t,
                                 const uint32_t window[2]) {
    const uint64_t part = narrow_search(t, window) ? 2u : 1u;
    if (t.lines) {
        return 5120u / part;
    }
    if (t.surface_grids) {
        return 3072u / part;
    }
    return t.extra_code ? 1184u : 2048u;
}

// Tracks from which the round-based method is the faster form of a call that
// asks for it: below, its rounds' latency (some 50 of 80 us) outweighs the
// plain kernel's divergence.  Plain sorted / rounds:
//   toy 200 000: 5 622 / 6 075, 400 000: 9 129 / 9 080, 1 000 000: 21 051 /
//   18 001; in the map 150 000: 6 096 / 6 118, 250 000: 9 962 / 7 903
//   toy with material maps 120 000: 5 061 / 6 342, 230 000: 9 663 / 9 639,
//   300 000: 11 057 / 10 229; in the map 120 000: 5 730 / 6 680, 230 000:
//   10 371 / 9 269
//   wire chamber, pT from 0.1 GeV, 12 289: 9 587 / 11 104, 20 000: 11 782 /
//   11 692; from 0.5 GeV 30 000: 3 763 / 4 376, 60 000: 5 228 / 4 682
//   a telescope without surface grids 1 000 000: 5 349 / 6 168; with volume
//   material 300 000: 2 476 / 3 454, 1 000 000: 8 135 / 8 473, in the map 9 235 /
//   9 084
inline uint64_t rounds_from(const launch_traits& t, bool field_map) {
    if (t.lines) {
        return 16384u;
    }
    if (!t.surface_grids) {
        return t.extra_code ? 1000000u : ~uint64_t(0);
    }
    if (field_map) {
        return 150000u;
    }
    return t.extra_code ? 230000u : 400000u;
}

// The same in double precision: toy in the map 75 000: 5 785 / 6 651, 100 000:
// 9 351 / 7 264; constant field 75 000: 3 544 / 5 817, 100 000: 5 679 / 6 314;
// with material maps 40 000: 4 396 / 6 300, 80 000: 7 953 / 7 096; wire chamber,
// pT from 0.1 GeV, 16 000: 12 835 / 13 846, 30 000: 16 817 / 14 452.
inline uint64_t rounds_from_fp64(const launch_traits& t) {
    return t.lines ? 25000u : 80000u;
}

// Tracks left to the tail of the round-based method, below which it begins
// when the launch does not say: n / 64, but no more than the kernel that runs
// a warp per track takes.  Beyond, the tail ran one thread per track, whose
// step is the slower one, and the longest track's steps are the tail's time.
// Rounds with n / 64 / with the bound, ms: wire chamber in the map, 2 M tracks
// from 0.1 GeV, one of them stepping 100 000 times 629 / 533, 200 / 178; toy
// with material maps in the map, 1 M from 0.1 GeV 98.2 / 49.3; in double
// precision 1 M toy tracks 55.1 / 46.5; 1 M toy tracks from 1 GeV 18.0 / 18.0.
constexpr uint32_t k_tail_wide = 8192u;
inline uint32_t default_tail_tracks(uint64_t n) {
    return n / 64u < k_tail_wide ? static_cast<uint32_t>(n / 64u)
                                 : k_tail_wide;
}

// Whether a plain propagation that asks for direction order is faster without
// it: where every track tests the same few surfaces an order gains little and
// scatters the results, unless they are staged or the batch is large.  Input
// order / sorted, fp32:
//   telescope (16 surfaces in the list) 10 000: 260 / 344, in the map 298 / 369;
//   without records 20 000: 297 / 323, 40 000: 352 / 335, 300 000: 1 543 / 1 328
//   the toy detector's modules as lists (1 096) 3 000: 14 098 / 12 685, 14 000:
//   14 539 / 11 937, 300 000 without records: 31 888 / 18 061
inline bool order_is_a_loss(const launch_traits& t, bool staged, uint64_t n) {
    return !t.surface_grids && !t.long_lists && !staged && n < 32768u;
}

// Register budget of the plain kernel, fp32: resident CTAs of 128 threads per
// SM, 4 (128 registers) while that keeps the whole batch resident, 512 tracks
// per SM; else 8 (64).  In a field map 16 (32 registers) from 1 536 per SM on
// when the volumes have surface grids and the window is wide: more warps hide
// the lookups and the grid's loads.  Tracks that test a list or one bin have
// less to hide.  4 / 8 / 12 / 16:
//   toy 75 000: 2 532 / 2 742 / 3 210 / 3 526, 150 000: 4 847 / 3 710 / 4 770 /
//   4 972, 1 200 000: - / 25 022 / 27 294 / 25 483; in the map 150 000: 7 772 /
//   6 169 / 7 846 / 8 051, 300 000: - / 11 694 / 13 054 / 10 778; with a window
//   of one bin 450 000: - / 7 111 / 8 181 / 9 599
//   wire chamber in the map 300 000: - / 19 504 / 23 051 / 17 542; toy with
//   material maps in the map 300 000: - / 12 556 / 13 829 / 11 860
//   telescope 10 000: 234 / 276 / 317 / 347; in the map 300 000: - / 2 051 /
//   2 706 / 2 927, 1 000 000: - / 6 570 / 8 231 / 9 537
//   the toy detector's modules as lists (1 096 in a volume), in the map, input
//   order 230 000: 49 412 / 28 715 / 34 391 / 34 001, sorted 25 674 / 18 328 /
//   18 072 / 22 662
inline int plain_budget(const launch_traits& t, const uint32_t window[2],
                        bool field_map, uint64_t tracks_per_sm) {
    if (tracks_per_sm < 512u) {
        return 4;
    }
    return field_map && t.surface_grids && window_bins(window) >= 16u &&
                   tracks_per_sm >= 1536u
               ? 16
               : 8;
}

// Whether the truth scan of n tracks runs a cluster of eight CTAs per track:
// unbounded is the number of surfaces the culling cannot skip (cylinders and
// lines), 256 the threads of a CTA.  Wire chamber, one CTA / a cluster: 1 track
// 250 / 83, 128: 255 / 159, 192: 280 / 202, 1 000: 721 / 771; fp64 1: 333 / 90,
// 192: 383 / 340, 256: 385 / 437.
inline bool scan_in_clusters(uint32_t unbounded, uint64_t n) {
    return unbounded > 256u && n <= 192u;
}

// Device scratch of a host call without jagged records: inputs (8 doubles a
// track), per-track outputs (status, six counters, path length, the 8 final
// parameters) and records (barcode, 6 + 21 + 1 floats, flags), each array
// from a 256-byte boundary on.
inline uint64_t host_scratch_bytes(uint64_t n, uint64_t max_records) {
    const auto al = [](uint64_t b) { return (b + 255u) & ~uint64_t(255u); };
    const uint64_t r = max_records * n;
    return 8u * al(8u * n) + al(n) + 15u * al(4u * n) + al(8u * r) +
           28u * al(4u * r) + al(r);
}

}  // namespace dprop
