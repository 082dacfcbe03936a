// Helix truth scan for navigation validation: the C ABI entry points
// dprop_helix_scan and dprop_validate_navigation (dprop.h).
//
// Kernels:
//   helix_scan_kernel    one CTA (or a cluster) per track: the surfaces are tested against
//                        the track's helix (scan_may_hit, core/helix.cuh) and
//                        the few it may hit are intersected (root search,
//                        one thread per surface); hits inside a mask and
//                        along the track are sorted by |path| (ties by
//                        surface index, which is the reference's stable
//                        order over the surface list) and cut after the
//                        first hit that leaves the world
//   validate_kernel      one thread per track: holes and extra surfaces of
//                        a propagation's records against the scan
// The surfaces of a detector are read by every track: they stay in L2.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "api_common.cuh"
#include "core/helix.cuh"

using namespace dprop;
using dprop::api::fail;

namespace {

// Threads of a track's CTA: most tracks' surfaces to search take one pass.
constexpr int k_scan_block = 256;
// Of a detector with no more surfaces than a warp has lanes: more warps would
// only be launched and wait at the barriers (telescope, field across it, 4 000
// tracks 158 us with 256 threads, 84 with 32; in double 1 000: 134 / 75).
constexpr int k_scan_block_few = 32;
// CTAs of a track's cluster where few tracks have many surfaces to search.
constexpr int k_scan_cluster = 8;
constexpr int k_validate_block = 256;

template <typename S>
struct scan_io {
    const S* trk[8];
    uint8_t* status;
    uint32_t* n_hits;
    uint64_t* barcode;
    S* path;
    S* loc[2];
    uint16_t* volume_link;
    uint32_t capacity;
};

// Hits of one track kept in shared memory until they are sorted.  A track
// with more of them (toy detector: 54 at most) goes through the result
// arrays instead.
constexpr uint32_t k_smem_hits = 128u;

template <typename S>
struct hit_list {
    S path[k_smem_hits];
    S loc0[k_smem_hits];
    S loc1[k_smem_hits];
    uint64_t barcode[k_smem_hits];
    uint16_t volume_link[k_smem_hits];
};

template <typename S>
__device__ __forceinline__ void write_hit(const scan_io<S>& io, uint64_t o,
                                          uint64_t barcode, S path, S loc0,
                                          S loc1, uint16_t volume_link) {
    io.barcode[o] = barcode;
    io.path[o] = path;
    if (io.loc[0]) io.loc[0][o] = loc0;
    if (io.loc[1]) io.loc[1][o] = loc1;
    io.volume_link[o] = volume_link;
}

template <typename S>
__device__ void swap_hits(const scan_io<S>& io, uint64_t a, uint64_t b) {
    const uint64_t bc = io.barcode[a];
    io.barcode[a] = io.barcode[b];
    io.barcode[b] = bc;
    const S p = io.path[a];
    io.path[a] = io.path[b];
    io.path[b] = p;
    for (int i = 0; i < 2; ++i) {
        if (io.loc[i]) {
            const S l = io.loc[i][a];
            io.loc[i][a] = io.loc[i][b];
            io.loc[i][b] = l;
        }
    }
    const uint16_t v = io.volume_link[a];
    io.volume_link[a] = io.volume_link[b];
    io.volume_link[b] = v;
}

// surface index of a barcode (bits 27..47)
__device__ __forceinline__ uint64_t sf_key(uint64_t bc) {
    return (bc >> 27) & 0x1fffffu;
}

// whether hit a comes after hit b
template <typename S>
__device__ __forceinline__ bool hit_after(S path_a, uint64_t bc_a, S path_b,
                                          uint64_t bc_b) {
    const S pa = fabs(path_a);
    const S pb = fabs(path_b);
    return pa > pb || (pa == pb && sf_key(bc_a) > sf_key(bc_b));
}

// Sort and cut of a track whose hits are all in the result arrays (one
// thread): insertion sort of the track's slots.  Returns the hits kept.
template <typename S>
__device__ uint32_t finish_in_results(const scan_io<S>& io, uint64_t t,
                                      uint64_t n, uint32_t found) {
    for (uint32_t i = 1; i < found; ++i) {
        for (uint32_t j = i; j > 0; --j) {
            const uint64_t a = static_cast<uint64_t>(j - 1) * n + t;
            const uint64_t b = static_cast<uint64_t>(j) * n + t;
            if (!hit_after(io.path[a], io.barcode[a], io.path[b],
                           io.barcode[b])) {
                break;
            }
            swap_hits(io, a, b);
        }
    }
    for (uint32_t k = 0; k < found; ++k) {
        if (io.volume_link[static_cast<uint64_t>(k) * n + t] ==
            static_cast<uint16_t>(DPROP_INVALID_LINK)) {
            return k + 1u;
        }
    }
    return found;
}

// One CTA per track.  Bound by the latency of the root searches (a chain of
// sine/cosine evaluations, 10 to 60 of them), not by memory.  The bounding
// test costs about 100 instructions a surface where a search takes 1 500 and
// more; on the toy detector it keeps about 5 % of the 4 158 surfaces: the 94
// portals and about 110 modules.  The kept surfaces are collected across the
// tests, so that the searches run with full warps, and the hits are ranked in
// shared memory instead of being sorted in the result arrays by one thread.
// 256 threads, so that most tracks take one pass of searches (128: 2.44
// against 2.18 ms).  8 192 toy tracks in fp32: 99.2 ms with a search per
// (track, surface), 2.0 ms now; 1 500 tracks in fp64 with the propagation
// they validate: 155.6 ms before, 3.0 ms now (B200).
//
// Block: threads of a CTA.  Ctas > 1: a cluster of that many per track divides
// the surfaces and collects the hits in its first CTA's shared memory.  Few
// tracks leave SMs idle, and the culling keeps every cylinder and line of a
// wire chamber (1 933 surfaces: eight passes of searches, one after the other;
// one track 250 us in one CTA, 83 in a cluster, in double 333 and 90).
template <typename S, bool W, int Block, int Ctas>
__global__ void __launch_bounds__(Block)
    helix_scan_kernel(const __grid_constant__ detector_view<S, W> det,
                      const scan_bound* __restrict__ bounds,
                      const __grid_constant__ scan_io<S> io, vec3<S> bfield,
                      S mask_tol, uint64_t n) {
    __shared__ hit_list<S> own_hits;
    __shared__ uint32_t todo[2 * Block];
    __shared__ uint32_t n_todo, own_found, n_kept;
    const uint64_t t = blockIdx.x / static_cast<uint32_t>(Ctas);
    const uint32_t part = blockIdx.x % static_cast<uint32_t>(Ctas);
    const uint32_t tid = threadIdx.x;
    hit_list<S>* all_hits = &own_hits;
    uint32_t* n_found = &own_found;
    if constexpr (Ctas > 1) {
        const auto cluster = cooperative_groups::this_cluster();
        all_hits = cluster.map_shared_rank(&own_hits, 0);
        n_found = cluster.map_shared_rank(&own_found, 0);
    }
    hit_list<S>& hits = *all_hits;
    if (tid == 0u) {
        n_todo = 0u;
        own_found = 0u;
    }
    helix<S> h;
    h.init(vec3<S>{io.trk[0][t], io.trk[1][t], io.trk[2][t]},
           vec3<S>{io.trk[4][t], io.trk[5][t], io.trk[6][t]}, io.trk[7][t],
           bfield);
    scan_probe probe;
    probe.init(h);
    const float tol = static_cast<float>(mask_tol);
    const root_cfg<S> cfg{S(unit::um), 1000u, S(5000) * S(unit::mm)};
    const uint32_t cap = io.capacity;
    if constexpr (Ctas > 1) {
        // the first CTA's counter is set, and its shared memory there
        cooperative_groups::this_cluster().sync();
    } else {
        __syncthreads();
    }
    constexpr uint32_t stride = Ctas * Block;
    for (uint32_t base = part * Block; base < det.n_surfaces; base += stride) {
        const uint32_t sf = base + tid;
        const bool keep =
            sf < det.n_surfaces && scan_may_hit(bounds[sf], probe, tol);
        const uint32_t kept = __ballot_sync(0xffffffffu, keep);
        uint32_t at = 0u;
        if ((tid & 31u) == 0u && kept != 0u) {
            at = atomicAdd(&n_todo, static_cast<uint32_t>(__popc(kept)));
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        if (keep) {
            todo[at + __popc(kept & ((1u << (tid & 31u)) - 1u))] = sf;
        }
        __syncthreads();
        uint32_t m = n_todo;
        __syncthreads();  // every thread has read it
        // a full CTA of surfaces, or the last ones
        const bool last = base + stride >= det.n_surfaces;
        const bool search = m >= Block || (last && m > 0u);
        while (m >= Block || (last && m > 0u)) {
            const uint32_t first = m > Block ? m - Block : 0u;
            if (first + tid < m) {
                helix_surface_hits(
                    det, todo[first + tid], h, mask_tol, cfg,
                    [&](const scan_hit<S>& hit) {
                        const uint32_t k = atomicAdd(n_found, 1u);
                        const uint64_t bc = det.surfaces[hit.sf].barcode;
                        if (k < k_smem_hits) {
                            hits.path[k] = hit.path;
                            hits.loc0[k] = hit.loc0;
                            hits.loc1[k] = hit.loc1;
                            hits.barcode[k] = bc;
                            hits.volume_link[k] = hit.volume_link;
                        } else if (k < cap) {
                            write_hit(io, static_cast<uint64_t>(k) * n + t, bc,
                                      hit.path, hit.loc0, hit.loc1,
                                      hit.volume_link);
                        }
                    });
            }
            m = first;
        }
        if (search) {
            __syncthreads();  // the searched entries may be overwritten
            if (tid == 0u) {
                n_todo = m;
            }
            __syncthreads();
        }
    }
    if constexpr (Ctas > 1) {
        // every CTA's hits are in the first one's list, which goes on alone
        cooperative_groups::this_cluster().sync();
        if (part != 0u) {
            return;
        }
    }
    const uint32_t found = own_found;
    if (found == 0u) {
        if (tid == 0u) {
            io.n_hits[t] = 0u;
            io.status[t] = DPROP_SCAN_EMPTY;
        }
        return;
    }
    if (tid == 0u) {
        n_kept = found;
    }
    __syncthreads();
    const bool in_smem = found <= k_smem_hits && found <= cap;
    const uint32_t held = found < k_smem_hits ? found : k_smem_hits;
    for (uint32_t k = tid; k < held; k += Block) {
        uint32_t slot = k;
        if (in_smem) {
            // the hit's place in the sorted list
            slot = 0u;
            for (uint32_t j = 0; j < found; ++j) {
                const bool before =
                    hit_after(hits.path[k], hits.barcode[k], hits.path[j],
                              hits.barcode[j]) ||
                    (j < k && !hit_after(hits.path[j], hits.barcode[j],
                                         hits.path[k], hits.barcode[k]));
                slot += before ? 1u : 0u;
            }
            if (hits.volume_link[k] ==
                static_cast<uint16_t>(DPROP_INVALID_LINK)) {
                atomicMin(&n_kept, slot + 1u);
            }
        }
        if (slot < cap) {
            write_hit(io, static_cast<uint64_t>(slot) * n + t, hits.barcode[k],
                      hits.path[k], hits.loc0[k], hits.loc1[k],
                      hits.volume_link[k]);
        }
    }
    __syncthreads();  // also orders the CTA's writes to the result arrays
    if (tid == 0u) {
        uint32_t kept = n_kept;
        if (!in_smem && found <= cap) {
            kept = finish_in_results(io, t, n, found);
        }
        io.n_hits[t] = kept;
        io.status[t] =
            found > cap ? DPROP_SCAN_OVERFLOW : DPROP_SCAN_OK;
    }
}

template <typename S>
dprop_status launch_scan(const dprop_detector* det, const double b[3],
                         const dprop_tracks* tracks, uint64_t n,
                         double mask_tol, const dprop_scan_results* r,
                         cudaStream_t st) {
    scan_io<S> io{};
    for (int i = 0; i < 3; ++i) {
        io.trk[i] = static_cast<const S*>(tracks->pos[i]);
        io.trk[4 + i] = static_cast<const S*>(tracks->dir[i]);
    }
    io.trk[3] = static_cast<const S*>(tracks->time);
    io.trk[7] = static_cast<const S*>(tracks->qop);
    io.status = r->status;
    io.n_hits = r->n_hits;
    io.barcode = r->barcode;
    io.path = static_cast<S*>(r->path);
    io.loc[0] = static_cast<S*>(r->loc[0]);
    io.loc[1] = static_cast<S*>(r->loc[1]);
    io.volume_link = r->volume_link;
    io.capacity = r->capacity;
    const vec3<S> bf{static_cast<S>(b[0]), static_cast<S>(b[1]),
                     static_cast<S>(b[2])};
    const auto run = [&](auto view) -> dprop_status {
        using view_t = decltype(view);
        constexpr bool W =
            std::is_same<view_t, detector_view<S, true>>::value;
        cudaLaunchConfig_t lc{};
        lc.stream = st;
        lc.gridDim = dim3(static_cast<unsigned int>(n));
        lc.blockDim = dim3(k_scan_block);
        cudaLaunchAttribute cluster{};
        const S tol = static_cast<S>(mask_tol);
        if (det->n_surfaces <= static_cast<uint32_t>(k_scan_block_few)) {
            lc.blockDim = dim3(k_scan_block_few);
            DPROP_CUDA(cudaLaunchKernelEx(
                &lc, helix_scan_kernel<S, W, k_scan_block_few, 1>, view,
                static_cast<const scan_bound*>(det->scan_bounds), io, bf, tol,
                n));
        } else if (scan_in_clusters(det->n_unbounded, n)) {
            lc.gridDim = dim3(static_cast<unsigned int>(n * k_scan_cluster));
            cluster.id = cudaLaunchAttributeClusterDimension;
            cluster.val.clusterDim.x = k_scan_cluster;
            cluster.val.clusterDim.y = 1;
            cluster.val.clusterDim.z = 1;
            lc.attrs = &cluster;
            lc.numAttrs = 1;
            DPROP_CUDA(cudaLaunchKernelEx(
                &lc, helix_scan_kernel<S, W, k_scan_block, k_scan_cluster>,
                view, static_cast<const scan_bound*>(det->scan_bounds), io, bf,
                tol, n));
        } else {
            DPROP_CUDA(cudaLaunchKernelEx(
                &lc, helix_scan_kernel<S, W, k_scan_block, 1>, view,
                static_cast<const scan_bound*>(det->scan_bounds), io, bf, tol,
                n));
        }
        return DPROP_OK;
    };
    if constexpr (sizeof(S) == 8) {
        return det->wires ? run(det->view_d_as<true>())
                          : run(det->view_d_as<false>());
    } else {
        return det->wires ? run(det->view_as<true>())
                          : run(det->view_as<false>());
    }
}

template <typename Ti, typename Tr>
__global__ void __launch_bounds__(k_validate_block)
    validate_kernel(const uint8_t* __restrict__ scan_status,
                    const uint32_t* __restrict__ n_hits,
                    const uint64_t* __restrict__ truth_bc,
                    const Ti* __restrict__ truth_path,
                    const uint16_t* __restrict__ truth_vlink,
                    const uint8_t* __restrict__ rec_status,
                    const uint32_t* __restrict__ n_records,
                    const uint64_t* __restrict__ rec_bc,
                    const Tr* __restrict__ rec_path, uint32_t max_records,
                    uint64_t n, double path_tol, uint32_t* n_missed,
                    uint32_t* n_extra) {
    const uint64_t t =
        static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) {
        return;
    }
    const uint32_t nt = (scan_status[t] == DPROP_SCAN_OK) ? n_hits[t] : 0u;
    const uint32_t nr = n_records[t] < max_records ? n_records[t] : max_records;
    uint32_t missed, extra;
    compare_trace(truth_bc, truth_path, truth_vlink, nt, rec_bc, rec_path, nr,
                  rec_status[t] == DPROP_TRK_EXITED, n, t, path_tol, missed,
                  extra);
    n_missed[t] = missed;
    n_extra[t] = extra;
}

template <typename Ti, typename Tr>
void launch_validate(const dprop_scan_results* s, const dprop_results* r,
                     uint32_t max_records, uint64_t n, double tol,
                     const dprop_validation* out, cudaStream_t st) {
    const unsigned int tb =
        static_cast<unsigned int>((n + k_validate_block - 1) / k_validate_block);
    validate_kernel<Ti, Tr><<<tb, k_validate_block, 0, st>>>(
        s->status, s->n_hits, s->barcode, static_cast<const Ti*>(s->path),
        s->volume_link, r->status, r->n_records, r->rec_barcode,
        static_cast<const Tr*>(r->rec_path), max_records, n, tol,
        out->n_missed, out->n_extra);
}

}  // namespace

extern "C" {

dprop_status dprop_validate_navigation(const dprop_scan_results* s,
                                       const dprop_results* r,
                                       uint32_t record_precision,
                                       uint32_t max_records, uint64_t n,
                                       double path_tolerance,
                                       const dprop_validation* out,
                                       void* stream) {
    if (!s || !r || !out) {
        return fail(DPROP_E_INVALID, "validate_navigation: NULL argument");
    }
    if ((s->precision != 4u && s->precision != 8u) ||
        (record_precision != 4u && record_precision != 8u)) {
        return fail(DPROP_E_INVALID,
                    "validate_navigation: precision must be 4 or 8");
    }
    if (!(path_tolerance >= 0.0)) {
        return fail(DPROP_E_INVALID,
                    "validate_navigation: negative path tolerance");
    }
    if (n == 0) {
        return DPROP_OK;
    }
    if (n > 0x7fffffffull) {
        return fail(DPROP_E_INVALID, "validate_navigation: too many tracks");
    }
    if (!s->status || !s->n_hits || !s->barcode || !s->path ||
        !s->volume_link || !r->status || !r->n_records ||
        (max_records > 0u && (!r->rec_barcode || !r->rec_path)) ||
        !out->n_missed || !out->n_extra) {
        return fail(DPROP_E_INVALID, "validate_navigation: missing array");
    }
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (s->precision == 8u) {
        if (record_precision == 8u) {
            launch_validate<double, double>(s, r, max_records, n,
                                            path_tolerance, out, st);
        } else {
            launch_validate<double, float>(s, r, max_records, n,
                                           path_tolerance, out, st);
        }
    } else {
        if (record_precision == 8u) {
            launch_validate<float, double>(s, r, max_records, n,
                                           path_tolerance, out, st);
        } else {
            launch_validate<float, float>(s, r, max_records, n,
                                          path_tolerance, out, st);
        }
    }
    DPROP_CUDA(cudaGetLastError());
    return DPROP_OK;
}

dprop_status dprop_helix_scan(const dprop_detector* det, const double b[3],
                              const dprop_tracks* tracks, uint64_t n,
                              double mask_tolerance,
                              const dprop_scan_results* r, void* stream) {
    if (!det || !b || !tracks || !r) {
        return fail(DPROP_E_INVALID, "helix_scan: NULL argument");
    }
    if (r->precision != 4u && r->precision != 8u) {
        return fail(DPROP_E_INVALID, "helix_scan: precision must be 4 or 8");
    }
    const double bb = b[0] * b[0] + b[1] * b[1] + b[2] * b[2];
    if (!(bb > 0.0) || !(bb < 1e30)) {
        return fail(DPROP_E_INVALID,
                    "helix_scan: the field must be finite and non-zero");
    }
    if (!(mask_tolerance >= 0.0) || !(mask_tolerance < 1e3)) {
        return fail(DPROP_E_INVALID,
                    "helix_scan: mask_tolerance must be in [0, 1000) mm");
    }
    if (n == 0) {
        return DPROP_OK;
    }
    if (n > 0x7fffffffull) {
        return fail(DPROP_E_INVALID, "helix_scan: too many tracks");
    }
    for (int i = 0; i < 3; ++i) {
        if (!tracks->pos[i] || !tracks->dir[i]) {
            return fail(DPROP_E_INVALID, "helix_scan: missing track array");
        }
    }
    if (!tracks->time || !tracks->qop || !r->status || !r->n_hits ||
        !r->volume_link || (r->capacity > 0u && (!r->barcode || !r->path))) {
        return fail(DPROP_E_INVALID, "helix_scan: missing array");
    }
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (r->precision == 8u) {
        return launch_scan<double>(det, b, tracks, n, mask_tolerance, r, st);
    }
    return launch_scan<float>(det, b, tracks, n, mask_tolerance, r, st);
}

}  // extern "C"
