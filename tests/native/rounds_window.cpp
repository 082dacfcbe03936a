// TEST-ONLY: the round-based propagation on the host with the step phase's
// own navigation state (nav_window: three candidates held, the re-intersected
// target written back), as the kernels run it.
#include "core_host.cpp"

namespace {

template <typename S, bool W>
void window_rounds(const detector_view<S, W>& det, const field_view<S>& field,
                   const prop_cfg<S>& cfg, const double* const* trk,
                   uint64_t n, const dprop_results* out, uint32_t rounds,
                   uint32_t step_budget, uint32_t yield_min,
                   uint64_t* seen_end) {
    using fast_state = track_state<S, false, nav_window<S>>;
    const uint32_t cap = cfg.max_records;
    std::vector<unsigned char> mem(carve_slots<S>(nullptr, n, W, nullptr) +
                                   256u);
    void* base = reinterpret_cast<void*>(
        (reinterpret_cast<uintptr_t>(mem.data()) + 255u) & ~uintptr_t(255u));
    slot_soa<S> s{};
    carve_slots<S>(base, n, W, &s);
    std::vector<uint32_t> stage(
        static_cast<size_t>(cap) * n * staged_record_words<S>() + 4u);
    uint32_t* stage_base = reinterpret_cast<uint32_t*>(
        (reinterpret_cast<uintptr_t>(stage.data()) + 15u) & ~uintptr_t(15u));
    record_sink<S> rec{};
    rec.n_tracks = n;
    rec.capacity = cap;
    rec.stage = stage_base;

    auto emit = [&](const track_outputs<S>& o, uint64_t t) {
        out->status[t] = o.status;
        out->n_records[t] = o.n_records;
        out->n_steps[t] = o.n_steps;
        out->n_trials[t] = o.n_trials;
        out->n_intersections[t] = o.n_isect;
        out->n_transports[t] = o.n_transport;
        out->n_material[t] = o.n_material;
        static_cast<double*>(out->path_length)[t] = o.path_length;
        for (int i = 0; i < 8; ++i) {
            static_cast<double*>(out->final_free[i])[t] = o.fin[i];
        }
    };
    for (uint64_t t = 0; t < n; ++t) {
        auto in = [&](int i) { return static_cast<S>(trk[i][t]); };
        phase_init<S, W>(s, n - 1u - t, static_cast<uint32_t>(t),
                         vec3<S>{in(0), in(1), in(2)}, in(3),
                         vec3<S>{in(4), in(5), in(6)}, in(7), det, cfg);
    }
    for (uint32_t r = 0; r < rounds; ++r) {
        std::vector<uint64_t> fast, nav;
        for (uint64_t slot = 0; slot < n; ++slot) {
            const uint8_t pc = s.pc[slot];
            if (pc == pc_nav) {
                nav.push_back(slot);
            } else if (pc != pc_done) {
                fast.push_back(slot);
            }
        }
        for (size_t g0 = 0; g0 < fast.size(); g0 += 32u) {
            const size_t m =
                fast.size() - g0 < 32u ? fast.size() - g0 : 32u;
            std::vector<fast_state> ts(m);
            std::vector<loop_state<S>> ls(m);
            std::vector<cand_window> win(m);
            std::vector<char> active(m, 1);
            for (size_t l = 0; l < m; ++l) {
                std::memset(static_cast<void*>(&ts[l]), 0xff, sizeof(ts[l]));
                std::memset(static_cast<void*>(&ls[l]), 0xff, sizeof(ls[l]));
                fast_load<S, W>(s, fast[g0 + l], ts[l], ls[l], win[l]);
            }
            for (uint32_t it = 0;; ++it) {
                uint32_t live = 0;
                for (size_t l = 0; l < m; ++l) {
                    if (!active[l]) continue;
                    active[l] = machine_is_fast(fast_advance<S, W>(
                        ts[l], ls[l], win[l], s, fast[g0 + l], det, field,
                        cfg, rec));
                    live += active[l] ? 1u : 0u;
                    *seen_end += ts[l].nav.next >= k_cache ? 1u : 0u;
                }
                if (live == 0u || it + 1u >= step_budget || live < yield_min) {
                    break;
                }
            }
            for (size_t l = 0; l < m; ++l) {
                const uint64_t slot = fast[g0 + l];
                fast_store<S, W>(s, slot, ts[l], ls[l], win[l]);
                if (ls[l].pc == pc_done) {
                    emit(fast_outputs(s, slot, ts[l], ls[l]), s.track[slot]);
                }
            }
        }
        for (const uint64_t slot : nav) {
            phase_nav<S, W>(s, slot, det, cfg);
        }
    }
    for (uint64_t slot = 0; slot < n; ++slot) {
        if (s.pc[slot] != pc_done) {
            emit(phase_tail<S, W>(s, slot, det, field, cfg, rec),
                 s.track[slot]);
        }
    }
    // records: staged rows to the result layout, widened
    std::vector<uint64_t> bc(static_cast<size_t>(cap) * n);
    std::vector<uint8_t> fl(static_cast<size_t>(cap) * n);
    std::vector<S> bound[6], cov[21], path(static_cast<size_t>(cap) * n);
    S* bptr[6];
    S* cptr[21];
    for (int i = 0; i < 6; ++i) {
        bound[i].resize(static_cast<size_t>(cap) * n);
        bptr[i] = bound[i].data();
    }
    for (int i = 0; i < 21; ++i) {
        cov[i].resize(static_cast<size_t>(cap) * n);
        cptr[i] = cov[i].data();
    }
    record_sink<S> direct{};
    direct.barcode = bc.data();
    direct.bound = bptr;
    direct.cov = cptr;
    direct.path = path.data();
    direct.flags = fl.data();
    direct.n_tracks = n;
    direct.capacity = cap;
    for (uint64_t t = 0; t < n; ++t) {
        const uint64_t slot = n - 1u - t;
        unstage_records<S>(stage_base, slot, s.rec_count[slot], t, direct);
        const uint32_t m = s.rec_count[slot] < cap ? s.rec_count[slot] : cap;
        for (uint32_t k = 0; k < m; ++k) {
            const uint64_t o = static_cast<uint64_t>(k) * n + t;
            out->rec_barcode[o] = bc[o];
            out->rec_flags[o] = fl[o];
            static_cast<double*>(out->rec_path)[o] = path[o];
            for (int i = 0; i < 6; ++i) {
                static_cast<double*>(out->rec_bound[i])[o] = bound[i][o];
            }
            for (int i = 0; i < 21; ++i) {
                static_cast<double*>(out->rec_cov[i])[o] = cov[i][o];
            }
        }
    }
}

template <typename S>
int window_run(const dprop_detector_desc* desc, int all_code,
               uint32_t field_kind, const double* b, const double* lo,
               const double* hi, const uint32_t* nn, const float* values,
               const dprop_config* c, const double* const* trk, uint64_t n,
               const dprop_results* out, uint32_t rounds, uint32_t budget,
               uint32_t yield_min, uint64_t* seen_end) {
    if (!validate_desc(desc).empty()) {
        return 1;
    }
    const host_tables<S> tables = convert_desc<S>(desc);
    std::vector<float4> nodes;
    const field_view<S> f =
        host_field<S>(field_kind, b, lo, hi, nn, values, nodes);
    const prop_cfg<S> cfg = make_prop_cfg<S>(*c);
    if (all_code) {
        window_rounds<S, true>(tables.template view_as<true>(), f, cfg, trk, n,
                               out, rounds, budget, yield_min, seen_end);
    } else {
        window_rounds<S, false>(tables.template view_as<false>(), f, cfg, trk,
                                n, out, rounds, budget, yield_min, seen_end);
    }
    return 0;
}

}  // namespace

extern "C" int rounds_window(int precision, const dprop_detector_desc* desc,
                             int all_code, uint32_t field_kind,
                             const double* b, const double* lo,
                             const double* hi, const uint32_t* nn,
                             const float* values, const dprop_config* cfg,
                             const double* const* trk, uint64_t n,
                             const dprop_results* out, uint32_t rounds,
                             uint32_t budget, uint32_t yield_min,
                             uint64_t* seen_end) {
    return precision == 8
               ? window_run<double>(desc, all_code, field_kind, b, lo, hi, nn,
                                    values, cfg, trk, n, out, rounds, budget,
                                    yield_min, seen_end)
               : window_run<float>(desc, all_code, field_kind, b, lo, hi, nn,
                                   values, cfg, trk, n, out, rounds, budget,
                                   yield_min, seen_end);
}
