"""Helpers of the GPU tests that compare launch forms."""
import numpy as np

DISCRETE = ("status", "n_records", "n_steps", "n_trials", "n_intersections",
            "n_transports", "n_material", "rec_barcode", "rec_flags")
NUMBERS = ("path_length", "final_free", "rec_path", "rec_bound")


def volume_material(tables):
    """The tables with every volume filled with their first slab material."""
    t = {k: v.copy() for k, v in tables.items()}
    slabs = t["slabs"]
    t["volumes"]["material"] = int(np.flatnonzero(
        (slabs["X0"] > 0) & (slabs["mean_excitation_energy"] > 0))[0])
    return t


def detector(name):
    """A committed geometry; 'telescope+material': filled with a slab's
    material."""
    from detray_b200 import geometry, propagator
    base = name.split("+")[0]
    full = {"toy": "toy_4brl_7edc", "maps": "toy_4brl_7edc_maps",
            "wire": "wire_chamber_10l_cells",
            "straw": "wire_chamber_10l_straws",
            "telescope": "telescope_10x1m_300um"}[base]
    tables = geometry.load_geometry(full)
    if name.endswith("+material"):
        tables = volume_material(tables)
    return propagator.Detector(tables)


def config(name, **kw):
    from detray_b200 import abi
    kw.setdefault("max_records", 48 if name[:4] in ("wire", "stra") else 24)
    window = (0, 0) if name.startswith("tele") else (3, 3)
    return abi.make_config(search_window=window, estimate_scattering_noise=0,
                           **kw)


def sample(name, n, seed=9):
    from detray_b200 import tracks
    if name.startswith("tele"):
        return tracks.telescope_tracks(n, seed=seed)
    return tracks.toy_tracks(n, seed=seed, pt_range=(0.5, 100.0),
                             eta_range=(-1.5, 1.5))


def run(det, field, cfg, dev, **launch):
    """Results of one call, as numpy arrays; unwritten entries are 0."""
    import torch

    from detray_b200 import propagator
    res = propagator.alloc_device_results(dev.shape[1], cfg.max_records,
                                          "cuda", dtype=dev.dtype)
    for t in res.tensors.values():
        t.zero_()
    propagator.propagate(cfg, det, field, dev, results=res,
                         launch=propagator.make_launch(
                             precision=8 if dev.dtype == torch.float64 else 0,
                             **launch))
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in res.tensors.items()}


def assert_same(a, b, what):
    """Equal discrete results; numbers within the parity tolerances (separate
    kernels may be contracted into fused multiply-adds differently)."""
    for k in DISCRETE:
        assert np.array_equal(a[k], b[k]), (what, k)
    double = a["path_length"].dtype == np.float64
    for k in NUMBERS:
        assert np.allclose(a[k], b[k], rtol=1e-9 if double else 1e-4,
                           atol=1e-9 if double else 2e-3,
                           equal_nan=True), (what, k)
    cov = [i * (11 - i) // 2 + i for i in range(6)]
    sig = np.sqrt(np.abs(a["rec_cov"][cov]))
    k = 0
    for i in range(6):
        for j in range(i, 6):
            d = np.abs(a["rec_cov"][k] - b["rec_cov"][k])
            tol = (1e-7 if double else 1e-3) * sig[i] * sig[j]
            assert (d <= tol + 1e-30).all(), (what, i, j)
            k += 1
