"""The round-based propagation simulated on the host with the navigation
state the step phase's kernels hold (nav_window): every track must end
bit-identical to the one-shot loop, whatever the rounds, the step budget and
the yield rule.  State a phase does not load is poison."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests.gpu_forms import volume_material

REPO = Path(__file__).resolve().parents[1]
T = 0.000299792458


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from detray_b200 import build
    out = tmp_path_factory.mktemp("window") / "libwindow.so"
    inc = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared",
                    f"-I{REPO / 'include'}", f"-I{build.CSRC}", f"-I{inc}",
                    str(REPO / "tests" / "native" / "rounds_window.cpp"),
                    "-o", str(out)], check=True)
    return C.CDLL(str(out))


def _results(n, cap):
    from detray_b200 import abi
    t = {k: np.zeros(n, np.uint32) for k in
         ("n_records", "n_steps", "n_trials", "n_intersections",
          "n_transports", "n_material")}
    t["status"] = np.zeros(n, np.uint8)
    t["path_length"] = np.zeros(n)
    t["final_free"] = np.zeros((8, n))
    t["rec_barcode"] = np.zeros((cap, n), np.uint64)
    t["rec_flags"] = np.zeros((cap, n), np.uint8)
    t["rec_path"] = np.zeros((cap, n))
    t["rec_bound"] = np.zeros((6, cap, n))
    t["rec_cov"] = np.zeros((21, cap, n))
    r = abi.Results()
    for k, v in t.items():
        if k in ("final_free", "rec_bound", "rec_cov"):
            for i in range(v.shape[0]):
                getattr(r, k)[i] = v[i].ctypes.data
        else:
            setattr(r, k, v.ctypes.data)
    return t, r


def _case(kind):
    from detray_b200 import abi, fields, geometry, tracks
    load = geometry.load_geometry
    noise = dict(estimate_scattering_noise=0)
    if kind == "telescope":
        return (load("telescope_10x1m_300um"), 0,
                tracks.telescope_tracks(300, seed=3),
                abi.make_config(max_records=16), None)
    if kind == "telescope_material":
        return (volume_material(load("telescope_10x1m_300um")), 1,
                tracks.telescope_tracks(300, seed=8),
                abi.make_config(max_records=16), None)
    if kind == "toy_map":
        return (load("toy_4brl_7edc"), 0,
                tracks.toy_tracks(400, seed=5, pt_range=(0.1, 100.0)),
                abi.make_config(max_records=32, search_window=(3, 3), **noise),
                fields.solenoid_map())
    if kind == "toy_maps":
        return (load("toy_4brl_7edc_maps"), 1,
                tracks.toy_tracks(300, seed=6),
                abi.make_config(max_records=5, search_window=(3, 3)), None)
    if kind == "wire":
        return (load("wire_chamber_10l_cells"), 1,
                tracks.toy_tracks(150, seed=13, pt_range=(0.1, 100.0),
                                  eta_range=(-1.0, 1.0),
                                  vertex_sigma=(0, 0, 0)),
                abi.make_config(max_records=64, search_window=(3, 3), **noise),
                None)
    return (load("toy_4brl_7edc"), 0, tracks.toy_tracks(400, seed=4),
            abi.make_config(max_records=32, search_window=(3, 3)), None)


@pytest.mark.parametrize("kind", ["telescope", "telescope_material", "toy",
                                  "toy_map", "toy_maps", "wire"])
@pytest.mark.parametrize("precision", [4, 8])
def test_window_rounds_equal_one_shot_loop(lib, kind, precision):
    from detray_b200 import geometry
    tables, all_code, trk, cfg, fmap = _case(kind)
    det = geometry.Descriptor(tables)
    n = trk.shape[1]
    trk = np.ascontiguousarray(trk)
    ptrs = (C.c_void_p * 8)(*[trk[i].ctypes.data for i in range(8)])
    if fmap is None:
        field = (0, (C.c_double * 3)(0.0, 0.0, 2.0 * T), None, None, None,
                 None)
    else:
        values = np.ascontiguousarray(fmap["values"], dtype=np.float32)
        field = (1, (C.c_double * 3)(), (C.c_double * 3)(*fmap["lo"]),
                 (C.c_double * 3)(*fmap["hi"]), (C.c_uint32 * 3)(*fmap["n"]),
                 values.ctypes.data_as(C.c_void_p))
    want, r = _results(n, cfg.max_records)
    assert lib.core_host_propagate(precision, C.byref(det.desc), *field,
                                   C.byref(cfg), ptrs, C.c_uint64(n),
                                   C.byref(r)) == 0
    if precision == 4:
        # the loop's path accumulator is double, the phases store a float
        want["path_length"] = want["path_length"].astype(np.float32)
    ends = C.c_uint64(0)
    # (rounds, step budget, yield lanes)
    for rounds, budget, yield_min in [(300, 16, 8), (300, 1, 1), (7, 3, 16)]:
        got, r = _results(n, cfg.max_records)
        assert lib.rounds_window(precision, C.byref(det.desc), all_code,
                                 *field, C.byref(cfg), ptrs, C.c_uint64(n),
                                 C.byref(r), rounds, budget, yield_min,
                                 C.byref(ends)) == 0
        for k, x in want.items():
            y = got[k]
            if k == "path_length" and precision == 4:
                y = y.astype(np.float32)
            assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f"), k
    if kind == "telescope":
        # more surfaces ahead than the cache holds: its end was reached
        assert ends.value > 0
