"""The forms of an open launch shape follow what a track spends its time on,
not which options its kernels are compiled with: a detector with material maps
or volume material is no wire detector.  The bounds are batch sizes at which
the other form was measured at least 1.2 times slower."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parents[1]
NEVER = 2**64 - 1


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    from detray_b200 import abi, build, geometry
    out = tmp_path_factory.mktemp("rules") / "librules.so"
    inc = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared",
                    f"-I{REPO / 'include'}", f"-I{build.CSRC}", f"-I{inc}",
                    str(REPO / "tests" / "native" / "launch_rules.cpp"),
                    "-o", str(out)], check=True)
    lib = C.CDLL(str(out))

    def get(tables, extra_code, field_map=0, window=3):
        desc = geometry.Descriptor(tables)
        v = (C.c_uint64 * 6)()
        w = (C.c_uint32 * 2)(window, window)
        assert lib.launch_rules(C.byref(desc.desc), extra_code, w, field_map,
                                v) == 0
        return dict(zip(("group", "group64", "adjoint", "adjoint_grad",
                         "rounds", "rounds64"), v))

    def budget(tables, extra_code, field_map, tracks_per_sm, window=3):
        desc = geometry.Descriptor(tables)
        w = (C.c_uint32 * 2)(window, window)
        return lib.plain_budget_of(C.byref(desc.desc), extra_code, w,
                                   field_map, C.c_uint64(tracks_per_sm))

    def drops_order(tables, staged, n):
        desc = geometry.Descriptor(tables)
        return bool(lib.drops_order(C.byref(desc.desc), staged,
                                    C.c_uint64(n)))

    get.tail = lambda n: lib.tail_of(C.c_uint64(n))
    lib.host_scratch.restype = C.c_uint64
    get.host_scratch = lambda n, r: lib.host_scratch(C.c_uint64(n),
                                                     C.c_uint64(r))
    def scan_clusters(tables, n):
        desc = geometry.Descriptor(tables)
        return bool(lib.scan_clusters(C.byref(desc.desc), C.c_uint64(n)))

    get.scan_clusters = scan_clusters
    get.budget = budget
    get.drops_order = drops_order
    get.load = geometry.load_geometry
    get.abi = abi
    return get


def test_material_maps_are_no_wire_detector(rules):
    toy = rules(rules.load("toy_4brl_7edc"), 0)
    maps = rules(rules.load("toy_4brl_7edc_maps"), 1)
    assert 3000 <= maps["group"] <= 5000 < toy["group"] <= 7000
    assert maps["group64"] <= 3500
    assert maps["adjoint"] <= 3000 and maps["adjoint_grad"] <= 1400
    assert maps["rounds"] >= 120000 and maps["rounds64"] >= 40000
    assert rules(rules.load("toy_4brl_7edc_maps"), 1, 1)["rounds"] >= 120000


def test_volume_material_is_no_wire_detector(rules):
    t = {k: v.copy() for k, v in rules.load("telescope_10x1m_300um").items()}
    slabs = t["slabs"]
    t["volumes"]["material"] = int(np.flatnonzero(
        (slabs["X0"] > 0) & (slabs["mean_excitation_energy"] > 0))[0])
    got = rules(t, 1)
    assert got["group"] <= 1800 and got["group64"] <= 1400
    assert got["rounds"] >= 700000


def test_material_maps_are_no_surface_grids(rules):
    """A telescope whose volumes have no grid, beside a grid that is a
    material map."""
    t = {k: v.copy() for k, v in rules.load("telescope_10x1m_300um").items()}
    maps = rules.load("toy_4brl_7edc_maps")
    abi = rules.abi
    kinds = maps["grids"]["kind"]
    i = int(np.flatnonzero(kinds >= 3)[0])
    g = maps["grids"][i:i + 1].copy()
    n = int(g["n_bins"][0][0] * g["n_bins"][0][1])
    g["bin_offset"] = 0
    g["transform"] = 0
    t["grids"] = g
    t["grid_bins"] = np.zeros(n, np.uint32)
    assert (t["volumes"]["grid"] == abi.DPROP_INVALID_INDEX).all()
    assert rules(t, 1)["rounds"] >= 700000


def test_telescope(rules):
    assert rules(rules.load("telescope_10x1m_300um"), 0)["rounds"] == NEVER


def test_wire_chamber(rules):
    for name in ("wire_chamber_10l_cells", "wire_chamber_10l_straws"):
        got = rules(rules.load(name), 1)
        assert 5000 <= got["group"] <= 8200
        assert got["group64"] <= 6000
        assert got["adjoint"] <= 5500 and got["adjoint_grad"] <= 2100
        assert got["rounds"] <= 30000


def test_budget_of_large_batches(rules):
    """32 registers per thread pay in a field map where volumes have surface
    grids, and only there."""
    big = 2000
    assert rules.budget(rules.load("toy_4brl_7edc"), 0, 1, big) == 16
    assert rules.budget(rules.load("wire_chamber_10l_cells"), 1, 1, big) == 16
    assert rules.budget(rules.load("toy_4brl_7edc"), 0, 0, big) == 8
    tele = rules.load("telescope_10x1m_300um")
    for extra in (0, 1):
        for field_map in (0, 1):
            assert rules.budget(tele, extra, field_map, big) == 8
            assert rules.budget(tele, extra, field_map, 511) == 4


def _grids_as_lists(tables, abi):
    """The surfaces of every volume's grid in its brute-force list."""
    t = {k: v.copy() for k, v in tables.items()}
    lists = []
    for v in t["volumes"]:
        own = list(t["bf_surfaces"][v["bf_begin"]:v["bf_end"]])
        if v["grid"] != abi.DPROP_INVALID_INDEX:
            g = t["grids"][v["grid"]]
            n = int(g["n_bins"][0]) * int(g["n_bins"][1])
            bins = t["grid_bins"][g["bin_offset"]:g["bin_offset"] + n]
            own += sorted(set(bins[bins != abi.DPROP_INVALID_INDEX].tolist()))
            v["grid"] = abi.DPROP_INVALID_INDEX
        v["bf_begin"], v["bf_end"] = len(lists), len(lists) + len(own)
        lists += own
    t["bf_surfaces"] = np.array(lists, np.uint32)
    t["grids"] = t["grids"][:0]
    t["grid_bins"] = t["grid_bins"][:0]
    return t


def test_requested_order_is_kept(rules):
    """A requested direction order is only left out for short lists, small
    batches and direct results."""
    tele = rules.load("telescope_10x1m_300um")
    assert rules.drops_order(tele, 0, 10000)
    assert not rules.drops_order(tele, 1, 20000)
    assert not rules.drops_order(tele, 0, 40000)
    toy = rules.load("toy_4brl_7edc")
    assert not rules.drops_order(toy, 0, 10000)
    lists = _grids_as_lists(toy, rules.abi)
    for n in (3000, 14000, 300000):
        assert not rules.drops_order(lists, 0, n)


def test_default_tail_fits_the_warp_per_track_kernel(rules):
    """What is left after the last round by default is no more than the kernel
    with a warp per track takes (8192 tracks), at any batch size."""
    assert rules.tail(0) == 0 and rules.tail(64) == 1
    assert rules.tail(200000) == 3125 and rules.tail(524287) == 8191
    for n in (524288, 524352, 1000000, 2000000, 2**31 - 1):
        assert rules.tail(n) == 8192


@pytest.mark.parametrize("n", [1, 3, 63, 64, 65, 1000, 4097])
@pytest.mark.parametrize("max_records", [0, 1, 7, 16, 32])
def test_host_scratch_holds_every_array(rules, n, max_records):
    """The arrays of a host call, each from a 256-byte boundary on."""
    r = n * max_records
    sizes = ([8 * n] * 8 + [n] + [4 * n] * (6 + 1 + 8)
             + [8 * r] + [4 * r] * (6 + 21 + 1) + [r])
    end = 0
    for s in sizes:
        end += -(-s // 256) * 256
    assert rules.host_scratch(n, max_records) >= end


def test_scan_of_few_tracks(rules):
    """Few tracks of a detector whose surfaces the truth scan cannot skip."""
    wire = rules.load("wire_chamber_10l_cells")
    assert rules.scan_clusters(wire, 1) and rules.scan_clusters(wire, 100)
    assert not rules.scan_clusters(wire, 1000)
    assert not rules.scan_clusters(rules.load("toy_4brl_7edc"), 1)
    assert not rules.scan_clusters(rules.load("telescope_10x1m_300um"), 1)


def test_narrow_windows(rules):
    """With a window of one bin the searches are a small part of a track: the
    warp-per-track form ends earlier, and 32 registers do not pay."""
    toy, maps, wire, tele = (rules.load(x) for x in (
        "toy_4brl_7edc", "toy_4brl_7edc_maps", "wire_chamber_10l_cells",
        "telescope_10x1m_300um"))
    assert 2500 <= rules(toy, 0, 0, 0)["group"] <= 4000
    assert rules(maps, 1, 0, 0)["group"] <= 2200
    assert rules(maps, 1, 0, 1)["group"] <= 2500
    assert rules(wire, 1, 0, 0)["group"] <= 5000
    assert rules(toy, 0, 0, 0)["group64"] <= 2200
    assert rules(maps, 1, 0, 0)["group64"] <= 1600
    # a detector without grids has no window
    assert rules(tele, 0, 0, 0) == rules(tele, 0, 0, 3)
    assert rules(toy, 0, 0, 2**32 - 1) == rules(toy, 0, 0, 3)
    for tables, extra in ((toy, 0), (maps, 1), (wire, 1)):
        assert rules.budget(tables, extra, 1, 3000, window=0) == 8
