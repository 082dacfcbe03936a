"""The host build of the core with traps on undefined behaviour (references
bound to null, signed overflow): propagations whose inputs reach the corners
run through."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from detray_b200 import build
    out = tmp_path_factory.mktemp("ub") / "libcore_ub.so"
    inc = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared",
                    "-fsanitize=null,signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error",
                    f"-I{REPO / 'include'}", f"-I{build.CSRC}", f"-I{inc}",
                    str(REPO / "tests" / "native" / "core_host.cpp"),
                    "-o", str(out)], check=True)
    return out


CHILD = """
import sys
sys.path.insert(0, {repo!r})
from tests.test_core_sanitized import child
child({lib!r}, {case!r}, {precision})
"""


def _case(case):
    from detray_b200 import abi, geometry, tracks
    if case == "telescope":  # a detector without any grid
        return (geometry.load_geometry("telescope_10x1m_300um"),
                tracks.telescope_tracks(50, seed=1),
                abi.make_config(max_records=16))
    # tracks along the discs of an endcap: the grid's reference plane is not
    # reached, and the wide window starts from a bin far outside
    trk = tracks.toy_tracks(20, seed=2)
    trk[0:2] = 0.0
    trk[0] = 60.0
    trk[2] = np.linspace(610.0, 1400.0, 20)
    trk[4:7] = 0.0
    trk[4] = 1.0
    trk[7] = 1e-4
    return (geometry.load_geometry("toy_4brl_7edc"), trk,
            abi.make_config(max_records=16, search_window=(700, 700)))


def child(path, case, precision):
    from detray_b200 import abi, geometry
    lib = C.CDLL(path)
    tables, trk, cfg = _case(case)
    det = geometry.Descriptor(tables)
    n = trk.shape[1]
    trk = np.ascontiguousarray(trk, dtype=np.float64)
    status = np.zeros(n, np.uint8)
    r = abi.Results()
    r.status = status.ctypes.data
    ptrs = (C.c_void_p * 8)(*[trk[i].ctypes.data for i in range(8)])
    b = (C.c_double * 3)(0.0, 0.0, 2.0 * 0.000299792458)
    rc = lib.core_host_propagate(precision, C.byref(det.desc), 0, b, None,
                                 None, None, None, C.byref(cfg), ptrs,
                                 C.c_uint64(n), C.byref(r))
    sys.exit(0 if rc == 0 else 3)


@pytest.mark.parametrize("case", ["telescope", "along_discs"])
@pytest.mark.parametrize("precision", [4, 8])
def test_no_undefined_behaviour(lib, case, precision):
    p = subprocess.run([sys.executable, "-c",
                        CHILD.format(repo=str(REPO), lib=str(lib), case=case,
                                     precision=precision)],
                       cwd=REPO, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-500:]
