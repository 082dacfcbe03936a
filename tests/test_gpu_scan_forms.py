"""The truth scan's forms - a cluster of CTAs per track for few tracks of a wire
chamber, one warp per track for a handful of surfaces - give the hits of one
CTA per track, bit for bit: the same tracks in a batch above the line, or
beside copies of themselves."""
import numpy as np
import pytest

from tests.gpu_forms import detector, sample

pytestmark = pytest.mark.gpu


def _scan(torch, det, b, trk, capacity):
    from detray_b200 import propagator
    r = propagator.helix_scan(det, b, trk, 1e-3, capacity)
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in r.items() if not k.startswith("_")}


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("name", ["wire", "straw"])
def test_cluster_per_track(name, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from detray_b200.units import T
    det = detector(name)
    b = (0.3 * T, 0.0, 1.8 * T)
    trk = torch.tensor(sample(name, 500), device="cuda",
                       dtype=torch.float64 if precision == 8
                       else torch.float32)
    # a capacity no track exceeds, one that most do
    for capacity in (128, 6):
        want = _scan(torch, det, b, trk, capacity)
        assert want["n_hits"].max() > 6
        for n in (1, 3, 192, 193):
            got = _scan(torch, det, b, trk[:, :n].contiguous(), capacity)
            for k in ("status", "n_hits"):
                assert np.array_equal(got[k], want[k][:n]), (n, k)
            # (the hits of a track above the capacity are unsorted)
            stored = ((np.arange(capacity)[:, None] < got["n_hits"][None, :])
                      & (got["status"] == 0)[None, :])
            for k in ("barcode", "path", "loc0", "loc1", "volume_link"):
                assert np.array_equal(got[k][stored],
                                      want[k][:, :n][stored]), (n, k)


@pytest.mark.parametrize("precision", [4, 8])
def test_few_surfaces_against_the_host(precision, core_host):
    """The telescope's 16 surfaces against the host build of the search (in
    double; a few um in single precision)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ctypes as C
    from detray_b200 import geometry
    from detray_b200.units import T
    tables = geometry.load_geometry("telescope_10x1m_300um")
    b = (0.0, 0.0, 2.0 * T)
    n, cap = 300, 32
    trk = np.ascontiguousarray(sample("telescope", n), dtype=np.float64)
    if precision == 4:
        trk = np.ascontiguousarray(trk.astype(np.float32).astype(np.float64))
    got = _scan(torch, detector("telescope"), b,
                torch.tensor(trk, device="cuda", dtype=torch.float64
                             if precision == 8 else torch.float32), cap)
    desc = geometry.Descriptor(tables)
    want = {"status": np.zeros(n, np.uint8), "n_hits": np.zeros(n, np.uint32),
            "barcode": np.zeros((cap, n), np.uint64),
            "path": np.zeros((cap, n)), "loc0": np.zeros((cap, n)),
            "loc1": np.zeros((cap, n)),
            "volume_link": np.zeros((cap, n), np.uint16)}
    ptrs = (C.c_void_p * 8)(*[trk[i].ctypes.data for i in range(8)])
    assert core_host.core_host_helix_scan(
        C.byref(desc.desc), (C.c_double * 3)(*b), ptrs, C.c_uint64(n),
        C.c_double(1e-3), C.c_uint32(cap),
        *[C.c_void_p(want[k].ctypes.data) for k in
          ("status", "n_hits", "barcode", "path", "loc0", "loc1",
           "volume_link")]) == 0
    assert want["n_hits"].mean() > 5
    same = ((got["status"] == want["status"])
            & (got["n_hits"].view(np.uint32) == want["n_hits"]))
    stored = np.arange(cap)[:, None] < np.where(same, want["n_hits"], 0)
    differ = (got["barcode"].view(np.uint64) != want["barcode"]) & stored
    same &= ~differ.any(axis=0)
    # single precision may see a track at a mask's edge differently
    assert same.mean() >= (1.0 if precision == 8 else 0.995)
    stored &= same[None, :]
    for k in ("path", "loc0", "loc1"):
        assert np.abs(got[k][stored] - want[k][stored]).max() <= (
            1e-6 if precision == 8 else 5e-2), k
