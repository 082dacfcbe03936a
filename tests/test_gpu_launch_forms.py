"""Open launch shapes of detectors with material maps, volume material and
wires, on both sides of the batch sizes where the form changes, against one
thread per track (a spelled-out shape)."""
import pytest

from tests.gpu_forms import assert_same, config, detector, run, sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,precision,sizes", [
    ("maps", 4, (1, 4096, 4097)), ("maps", 8, (33, 3072, 3073)),
    ("telescope+material", 4, (31, 1536, 1537)),
    ("telescope+material", 8, (1, 1184, 1185)),
    ("wire", 4, (8192, 8193)), ("straw", 4, (4097,)),
    ("wire", 8, (5120, 5121)),
])
def test_forms_agree(name, precision, sizes):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from detray_b200 import propagator
    from detray_b200.units import T
    det = detector(name)
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    cfg = config(name)
    dev = torch.tensor(sample(name, max(sizes)), device="cuda",
                       dtype=torch.float64 if precision == 8
                       else torch.float32)
    for n in sizes:
        part = dev[:, :n].contiguous()
        a = run(det, field, cfg, part, ctas_per_sm=8)
        for kw in (dict(), dict(sort_tracks=1),
                   dict(sort_tracks=1, method=1)):
            assert_same(a, run(det, field, cfg, part, **kw), (n, kw))


def test_wide_window_off_the_grid():
    """Tracks along the discs of an endcap never reach its grid's reference
    plane: their bin lies far outside, and a window of 700 bins around it must
    not wrap into an empty range that takes the portals along with it (the
    warp-per-track form deals portals and bins out in one row)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import numpy as np
    from detray_b200 import abi, propagator
    from detray_b200.units import T
    det = detector("toy")
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    cfg = abi.make_config(max_records=16, search_window=(700, 700))
    trk = np.zeros((8, 20))
    trk[0] = 60.0
    trk[2] = np.linspace(610.0, 1400.0, 20)
    trk[4] = 1.0
    trk[7] = 1e-4
    dev = torch.tensor(trk, dtype=torch.float32, device="cuda")
    a = run(det, field, cfg, dev, ctas_per_sm=8)
    assert (a["status"] == abi.TRK_EXITED).all()
    assert_same(a, run(det, field, cfg, dev), "window")
