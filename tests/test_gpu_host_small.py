"""Host calls of a few tracks: every array of the call's device scratch has
its room (each starts on a 256-byte boundary, which is most of the scratch for
one track), and the results are the device call's."""
import numpy as np
import pytest

from tests.gpu_forms import config, detector, run, sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 65, 1000])
@pytest.mark.parametrize("max_records", [1, 16])
def test_small_host_call(n, max_records):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from detray_b200 import propagator
    from detray_b200.units import T
    propagator.release_cache()
    det = detector("toy")
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    cfg = config("toy", max_records=max_records)
    # float values, so that the device call starts from the same numbers
    trk = sample("toy", n).astype(np.float32)
    got = propagator.propagate_host(cfg, det, field, trk.astype(np.float64))
    want = run(det, field, cfg, torch.tensor(trk, device="cuda"))
    for k in ("status", "n_records", "n_steps", "n_trials", "n_intersections",
              "n_transports", "n_material", "path_length", "final_free"):
        assert got[k].tobytes() == want[k].tobytes(), k
    stored = np.arange(max_records)[:, None] < got["n_records"][None, :]
    for k in ("rec_barcode", "rec_path", "rec_flags"):
        assert np.array_equal(got[k][stored], want[k][stored]), k
    for k in ("rec_bound", "rec_cov"):
        assert np.array_equal(got[k][:, stored], want[k][:, stored]), k
