"""The autotuner knows the form a launch without a shape takes: for a small
event that is a warp per track, several times faster than any spelled-out
shape (300 toy tracks: 0.35 against 1.8 ms)."""
import pytest

from tests.gpu_forms import config, detector, run, sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
def test_small_event(graph):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from detray_b200 import propagator
    from detray_b200.units import T
    det = detector("toy")
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    cfg = config("toy")
    dev = torch.tensor(sample("toy", 300), device="cuda",
                       dtype=torch.float32)
    lc, times = propagator.autotune(cfg, det, field, dev, use_graph=graph)
    assert lc.by_size == 1
    assert min(times) == times[1]
    want = run(det, field, cfg, dev)
    res = propagator.alloc_device_results(300, cfg.max_records, "cuda")
    for t in res.tensors.values():
        t.zero_()
    propagator.propagate(cfg, det, field, dev, results=res, launch=lc)
    torch.cuda.synchronize()
    for k, v in res.tensors.items():
        got = v.cpu().numpy()
        assert got.tobytes() == want[k].tobytes(), k
    propagator.release_cache()
