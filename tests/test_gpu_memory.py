"""Device memory the library keeps between calls: what is optional gives way
to what a call needs."""
import pytest

pytestmark = pytest.mark.gpu

GB = 1 << 30


@pytest.fixture
def setup():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from detray_b200 import geometry, propagator
    from detray_b200.units import T
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    propagator.release_cache()
    det = propagator.Detector(geometry.load_geometry("toy_4brl_7edc"))
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    yield torch, det, field
    propagator.release_cache()
    torch.cuda.empty_cache()


def _device_tracks(torch, n, seed):
    from detray_b200 import tracks
    return torch.tensor(tracks.toy_tracks(n, seed=seed), dtype=torch.float32,
                        device="cuda")


def _fill(torch, leave):
    """Take all device memory but ``leave`` bytes."""
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("graph", [0, 1])
def test_staging_area_gives_way(setup, graph):
    """A persistent call whose slots fit only where a sorted plain call left
    its staging area (300 000 x 32 records of 128 bytes: 1.2 GB)."""
    torch, det, field = setup
    from detray_b200 import abi, propagator
    cfg = abi.make_config(max_records=32, search_window=(3, 3))
    trk = _device_tracks(torch, 300000, 41)
    res = propagator.alloc_device_results(300000, 32, "cuda")
    few = trk[:, :150000].contiguous()
    rounds = propagator.make_launch(method=abi.METHOD_PERSISTENT,
                                    ctas_per_sm=3, use_graph=graph)
    propagator.propagate(cfg, det, field, few, results=res, launch=rounds)
    torch.cuda.synchronize()
    want = res.tensors["n_steps"][:150000].clone()
    propagator.release_cache()
    propagator.propagate(cfg, det, field, trk, results=res,
                         launch=propagator.make_launch(sort_tracks=1))
    torch.cuda.synchronize()
    # the slots and staged rows take 0.7 GB
    filled = _fill(torch, GB // 2)
    res.tensors["n_steps"].zero_()
    propagator.propagate(cfg, det, field, few, results=res, launch=rounds)
    torch.cuda.synchronize()
    del filled
    assert torch.equal(res.tensors["n_steps"][:150000], want)


def test_host_pipeline_without_room_for_staging(setup):
    """Jagged host call of 120 000 tracks, 64 records each: four chunks of
    32 768 take 0.51 GB each, 0.78 GB with staging."""
    torch, det, field = setup
    import numpy as np
    from detray_b200 import abi, propagator, tracks
    cfg = abi.make_config(max_records=64, search_window=(3, 3))
    trk = tracks.toy_tracks(120000, seed=42)
    launch = propagator.make_launch(sort_tracks=1)

    def run():
        return propagator.propagate_host(cfg, det, field, trk, launch=launch,
                                         jagged=True)

    want = run()
    propagator.release_cache()
    filled = _fill(torch, int(2.5 * GB))
    got = run()
    del filled
    total = int(want["rec_offsets"][-1])
    assert total == int(got["rec_offsets"][-1])
    for k in ("status", "n_records", "n_steps", "rec_offsets"):
        assert np.array_equal(want[k], got[k]), k
    assert np.array_equal(want["rec_barcode"][:total],
                          got["rec_barcode"][:total])
    assert np.array_equal(want["rec_bound"][:, :total].view(np.uint32),
                          got["rec_bound"][:, :total].view(np.uint32))


def test_graphs_share_a_bound_on_staging(setup):
    """Cached graphs of sorted plain calls own their staging areas (here 3.1 GB
    each): together they hold at most 8 GiB, the next ones write directly."""
    torch, det, field = setup
    from detray_b200 import abi, propagator
    cfg = abi.make_config(max_records=24, search_window=(3, 3))
    n = 1000000
    trk = _device_tracks(torch, n, 43)
    launch = propagator.make_launch(sort_tracks=1, use_graph=1)
    res = propagator.alloc_device_results(n, 24, "cuda")
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    steps = []
    for k in range(4):
        # another number of tracks is another graph
        m = n - 32 * k
        sub = trk[:, :m].contiguous()
        propagator.propagate(cfg, det, field, sub, results=res, launch=launch)
        torch.cuda.synchronize()
        steps.append(res.tensors["n_steps"][:n - 96].clone())
        del sub
    torch.cuda.empty_cache()
    left, _ = torch.cuda.mem_get_info()
    assert free - left < 9 * GB
    for s in steps[1:]:
        assert torch.equal(s, steps[0])
