"""Calls on several streams, and from several host threads, that share the
library's kept scratch (direction sort, persistent method, staged results):
each gets the results of a call made alone, bit for bit."""
import threading

import pytest

pytestmark = pytest.mark.gpu

N = 40000
FORMS = {
    "rounds": dict(method=1, ctas_per_sm=3),
    "rounds_sorted": dict(method=1, ctas_per_sm=3, sort_tracks=1),
    "plain_sorted": dict(sort_tracks=1),
}


@pytest.fixture(scope="module")
def setup():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from detray_b200 import abi, geometry, propagator, tracks
    from detray_b200.units import T
    det = propagator.Detector(geometry.load_geometry("toy_4brl_7edc"))
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    cfg = abi.make_config(max_records=24, search_window=(3, 3),
                          estimate_scattering_noise=0)
    trk = [torch.tensor(tracks.toy_tracks(N, seed=s), dtype=torch.float32,
                        device="cuda") for s in (31, 32)]

    def call(side, form, res, stream=None):
        propagator.propagate(cfg, det, field, trk[side], results=res,
                             launch=propagator.make_launch(**FORMS[form]),
                             stream=stream)

    def results():
        r = propagator.alloc_device_results(N, cfg.max_records, "cuda")
        for t in r.tensors.values():
            t.zero_()
        return r

    return torch, call, results


@pytest.mark.parametrize("threads", [False, True],
                         ids=["streams", "threads"])
@pytest.mark.parametrize("forms", [
    ("rounds", "plain_sorted"), ("plain_sorted", "plain_sorted"),
    ("rounds_sorted", "rounds_sorted"), ("rounds", "rounds")])
def test_overlapping_calls(setup, forms, threads):
    torch, call, results = setup
    alone, got, streams = [], [], []
    for side, form in enumerate(forms):
        r = results()
        call(side, form, r)
        torch.cuda.synchronize()
        alone.append(r)
        got.append([results() for _ in range(4)])
        streams.append(torch.cuda.Stream())
    torch.cuda.synchronize()

    def run(side):
        for r in got[side]:
            call(side, forms[side], r, streams[side])

    if threads:
        ts = [threading.Thread(target=run, args=(s,)) for s in (0, 1)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for k in range(4):
            for side in (0, 1):
                call(side, forms[side], got[side][k], streams[side])
    torch.cuda.synchronize()
    for side in (0, 1):
        for r in got[side]:
            for k, x in alone[side].tensors.items():
                assert torch.equal(x.view(torch.uint8),
                                   r.tensors[k].view(torch.uint8)), (side, k)


def test_captured_sorted_call(setup):
    """A sorted call captured into the caller's graph needs no more than the
    sort's scratch (a call with fewer records is enough of a warm-up), and
    its replays stay valid when a later call outgrows that."""
    torch, call, results = setup
    from detray_b200 import abi, geometry, propagator, tracks
    from detray_b200.units import T
    det = propagator.Detector(geometry.load_geometry("toy_4brl_7edc"))
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    launch = propagator.make_launch(sort_tracks=1)

    def run(n, max_records, res=None):
        cfg = abi.make_config(max_records=max_records, search_window=(3, 3),
                              estimate_scattering_noise=0)
        dev = torch.tensor(tracks.toy_tracks(n, seed=33), dtype=torch.float32,
                           device="cuda")
        if res is None:
            res = propagator.alloc_device_results(n, max_records, "cuda")
            for t in res.tensors.values():
                t.zero_()
        return lambda: propagator.propagate(cfg, det, field, dev, results=res,
                                            launch=launch), res

    propagator.release_cache()
    warm, _ = run(20000, 2)
    warm()
    torch.cuda.synchronize()
    captured, res = run(20000, 24)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured()
    larger, _ = run(200000, 32)
    larger()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    direct, want = run(20000, 24)
    direct()
    torch.cuda.synchronize()
    # direct stages its results, the captured call does not: the bits agree
    for k, x in want.tensors.items():
        assert torch.equal(x.view(torch.uint8),
                           res.tensors[k].view(torch.uint8)), k


@pytest.mark.parametrize("form", ["fp64_plain", "fp64_rounds", "adjoint"])
def test_overlapping_calls_of_the_other_kernels(setup, form):
    """Double precision and the adjoint keep their own sort scratch and
    slots: two streams, sorted calls in turn."""
    torch = setup[0]
    from detray_b200 import abi, adjoint, geometry, propagator, tracks
    from detray_b200.units import T
    det = propagator.Detector(geometry.load_geometry("toy_4brl_7edc"))
    field = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    cfg = abi.make_config(max_records=16, search_window=(3, 3),
                          estimate_scattering_noise=0)
    dtype = torch.float32 if form == "adjoint" else torch.float64
    shape = dict(method=1, ctas_per_sm=2) if form == "fp64_rounds" else {}
    launch = propagator.make_launch(
        sort_tracks=1, precision=8 if dtype == torch.float64 else 0, **shape)
    trk = [torch.tensor(tracks.toy_tracks(20000, seed=s), dtype=dtype,
                        device="cuda") for s in (35, 36)]

    def call(side, stream):
        with torch.cuda.stream(stream):
            if form == "adjoint":
                return adjoint.propagate_adjoint(cfg, det, field, trk[side],
                                                 launch).results.tensors
            return propagator.propagate(cfg, det, field, trk[side],
                                        launch=launch).tensors

    streams = [torch.cuda.Stream() for _ in trk]
    torch.cuda.synchronize()
    alone = []
    for side in (0, 1):
        alone.append(call(side, streams[side]))
        torch.cuda.synchronize()
    got = [(side, call(side, streams[side])) for _ in range(4)
           for side in (0, 1)]
    torch.cuda.synchronize()
    for side, b in got:
        a = alone[side]
        for k in ("status", "n_records", "n_steps", "n_trials",
                  "n_intersections"):
            assert torch.equal(a[k], b[k]), k
        for k in ("path_length", "final_free"):
            assert torch.equal(a[k].view(torch.uint8),
                               b[k].view(torch.uint8)), k
