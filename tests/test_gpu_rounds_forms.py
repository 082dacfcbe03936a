"""The round-based method with its shape spelled out (left open, a small batch
takes another form), and on both sides of the batch sizes from which it is
the open shape's form: against the plain kernel, one thread per track."""
import numpy as np
import pytest

from tests.gpu_forms import (DISCRETE, NUMBERS, assert_same, config, detector,
                             run, sample)

pytestmark = pytest.mark.gpu

ROUNDS = {4: dict(method=1, ctas_per_sm=3), 8: dict(method=1, ctas_per_sm=2)}


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _field(kind):
    from detray_b200 import fields, propagator
    from detray_b200.units import T
    if kind == "map":
        return propagator.Field.grid(fields.solenoid_map())
    return propagator.Field.constant((0.0, 0.0, 2.0 * T))


def _tensor(torch, trk, precision):
    return torch.tensor(trk, device="cuda", dtype=torch.float64
                        if precision == 8 else torch.float32)


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("name", ["toy", "wire"])
def test_ragged_batches(torch_cuda, name, precision):
    """Batch sizes around the warp, the CTA and the queue tile."""
    det, field, cfg = detector(name), _field("const"), config(name)
    trk = sample(name, 4097)
    for n in (1, 31, 32, 33, 127, 129, 4095, 4096, 4097):
        dev = _tensor(torch_cuda, np.ascontiguousarray(trk[:, :n]), precision)
        a = run(det, field, cfg, dev, ctas_per_sm=8)
        for kw in (dict(), dict(sort_tracks=1),
                   dict(sort_tracks=1, use_graph=1),
                   dict(sort_tracks=1, sort_interval=1),
                   dict(sort_tracks=1, tail_tracks=1)):
            assert_same(a, run(det, field, cfg, dev, **ROUNDS[precision],
                               **kw), (n, kw))


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("name,field", [
    ("toy", "map"), ("maps", "map"), ("straw", "const"),
    ("telescope", "const"), ("telescope+material", "const")])
def test_detectors(torch_cuda, name, field, precision):
    det, fld, cfg = detector(name), _field(field), config(name)
    dev = _tensor(torch_cuda, sample(name, 20000), precision)
    a = run(det, fld, cfg, dev, ctas_per_sm=8)
    for kw in (dict(), dict(sort_tracks=1)):
        assert_same(a, run(det, fld, cfg, dev, **ROUNDS[precision], **kw), kw)


@pytest.mark.parametrize("name,field,precision,line", [
    ("toy", "const", 4, 400000), ("toy", "map", 4, 150000),
    ("maps", "const", 4, 230000), ("wire", "const", 4, 16384),
    ("toy", "map", 8, 80000), ("wire", "const", 8, 25000)])
def test_open_shape_around_the_line(torch_cuda, name, field, precision, line):
    det, fld = detector(name), _field(field)
    cfg = config(name, max_records=8)
    dev = _tensor(torch_cuda, sample(name, line), precision)
    for n in (line - 1, line):
        part = dev[:, :n].contiguous()
        a = run(det, fld, cfg, part, ctas_per_sm=8)
        assert_same(a, run(det, fld, cfg, part, sort_tracks=1, method=1), n)


@pytest.mark.parametrize("n", [1, 4097, 70001])
@pytest.mark.parametrize("jagged", [True, False])
def test_host_buffers(torch_cuda, n, jagged):
    """Host tracks in double, fp32 arithmetic: one chunk, and three chunks
    whose rounds start one behind the other."""
    from detray_b200 import propagator
    det, field, cfg = detector("toy"), _field("const"), config("toy")
    trk = sample("toy", n).astype(np.float32)
    a = run(det, field, cfg, _tensor(torch_cuda, trk, 4), ctas_per_sm=8)
    for sort in (0, 1):
        b = propagator.propagate_host(
            cfg, det, field, trk.astype(np.float64),
            launch=propagator.make_launch(sort_tracks=sort, **ROUNDS[4]),
            jagged=jagged)
        stored = np.minimum(a["n_records"], cfg.max_records)
        keep = np.arange(cfg.max_records)[:, None] < stored[None, :]
        if jagged:
            off = b["rec_offsets"]
            assert np.array_equal(np.diff(off), stored)
            total = int(off[-1])

            def records(x):
                return x[..., :total]

            def wanted(x):
                # track by track
                return np.swapaxes(x, -1, -2)[..., keep.T]
        else:
            def records(x):
                return x[..., keep]
            wanted = records
        for k in DISCRETE:
            x, y = a[k], b[k]
            if k.startswith("rec_"):
                x, y = wanted(x), records(y)
            assert np.array_equal(x, y), (sort, k)
        for k in NUMBERS + ("rec_cov",):
            x, y = a[k], b[k]
            if k.startswith("rec_"):
                x, y = wanted(x), records(y)
            if k == "rec_cov":
                d = [i * (11 - i) // 2 + i for i in range(6)]
                sig = np.sqrt(np.abs(x[d]))
                i, j = np.triu_indices(6)
                assert (np.abs(x - y) <=
                        1e-3 * sig[i] * sig[j] + 1e-30).all(), (sort, k)
            else:
                assert np.allclose(x, y, rtol=1e-4, atol=2e-3), (sort, k)
