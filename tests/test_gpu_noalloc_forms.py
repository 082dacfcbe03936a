"""dprop_propagate_noalloc takes no device memory after the first call on the
device, whatever form later batches, detectors and configurations take.  In a
process of its own: the driver loads a kernel's code, and reserves its local
memory, once per process."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

REPO = Path(__file__).resolve().parents[1]


def child():
    import ctypes as C

    import torch

    from detray_b200 import abi, fields, propagator
    from detray_b200.units import T
    from tests.gpu_forms import config, detector, sample
    lib = propagator.load_library()
    lib.dprop_propagate_noalloc.argtypes = [
        C.POINTER(abi.Config), C.c_void_p, C.c_void_p, C.POINTER(abi.Tracks),
        C.POINTER(abi.Results), C.c_uint64, C.c_void_p]
    dets = {k: detector(k) for k in ("toy", "wire", "telescope")}
    const = propagator.Field.constant((0.0, 0.0, 2.0 * T))
    fmap = propagator.Field.grid(fields.solenoid_map())
    stream = torch.cuda.current_stream()

    def call(name, field, n, gradient=0):
        cfg = config(name, max_records=8, use_field_gradient=gradient)
        trk = torch.tensor(sample(name, n), dtype=torch.float32,
                           device="cuda")
        res = propagator.alloc_device_results(n, 8, "cuda")
        ts = propagator.tracks_struct(trk)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        assert lib.dprop_propagate_noalloc(
            C.byref(cfg), dets[name].handle, field.handle, C.byref(ts),
            C.byref(res.struct), n, C.c_void_p(stream.cuda_stream)) == 0
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]

    call("toy", const, 10000)  # the first call
    grown = {}
    for name in dets:
        for n in (1, 2000, 2500, 3500, 10000, 60000, 100000, 230000):
            for field in (const, fmap):
                key = (name, n, field is fmap)
                grown[key] = call(name, field, n)
        grown[(name, "gradient")] = call(name, fmap, 20000, 1)
    bad = {k: v for k, v in grown.items() if v}
    assert not bad, bad


def test_later_forms_take_no_memory():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = subprocess.run([sys.executable, "-c", "import sys; sys.path.insert(0, "
                        f"{str(REPO)!r}); from tests.test_gpu_noalloc_forms "
                        "import child; child()"], cwd=REPO,
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-1500:]
