"""First calls from several threads at once, in a fresh process."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys, threading
sys.path.insert(0, sys.argv[1])
import torch
from fdk import models, native

rows = [17, 33, 65, 97, 129, 161, 193, 257]  # batch tiles, and so shared-memory plans, of their own
k, n = 512, 640
gen = torch.Generator(device="cuda").manual_seed(0)
layer = models.QuantisedLinear.create(torch.randn((n, k), generator=gen, device="cuda").bfloat16(), models.QuantisationConfig(4, 64))
dense = native.dequantise(layer.weight_data, layer.lut, layer.scale, 4).double()
layer.tiled(), layer.lut_bytes()
xs = [torch.randn((m, k), generator=gen, device="cuda").bfloat16() for m in rows]
torch.cuda.synchronize()
start, failures = threading.Barrier(len(rows)), []

def calls(x):
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            native.workspace(x.device)
            start.wait()
            outs = [layer(x) for _ in range(20)]
            torch.cuda.current_stream().synchronize()
            assert native.device_status() == 0
        want = x.double() @ dense.t()
        assert all(torch.equal(y, outs[0]) for y in outs)
        assert ((outs[0].double() - want).norm() / want.norm()).item() < 2.0**-9 + 1e-5  # one rounding to bf16
    except BaseException as error:
        failures.append(repr(error))
        start.abort()

threads = [threading.Thread(target=calls, args=(x,)) for x in xs]
[t.start() for t in threads]
[t.join() for t in threads]
sys.exit(repr(failures) if failures else 0)
"""


def test_first_calls_from_several_threads():
    """The kernels' shared-memory limit is set by whoever comes first, to a value that suits every later call."""
    package = Path(__file__).resolve().parents[1] / "fused-dequantisation-kernels_b200"
    done = subprocess.run([sys.executable, "-c", SCRIPT, str(package)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
