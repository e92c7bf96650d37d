import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "sponge2.0_b200"))
sys.path.insert(0, os.path.join(ROOT, "oracle"))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


@pytest.fixture(scope="session")
def oracle():
    if not os.path.exists(os.path.join(ROOT, "oracle", "libspgnb_oracle.so")):
        subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle")], check=True)
    import oracle as O
    return O.Oracle()


def rel_rms(a, b):
    import numpy as np
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.sqrt(((a - b) ** 2).sum(axis=-1).mean()) / np.sqrt((b ** 2).sum(axis=-1).mean()))


@pytest.fixture(scope="session")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def kernel_launches(torch, fn):
    """The GPU kernels fn() runs, in order: {name, grid, block, shared} each.
    For a process of its own (in_fresh_process): the tracer loses the first
    kernels of a profile late in a long test run."""
    import json
    import tempfile
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        prof.export_chrome_trace(path)
        with open(path) as f:
            events = json.load(f)["traceEvents"]
    kernels = sorted((e for e in events if e.get("cat") == "kernel"), key=lambda e: e["ts"])
    return [{"name": e["name"], "grid": e["args"]["grid"], "block": e["args"]["block"],
             "shared": e["args"]["shared memory"]} for e in kernels]


def in_fresh_process(module, function):
    """What the test module's function returns (JSON values) in a new process."""
    import json
    code = (f"import conftest, json, {module}\n"
            f"print('RESULT ' + json.dumps({module}.{function}()))")
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.abspath(__file__)),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return json.loads(r.stdout.split("RESULT ", 1)[1])
