import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def oracle_mod():
    """The CPU checker (oracle/), built on first use."""
    from oracle import build_oracle

    build_oracle.build_oracle()
    from oracle import oracle

    return oracle


@pytest.fixture(scope="session")
def cuda_lib():
    """The CUDA library behind the C ABI; GPU tests fail loudly if it is missing."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hades_b200 import _lib

    lib = _lib.load()
    yield lib
    assert _lib.device_status() == 0, "a kernel recorded a device-side error"


GOLDEN = ROOT / "tests" / "golden"


@pytest.fixture
def kernels_of(tmp_path):
    """kernels_of(call): the kernels that the call launches, as the profiler names them: dicts of name, grid, block,
    registers per thread, in the order of their start."""
    import json

    import torch
    from torch.profiler import ProfilerActivity, profile

    def run(call):
        call()
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        prof.export_chrome_trace(str(tmp_path / "trace.json"))
        events = [e for e in json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
                  if e.get("cat") == "kernel" and "grid" in e.get("args", {})]
        if not events:
            pytest.skip("the profiler reports no kernels here")
        return [{"name": e["name"].replace("(anonymous namespace)::", ""), "grid": e["args"]["grid"][0],
                 "block": e["args"]["block"][0], "registers": e["args"]["registers per thread"]}
                for e in sorted(events, key=lambda e: e["ts"])]

    return run
