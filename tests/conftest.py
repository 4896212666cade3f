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
def kernels_of():
    """kernels_of(call): the kernels that the call launches, by capturing it: dicts of name (as linked), the numbers among
    its template arguments, grid, block, registers per thread."""
    import ctypes as C
    import re

    import torch

    class Params(C.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
        _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("smem", C.c_uint),
                    ("args", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]

    def run(call):
        driver = C.CDLL("libcuda.so.1")

        def check(rc):
            assert rc == 0, f"CUDA driver error {rc}"

        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            kept = call()  # noqa: F841
        handle, count = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t()
        check(driver.cuGraphGetNodes(handle, None, C.byref(count)))
        nodes = (C.c_void_p * count.value)()
        check(driver.cuGraphGetNodes(handle, nodes, C.byref(count)))
        out = []
        for node in nodes:
            kind = C.c_int()
            check(driver.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
            if kind.value != 0:  # CU_GRAPH_NODE_TYPE_KERNEL
                continue
            p, func, name, registers = Params(), C.c_void_p(), C.c_char_p(), C.c_int()
            check(driver.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)))
            func.value = p.func
            if not p.func:
                check(driver.cuKernelGetFunction(C.byref(func), C.c_void_p(p.kern)))
            check(driver.cuFuncGetName(C.byref(name), func))
            check(driver.cuFuncGetAttribute(C.byref(registers), 4, func))  # CU_FUNC_ATTRIBUTE_NUM_REGS
            text = name.value.decode()
            out.append({"name": text, "arguments": [int(x) for x in re.findall(r"L[ib](\d+)E", text)], "grid": p.grid[0],
                        "block": p.block[0], "registers": registers.value})
        return out

    return run
