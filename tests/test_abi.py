"""The C-ABI library loads without a GPU and exports every symbol that include/*.h declares;
the ctypes prototype table covers the same set."""
import ctypes
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def declared_symbols():
    names = set()
    for h in (ROOT / "include").glob("*.h"):
        text = re.sub(r"/\*.*?\*/", "", h.read_text(), flags=re.S)
        names |= set(re.findall(r"\b(hb_[a-z0-9_]+)\s*\(", text))
    return names


@pytest.fixture(scope="module")
def built_lib():
    from hades_b200 import _build

    return _build.build()


def test_header_symbols_exported(built_lib):
    lib = ctypes.CDLL(str(built_lib))
    names = declared_symbols()
    assert len(names) > 30
    missing = [n for n in sorted(names) if not hasattr(lib, n)]
    assert not missing, f"declared in include/*.h but not exported: {missing}"


def test_prototype_table_matches_header(built_lib):
    from hades_b200 import _lib

    assert set(_lib.PROTOTYPES) == declared_symbols()
    _lib.load()  # binds every prototype; raises if one is absent


def test_no_gpu_calls_return_status_not_crash(built_lib):
    from hades_b200 import _lib

    lib = _lib.load()
    assert lib.hb_version() >= 100
    # argument validation happens before any CUDA work
    rc = lib.hb_rows_gather(None, None, None, None, 5, 16, 8, 0, None)
    assert rc == 1 and b"null" in lib.hb_last_error()
    rc = lib.hb_rows_gather(None, None, None, None, 0, 16, 3, 0, None)
    assert rc == 1
    assert lib.hb_index_size(None) == -1


@pytest.mark.parametrize("kind,change,why", [
    (0, {"emb_elem_bytes": 8}, b"fp32 (4) or fp16 (2)"), (1, {"emb_elem_bytes": 8}, b"fp32 (4) or fp16 (2)"),
    (0, {"s1": None}, b"optimiser description"), (0, {"step": None}, b"optimiser description"),
    (1, {"id_stride": 0}, b"optimiser description"), (1, {"rows": 0}, b"optimiser description"),
    (2, {}, b"unknown optimiser")])
def test_step_refuses_what_the_updates_refuse(built_lib, kind, change, why):
    """The description is checked before anything that it points to is looked at (addresses here are made up)."""
    from hades_b200 import _lib

    lib = _lib.load()
    d = _lib.StepDesc()
    d.index = d.cache_rows = d.table = d.class_table = 256
    d.staging = _lib.StagingDesc(256, 256, 256, 256, 256, 8, 4)
    d.row_bytes, d.dim, d.table_rows, d.class_len = 16, 4, 100, 100
    d.opt = _lib.OptimDesc(kind, 4, 256, 256, 256, 256, 0, 1, 100, 0.01, 0.9, 0.999, 1e-8)
    for k, v in change.items():
        setattr(d.opt, k, v)
    assert lib.hb_step_supported(ctypes.byref(d)) == 0 and why in lib.hb_last_error()


@pytest.mark.parametrize("peer", [0, 1])
@pytest.mark.parametrize("maintain", [0, 1])
def test_expansion_of_full_lists_holds_its_rows_in_registers(built_lib, peer, maintain):
    """runs_expand_kernel for rows of 512 bytes, 32 entries a warp: eight rows in flight and no spills."""
    from hades_b200 import _build

    log = _build.OBJ / "runs.ptxas"
    if not log.exists():
        pytest.skip("the objects were built elsewhere")
    name = f"runs_expand_kernelILb{peer}ELi512ELb{maintain}ELb1E"
    if peer and maintain:
        assert name not in log.read_text()  # several GPUs: maintenance has launches of its own
        return
    entry = log.read_text().split(name, 1)[1].split("Compiling entry function", 1)[0]
    assert " 0 bytes spill stores, 0 bytes spill loads" in entry, entry[:600]


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from hades_b200 import _lib

    monkeypatch.setattr(_lib, "_LIB", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "nope.so")
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        _lib.load()


def test_reference_side_bridge_compiles():
    """hades_b200/bridge/hades_b200_bridge.cc (the translation unit a maintainer of the reference
    adds beside src/pybind.cc) compiles against the torch headers and include/hades_b200.h."""
    import shutil
    import subprocess
    import sysconfig
    from pathlib import Path

    import torch

    root = Path(__file__).resolve().parent.parent
    tdir = Path(torch.__file__).parent
    gxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else shutil.which("g++")
    cmd = [gxx, "-std=c++17", "-fsyntax-only", str(root / "hades_b200" / "bridge" / "hades_b200_bridge.cc"),
           "-I", str(root / "include"), "-I", str(tdir / "include"),
           "-I", str(tdir / "include/torch/csrc/api/include"), "-I", sysconfig.get_paths()["include"],
           "-I", "/usr/local/cuda/include"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
