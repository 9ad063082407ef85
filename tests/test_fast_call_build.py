"""csrc/fast_call.cpp is built for one Python and one torch and is optional: a file built for others is not loaded, a build that fails is a warning,
and importing the operators maps nothing."""
import os
import subprocess
import sys

import pytest
import torch

from qspec_b200 import build, ops


def test_path_names_what_it_is_built_for(monkeypatch):
    here = build.fast_path()
    assert torch.__version__ in here and f"{sys.version_info[0]}{sys.version_info[1]}" in here
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.fast_path() != here


def test_file_for_another_torch_is_not_loaded(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "OUT_DIR", str(tmp_path))
    monkeypatch.setattr(ops, "_fast", False)
    (tmp_path / os.path.basename(build.fast_path())).write_bytes(b"no library")         # the right name, but not a library: the ordinary way
    assert ops._load_fast() is None
    (tmp_path / os.path.basename(build.fast_path())).unlink()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    (tmp_path / os.path.basename(build.fast_path())).write_bytes(b"no library")
    monkeypatch.undo()
    monkeypatch.setattr(build, "OUT_DIR", str(tmp_path))
    monkeypatch.setattr(ops, "_fast", False)
    assert ops._load_fast() is None                                                      # only a file of another torch lies there


def test_rebuilt_when_the_header_is_newer(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "OUT_DIR", str(tmp_path))
    path = build.fast_path()
    open(path, "w").close()
    ran = []
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: ran.append(a) or subprocess.CompletedProcess(a, 1, "", "no compiler"))
    assert build.build_fast() == path and not ran                                        # newer than its sources
    header = os.path.getmtime(os.path.join(build.HERE, "..", "include", "qspec_b200.h"))
    os.utime(path, (header - 10, header - 10))
    with pytest.raises(RuntimeError):
        build.build_fast()
    assert ran


def test_failed_build_is_a_warning(monkeypatch):
    def fail(force=False):
        raise RuntimeError("no g++")
    monkeypatch.setattr(build, "build_fast", fail)
    with pytest.warns(UserWarning, match="no g\\+\\+"):
        build.build_fast_if_possible()
    if os.path.exists(build.LIB_PATH):
        with pytest.warns(UserWarning, match="no g\\+\\+"):
            assert build.build_library() == build.LIB_PATH


def test_import_maps_nothing():
    code = "import qspec_b200.ops; print(any('_fast' in line or 'libqspec' in line for line in open('/proc/self/maps')))"
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=build.HERE + "/..", timeout=300)
    assert run.stdout.strip() == "False", run.stdout + run.stderr


@pytest.mark.gpu
def test_built_path_is_loaded_by_the_first_call():
    if not os.path.exists(build.fast_path()):
        pytest.skip("csrc/fast_call.cpp is not built")
    w = torch.zeros(32, 64, dtype=torch.int8, device="cuda")
    x, s = torch.ones(1, 128, dtype=torch.float16, device="cuda"), torch.ones(32, dtype=torch.float16, device="cuda")
    for _ in range(2):                                                                   # the first call has no workspace yet
        ops.gemm_w4a16(x, w, s, None, torch.empty(1, 32, dtype=torch.float16, device="cuda"))
    assert hasattr(ops._fast, "linear")
