"""What ``csrc/build.py`` compiles and where the package keeps it (no compiler and no GPU needed)."""

import fnmatch
import subprocess
import sysconfig
import tomllib
import warnings
from pathlib import Path

import pytest
import torch

from cornstarch_b200.csrc import build as B
from cornstarch_b200.ops import _native as nat


def test_every_source_is_packaged():
    """An installed copy builds its library from the sources that came with it."""
    meta = tomllib.loads((Path(__file__).resolve().parent.parent / "pyproject.toml").read_text())
    patterns = meta["tool"]["setuptools"]["package-data"]["cornstarch_b200.csrc"]
    for src in (*B.sources(), *B._headers(), B.HOST_OPS_SRC):
        assert any(fnmatch.fnmatch(src.name, p) for p in patterns), src.name


def test_host_module_belongs_to_one_torch_and_python():
    name = B.host_ops_path().name
    assert torch.__version__ in name and name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))


def test_host_module_is_compiled_for_this_torch(tmp_path, monkeypatch):
    """The ABI of torch's libraries, an output name that no other build uses, and nothing left behind where the compiler fails."""
    cmds, rc = [], 0

    def run(cmd, **kw):
        cmds.append(cmd)
        Path(cmd[cmd.index("-o") + 1]).write_text("")
        return subprocess.CompletedProcess(cmd, rc, "", "")

    path = tmp_path / B.host_ops_path().name
    monkeypatch.setattr(B, "host_ops_path", lambda: path)
    monkeypatch.setattr(B.subprocess, "run", run)
    monkeypatch.setattr(B, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    for _ in range(2):
        assert B.build_host_ops(force=True) == path and path.exists()
    assert all(f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}" in c for c in cmds)
    outs = [c[c.index("-o") + 1] for c in cmds]
    assert len({*outs, str(path)}) == 3
    rc = 1
    with pytest.raises(RuntimeError, match="host_ops.cpp"):
        B.build_host_ops(force=True)
    assert [p.name for p in tmp_path.iterdir()] == [path.name]


@pytest.mark.parametrize("broken", [False, True])
def test_without_a_host_module_calls_go_through_ctypes(tmp_path, monkeypatch, broken):
    path = tmp_path / B.host_ops_path().name
    if broken:
        path.write_text("not a shared object")
    monkeypatch.setattr(B, "host_ops_path", lambda: path)
    monkeypatch.setattr(nat, "_HOST", None)
    with pytest.warns(RuntimeWarning, match="csrc.build"):
        assert nat.host_ops() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert nat.host_ops() is None  # said once
