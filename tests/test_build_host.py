"""When the host module is built again, and that nothing ever sees half of it."""
import os
import subprocess

import pytest
import torch

from nsa_optim_b200.ops import build


@pytest.fixture
def runs(monkeypatch, tmp_path):
    """The commands of a build into a folder of its own, by a compiler that writes a line."""
    commands = []

    def run(cmd, **kw):
        commands.append(cmd)
        assert not os.path.samefile(os.path.dirname(cmd[cmd.index("-o") + 1]), tmp_path)      # not in the place of the finished file
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write(f"build {len(commands)}")
        return subprocess.CompletedProcess(cmd, len(commands) == 3, "", "")

    monkeypatch.setattr(build, "OBJ", str(tmp_path / "_build"))
    monkeypatch.setattr(build, "HOST", str(tmp_path / "_nsa_host.so"))
    monkeypatch.setattr(build, "nvcc_path", lambda: "/usr/local/cuda/bin/nvcc")
    monkeypatch.setattr(build.subprocess, "run", run)
    return commands


def test_built_again_for_another_pytorch(runs, monkeypatch, tmp_path):
    read = lambda: (tmp_path / "_nsa_host.so").read_text()                                 # noqa: E731
    build.build_host()
    build.build_host()
    assert len(runs) == 1 and read() == "build 1"
    monkeypatch.setattr(torch, "__version__", "0.0")
    build.build_host()
    build.build_host()
    assert len(runs) == 2 and read() == "build 2"
    with pytest.raises(RuntimeError):
        build.build_host(force=True)                     # a compiler that fails leaves the old one
    assert read() == "build 2" and sorted(os.listdir(tmp_path / "_build")) == ["_nsa_host.stamp"]
    monkeypatch.setattr(build.sys, "version", "another")
    build.build_host()
    assert len(runs) == 4 and read() == "build 4"
