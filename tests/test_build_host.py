"""The library's device code is linked unpacked: a module that nvcc compressed is unpacked
within the first call that uses it (11 ms of the first PhotonMap frame of a process)."""
import subprocess

from renderx_gb300 import build


def test_device_code_is_not_compressed(monkeypatch):
    cmds = []

    def run(cmd, **kw):
        cmds.append(cmd)
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build.subprocess, "run", run)
    build._compile("x.cu", False)
    assert "--compress-mode=none" in cmds[0] and "-c" in cmds[0]
