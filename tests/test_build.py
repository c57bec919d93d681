"""CPU: when the host extension, which is compiled against torch's and CPython's own classes, has to be built again."""
import os
import sysconfig

import torch

from packkv_b200 import build


def test_host_extension_is_rebuilt_for_another_torch_python_or_command(tmp_path, monkeypatch):
    lib, stamp = tmp_path / "_host.so", tmp_path / "_host.stamp"
    monkeypatch.setattr(build, "HOST_LIB", str(lib))
    monkeypatch.setattr(build, "HOST_STAMP", str(stamp))
    assert build._host_stale()
    lib.write_bytes(b"")
    assert build._host_stale()                               # of unknown make
    stamp.write_text(build._host_key())
    assert not build._host_stale()
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", torch.__version__ + "x")
        assert build._host_stale()
    with monkeypatch.context() as m:
        soabi = sysconfig.get_config_var("SOABI")
        m.setattr(sysconfig, "get_config_var", lambda name: soabi + "x")
        assert build._host_stale()
    with monkeypatch.context() as m:
        command = build._host_command()
        m.setattr(build, "_host_command", lambda: command + ["-g"])
        assert build._host_stale()
    assert not build._host_stale()
    os.utime(lib, (0, 0))                                    # older than its source
    assert build._host_stale()


def test_cluster_barriers_of_a_whole_warp_follow_a_convergence_point():
    """barrier.cluster with .aligned is executed by the threads of a warp as one: a __syncwarp() or __syncthreads() stands on the lines before it."""
    with open(os.path.join(build.CSRC, "attn.cu")) as f:
        lines = [line for line in f.read().splitlines() if line.strip() and not line.strip().startswith("//")]
    at = [i for i, line in enumerate(lines) if "barrier.cluster." in line and ".aligned" in line]
    assert at
    for i in at:
        assert any("__syncwarp()" in line or "__syncthreads()" in line for line in lines[i - 4: i]), lines[i].strip()
