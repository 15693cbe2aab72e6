"""The native call module belongs to one torch build."""
import subprocess
import sys

import torch

from conftest import ROOT


def test_host_module_is_stale_under_another_torch(monkeypatch, tmp_path):
    from gemq_b200.csrc import build
    monkeypatch.setattr(build.os.path, "getmtime", lambda path: 0.0)  # no source is newer
    monkeypatch.setattr(build, "HOST_STAMP", str(tmp_path / "host.torch"))
    assert build.host_stale()
    (tmp_path / "host.torch").write_text(build.torch_build())
    assert not build.host_stale()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.host_stale()


def test_missing_host_module_says_how_to_build_it():
    code = "import sys; sys.modules['gemq_b200._host'] = None\nimport gemq_b200._capi"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode != 0 and "python -m gemq_b200.csrc.build" in r.stderr, r.stderr[-500:]
