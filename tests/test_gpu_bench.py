"""bench.py's 3D section where the reference's CPU build is not there."""
import argparse

import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def test_3d_section_without_the_reference_build(monkeypatch, tmp_path):
    import bench
    from oracle import refbind

    torch = torch_cuda()
    monkeypatch.setattr(refbind, "LIB_PATH", str(tmp_path / "none.so"))
    out = bench.threed_section(argparse.Namespace(steps=3), torch.device("cuda"), True)
    assert "unavailable" in out["cpu_reference"] and out["rect3d"]["solves_per_s"] > 0 and out["composite3d"]["solves_per_s"] > 0
