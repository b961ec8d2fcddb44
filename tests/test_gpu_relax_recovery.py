"""Builds and runs tests/cpp/relax_recovery.cu: the 2D model's sort after a device error."""
import subprocess
from pathlib import Path

import pytest

from libcl_gb300.build import ARCH, LIBDIR, NVCC, NVCC_FLAGS

ROOT = Path(__file__).resolve().parent.parent
pytestmark = pytest.mark.gpu


def test_2d_sort_recovers_from_a_device_error(cuda, tmp_path):
    exe = tmp_path / "relax_recovery"
    rest = [str(o) for o in sorted((LIBDIR / "obj").glob("*.o")) if o.stem != "fluid2d"]
    cmd = [NVCC, *ARCH, *NVCC_FLAGS, "-w", str(ROOT / "tests" / "cpp" / "relax_recovery.cu"), *rest, "-o", str(exe), "-lcuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr
