"""The staged coefficient stream of the tiled wavelets (csrc/stages.cuh) on host
threads: a bounded wait that runs out leaves no lane of a warp waiting for the
others, the copies in flight land first, and a fence orders a stage's reads
before the copy that writes it again (a C++ check compiled here)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_staged_stream_on_host_threads(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "stages_check"
    subprocess.run([cxx, "-x", "c++", "-O1", "-std=c++17", "-pthread", f"-I{ROOT / 'stl-dev-mpi_b200' / 'csrc'}",
                    str(ROOT / "tests" / "stages_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "fails 0" in r.stdout
