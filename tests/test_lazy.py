"""CPU: the lazily reduced transforms (cuda_b200/csrc/lazy_core.cuh), compiled for the host."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_lazy_transforms_host_build(tmp_path):
    """Transforms of 2 to 16 points on extreme 64-bit words and on products: congruent to
    the canonical ones, every intermediate within the three-word range."""
    exe = tmp_path / "lazy_selftest"
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "lazy_selftest.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
