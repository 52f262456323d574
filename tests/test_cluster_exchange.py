"""CPU: the exchange bookkeeping of the cluster kernel (cuda_b200/csrc/cluster_exchange.h)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_exchanges_after_a_wait_gave_up(tmp_path):
    """A host model under random schedules: when CTAs give up, no barrier is armed twice and the words
    on their way to each are accounted for."""
    exe = tmp_path / "cluster_exchange_selftest"
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "cluster_exchange_selftest.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
